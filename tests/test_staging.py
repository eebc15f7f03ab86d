"""The host copies into page-locked memory (csrc/staging.cuh), compiled by the host's compiler alone."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = os.path.join(ROOT, "dinara-align_b200", "csrc")

# Sizes either side of the 64 KB from which stores pass the caches, of 16 bytes and of a thread's half megabyte, from
# sources on and off a boundary, the bytes on either side left as they were.
COPIES = r"""
#include "staging.cuh"
#include <cstdio>
#include <vector>
int main() {
    const size_t sizes[] = {0, 1, 15, 16, 17, 65535, 65536, 65537, 65551, 524287, 524288, 524289, 1048575, 1048576,
                            3000001, 4194303, 4194304, 4194321, 9000007};
    for (size_t size : sizes)
        for (size_t off : {size_t(0), size_t(5)}) {
            std::vector<uint8_t> from(size + off + 1), room(size + 128 + 64, 0xAB);
            for (size_t i = 0; i < from.size(); ++i) from[i] = uint8_t(i * 2654435761u >> 24);
            uint8_t *to = room.data() + (64 - reinterpret_cast<uintptr_t>(room.data()) % 64) % 64 + 64;
            dinara::stage_copy(to, from.data() + off, size);
            if (std::memcmp(to, from.data() + off, size) != 0 || to[-1] != 0xAB || to[size] != 0xAB) {
                std::printf("%zu bytes from %zu\n", size, off);
                return 1;
            }
        }
    return 0;
}
"""


def _run(tmp_path, source, *flags):
    path, program = tmp_path / "copies.cpp", tmp_path / "copies"
    path.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", SOURCES, *flags, str(path), "-o", str(program), "-lpthread"],
                   check=True, capture_output=True, text=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr


@pytest.mark.parametrize("host", ["this", "without SSE2"])
def test_copies(tmp_path, host):
    """On this host, and as a host that has neither the stores past the caches nor their header builds it."""
    flags = []
    if host != "this":
        (tmp_path / "emmintrin.h").write_text("#error a header of other hosts\n")
        flags = ["-U__SSE2__", "-I", str(tmp_path)]
    _run(tmp_path, COPIES, *flags)


# A thread cannot be started from the `ALLOWED`th on.
FAILING = r"""
#include <cerrno>
#include <dlfcn.h>
#include <pthread.h>
extern "C" int pthread_create(pthread_t *thread, const pthread_attr_t *attributes, void *(*body)(void *), void *argument) {
    static int calls = 0;
    if (calls++ % 8 >= ALLOWED) return EAGAIN;
    using Create = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Create create = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
    return create(thread, attributes, body, argument);
}
"""


@pytest.mark.parametrize("allowed", [0, 1, 3])
def test_copies_where_threads_cannot_start(tmp_path, allowed):
    """They end with every byte copied, not with the process."""
    _run(tmp_path, FAILING + COPIES, f"-DALLOWED={allowed}", "-rdynamic", "-ldl")
