"""The library linked once more with a limit on device memory, to see what calls
do when an allocation fails: cudaMalloc and cudaMallocArray are wrapped at link
time (ld --wrap) and refuse what would pass the limit, with the error the
runtime gives when a device is full.  Loaded by a process of its own (run)."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

from hydrant_gb300 import build as hb

ROOT = Path(__file__).resolve().parent.parent

WRAP = r"""
#include <cuda_runtime_api.h>
#include <map>
#include <mutex>
static std::mutex mu;
static std::map<const void *, size_t> sizes;
static size_t live = 0, limit = ~size_t(0), most = 0;
static int arrays = 1, array_calls = 0;
static bool take(size_t n) {
    std::lock_guard<std::mutex> l(mu);
    if (live + n > limit) return false;
    live += n;
    if (live > most) most = live;
    return true;
}
static void keep(const void *p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    sizes[p] = n;
}
static void give(const void *p) {
    std::lock_guard<std::mutex> l(mu);
    auto i = sizes.find(p);
    if (i == sizes.end()) return;
    live -= i->second;
    sizes.erase(i);
}
extern "C" {
cudaError_t __real_cudaMalloc(void **, size_t);
cudaError_t __real_cudaFree(void *);
cudaError_t __real_cudaMallocArray(cudaArray_t *, const cudaChannelFormatDesc *, size_t, size_t,
                                   unsigned int);
cudaError_t __real_cudaFreeArray(cudaArray_t);
cudaError_t __wrap_cudaMalloc(void **p, size_t n) {
    if (!take(n)) return cudaErrorMemoryAllocation;
    cudaError_t e = __real_cudaMalloc(p, n);
    if (e == cudaSuccess) keep(*p, n);
    return e;
}
cudaError_t __wrap_cudaFree(void *p) {
    give(p);
    return __real_cudaFree(p);
}
cudaError_t __wrap_cudaMallocArray(cudaArray_t *a, const cudaChannelFormatDesc *d, size_t w,
                                   size_t h, unsigned int flags) {
    const size_t n = (size_t)(d->x + d->y + d->z + d->w) / 8 * w * (h ? h : 1);
    ++array_calls;
    if (!arrays || !take(n)) return cudaErrorMemoryAllocation;
    cudaError_t e = __real_cudaMallocArray(a, d, w, h, flags);
    if (e == cudaSuccess) keep(*a, n);
    return e;
}
cudaError_t __wrap_cudaFreeArray(cudaArray_t a) {
    give(a);
    return __real_cudaFreeArray(a);
}
cudaError_t __real_cudaMemGetInfo(size_t *, size_t *);
cudaError_t __wrap_cudaMemGetInfo(size_t *f, size_t *t) {
    cudaError_t e = __real_cudaMemGetInfo(f, t);
    std::lock_guard<std::mutex> l(mu);
    if (e == cudaSuccess && limit < *t) {
        *t = limit;
        *f = limit > live ? limit - live : 0;
    }
    return e;
}
void test_memory_limit(size_t n) { limit = n; most = live; }
size_t test_memory_live(void) { return live; }
size_t test_memory_most(void) { return most; }
void test_memory_arrays(int allowed) { arrays = allowed; }
int test_memory_array_calls(void) { return array_calls; }
}
"""

PRELUDE = """
import ctypes as C, sys
from pathlib import Path
sys.path.insert(0, {root!r})
from hydrant_gb300 import _abi
_abi.LIB_PATH = Path({lib!r})
mem = _abi.lib()
mem.test_memory_limit.argtypes = [C.c_size_t]
mem.test_memory_live.restype = mem.test_memory_most.restype = C.c_size_t
"""


def build(folder: Path) -> Path:
    objs = [hb.BUILD / (Path(s).stem + ".o") for s in hb.SOURCES]
    if not all(o.exists() for o in objs):
        pytest.skip("the library's object files are not here")
    src, lib = folder / "wrap.cc", folder / "liblimited.so"
    src.write_text(WRAP)
    names = ("cudaMalloc", "cudaFree", "cudaMallocArray", "cudaFreeArray", "cudaMemGetInfo")
    cmd = [hb.nvcc(), *hb.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", str(lib),
           str(src), *map(str, objs), *(f"-Xlinker=--wrap={n}" for n in names), "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return lib


def run(lib: Path, code: str) -> str:
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=str(ROOT), lib=str(lib)) + code],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
