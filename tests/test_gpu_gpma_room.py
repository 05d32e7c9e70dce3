"""GPMA batches whose buckets find no memory: the sorted front takes them, as
it took every batch before there were buckets.  The engine's objects are linked
here with an allocator that refuses requests above a limit."""
import ctypes

import pytest

from harness import link

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstring>
#include <vector>
#include "gpma.cuh"
#include "kernels.cuh"
#include "lpma.h"
static size_t g_limit = ~size_t(0), g_refused = 0, g_most = 0;
cudaError_t lpma::pool_alloc(void **p, size_t bytes, cudaStream_t s) {
    if (bytes > g_limit) {
        g_refused++;
        return cudaErrorMemoryAllocation;
    }
    if (bytes > g_most) g_most = bytes;
    return cudaMallocAsync(p, bytes, s);
}
using namespace lpma;
// Two arrays of V rows get `load` keys each and then the batch: one with room
// for everything, one with no room for the buckets' one allocation.  0: both
// hold the same slots in the end, and the second was refused that allocation
// (once: no call after it asks for it for a while).
extern "C" __attribute__((visibility("default"))) int probe(uint32_t V, const uint64_t *load, size_t n_load,
                                                            const uint64_t *ins, size_t n_ins, const uint64_t *del,
                                                            size_t n_del) {
    uint64_t *d = nullptr;
    if (cudaMalloc(&d, (n_load + n_ins + n_del) * 8)) return 1;
    uint64_t *di = d + n_load, *dd = di + n_ins;
    if (cudaMemcpy(d, load, n_load * 8, cudaMemcpyHostToDevice) || cudaMemcpy(di, ins, n_ins * 8, cudaMemcpyHostToDevice) ||
        cudaMemcpy(dd, del, n_del * 8, cudaMemcpyHostToDevice))
        return 2;
    std::vector<uint64_t> k[2];
    std::vector<uint8_t> v[2];
    size_t arena = 0;
    for (int turn = 0; turn < 2; turn++) {
        GpmaState *g = nullptr;
        LpmaStats st;
        g_limit = ~size_t(0);
        if (gpma_create(V, 0.15, 0, &g) || gpma_update(g, d, nullptr, n_load, nullptr, 0, 0, &st)) return 3;
        g_most = g_refused = 0;
        if (turn) g_limit = arena - 1;
        if (gpma_update(g, di, nullptr, n_ins, dd, n_del, 0, &st)) return 4;
        if (!turn) arena = g_most;
        if (g_refused != (turn ? 1u : 0u)) return 5;
        // a rejected key, and the batch taken back
        uint64_t bad = ~0ull;
        if (cudaMemcpy(d, &bad, 8, cudaMemcpyHostToDevice) ||
            gpma_update(g, d, nullptr, 1, nullptr, 0, 0, &st) != LPMA_ERR_INVALID_KEY)
            return 6;
        if (cudaMemcpy(d, load, 8, cudaMemcpyHostToDevice)) return 7;
        if (gpma_update(g, dd, nullptr, n_del, di, n_ins, 0, &st)) return 8;
        uint64_t size;
        uint32_t seg, h;
        gpma_geometry(g, &size, &seg, &h, nullptr);
        k[turn].resize(size), v[turn].resize(size);
        if (gpma_export_layout(g, k[turn].data(), v[turn].data(), size, nullptr, 0, 0)) return 9;
        if (turn && g_refused != 1) return 10;
        gpma_destroy(g);
    }
    g_limit = ~size_t(0);
    cudaFree(d);
    return k[0] == k[1] && v[0] == v[1] ? 0 : 11;
}
"""


@pytest.mark.parametrize("n", [300, 5000, 60000])
def test_no_room_for_the_buckets(engine, oracle, tmp_path, n):
    import numpy as np
    lib = link(tmp_path, "gpma_room", PROGRAM, without=("abi.o", "pool.o", "noalloc.o", "loader.o"))
    V = 1 << 13
    e = oracle.shuffle(oracle.rmat_edges(5, 13, 32), 2)
    e = ((e >> np.uint64(42)) << np.uint64(32)) | ((e >> np.uint64(20)) & np.uint64(0x3FFFFF))  # src << 32 | dst
    load, ins = e[:120000].copy(), e[120000:120000 + n].copy()
    dels = load[: n // 3].copy()
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    lib.probe.argtypes = [ctypes.c_uint32] + [ctypes.c_void_p, ctypes.c_size_t] * 3
    assert lib.probe(V, p(load), load.size, p(ins), ins.size, p(dels), dels.size) == 0
