"""The recount behind the executors of a call with an expiry threshold: it
writes into the host's status mirror, so it does so only for a call that
waits for it.  A call that is rejected, whose sort gave up or whose buckets
overflowed returns without waiting, and its recount writes nothing."""
import ctypes

import numpy as np
import pytest

from harness import link
from test_gpu_parity import _dev, assert_same

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstring>
#include "kernels.cuh"
using namespace lpma;
// nseg segments of 3 keys; out: the mirror's counted and cnt_total, the
// status block's cnt_total and sum_done
extern "C" __attribute__((visibility("default"))) int probe(unsigned error, unsigned part_ovf, unsigned nseg,
                                                            unsigned long long *out) {
    DevStatus *st = nullptr, *pub = nullptr, *pub_dev = nullptr, init;
    unsigned char *cnt = nullptr;
    std::memset(&init, 0, sizeof(init));
    init.error = error, init.part_ovf = part_ovf, init.seq = 9;
    if (cudaMalloc(&st, sizeof(DevStatus)) || cudaMalloc(&cnt, nseg + 64) || cudaMemset(cnt, 3, nseg + 64) ||
        cudaMemcpy(st, &init, sizeof(init), cudaMemcpyHostToDevice) || cudaMallocHost(&pub, sizeof(DevStatus)) ||
        cudaHostGetDevicePointer((void **)&pub_dev, pub, 0))
        return 1;
    std::memset(pub, 0, sizeof(DevStatus));
    pub->counted = 8, pub->cnt_total = 77;
    launch_sum_cnt(cnt, nseg, st, 0, pub_dev);
    if (cudaDeviceSynchronize() || cudaMemcpy(&init, st, sizeof(init), cudaMemcpyDeviceToHost)) return 2;
    out[0] = pub->counted, out[1] = pub->cnt_total, out[2] = init.cnt_total, out[3] = init.sum_done;
    return cudaFree(st) || cudaFree(cnt) || cudaFreeHost(pub);
}
"""

ERR_KEY, ERR_TIMEOUT = 1, 4  # lpma_common.cuh


def test_recount_of_a_refused_call_writes_nothing(engine, tmp_path):
    lib = link(tmp_path, "recount", PROGRAM)
    out = (ctypes.c_ulonglong * 4)()
    for nseg in (1, 15, 511, 100000):
        assert lib.probe(0, 0, nseg, out) == 0
        assert list(out)[:3] == [9, 3 * nseg, 3 * nseg] and out[3] >= 1
        for error, ovf in ((ERR_KEY, 0), (ERR_TIMEOUT, 0), (0, 1), (ERR_KEY, 1)):
            assert lib.probe(error, ovf, nseg, out) == 0
            assert list(out) == [8, 77, 0, 0]


@pytest.mark.parametrize("scale", [6, 12])
def test_rejected_calls_between_ticks(engine, oracle, scale):
    """A rejected call with a threshold, then the tick itself: the stored
    count is the tick's own."""
    V = 1 << scale
    pool = oracle.shuffle(oracle.rmat_edges(5, scale, 16), 6)
    n = min(300, pool.size // 8)
    pool = pool | (np.arange(pool.size, dtype=np.uint64) // np.uint64(n) + np.uint64(1))
    g, o = engine.Lpma(V), oracle.OracleLpma(V)
    for t in range(8):
        ins = pool[n * t:n * t + n]
        thres = max(1, t - 3)
        bad = ins.copy()
        bad[-1] = np.uint64(V) << np.uint64(42)
        with pytest.raises(engine.LpmaError):
            g.update(ins=_dev(bad), thres=thres)
        sg = g.update(ins=_dev(ins), thres=thres)
        o.update(ins=ins, thres=thres)
        assert sg["num_items"] == o.num_items()
        assert_same(g, o, "tick %d" % t)
    g.close()
