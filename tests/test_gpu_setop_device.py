"""Set operations on device arrays, with the offsets checked on the device: results at the
lengths where the lookups change (32 keys, tiles of 512, lists more than 16 times as long as the
other), and the errors of the host check."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 5, 31, 32, 33, 64, 65, 128, 129, 511, 512, 513, 1024, 1025, 3000]


def _p(t, kind=ctypes.c_int32):
    return None if t is None else ctypes.cast(t.data_ptr(), ctypes.POINTER(kind))


def _call(gpu, op, a, ao, b, bo, n, counts, out, oo):
    i64 = ctypes.c_int64
    return gpu.lib().jgpm_setop_batch(op, _p(a), _p(ao, i64), _p(b), _p(bo, i64), n, None, None,
                                      _p(counts), _p(out), _p(oo, i64))


def _offsets(lists):
    return np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int64)


@pytest.mark.parametrize("op", range(4))
def test_results_at_step_edges(gpu, op):
    rng = np.random.default_rng(op)
    span = [4000, 100000]  # dense and sparse
    pairs = [(rng.choice(span[k % 2], x, replace=False), rng.choice(4000, y, replace=False))
             for k, x in enumerate(LENGTHS) for y in LENGTHS]
    A = [np.sort(x).astype(np.int32) for x, _ in pairs]
    B = [np.sort(y).astype(np.int32) for _, y in pairs]
    # the largest id is a key like any other where no bound is given
    A[-1][-1] = B[-1][-1] = np.iinfo(np.int32).max
    ref = [np.intersect1d(x, y) if op < 2 else np.setdiff1d(x, y) for x, y in zip(A, B)]
    cap = [min(len(x), len(y)) if op == 0 else len(x) for x, y in zip(A, B)]
    oo = np.concatenate([[0], np.cumsum(cap)]).astype(np.int64)
    dev = [torch.from_numpy(np.concatenate(x)).cuda() for x in (A, B)]
    off = [torch.from_numpy(_offsets(x)).cuda() for x in (A, B)]
    counts = torch.full((len(A),), -1, dtype=torch.int32, device="cuda")
    out = torch.full((int(oo[-1]),), -7, dtype=torch.int32, device="cuda")
    d_oo = torch.from_numpy(oo).cuda()
    # no synchronisation: the call waits for what is queued on the default stream
    mat = op in (0, 2)
    assert _call(gpu, op, dev[0], off[0], dev[1], off[1], len(A), counts,
                 out if mat else None, d_oo if mat else None) == 0
    assert counts.cpu().tolist() == [len(x) for x in ref]
    if mat:
        got = out.cpu().numpy()
        for i, x in enumerate(ref):
            assert (got[oo[i]: oo[i] + len(x)] == x).all(), i
            assert (got[oo[i] + len(x): oo[i + 1]] == -7).all(), i


# counts on the host with everything else on the device: they are staged, and a refused call
# must not copy the staging buffer back
@pytest.mark.parametrize("counts_at", ["cuda", "host"])
@pytest.mark.parametrize("where", ["host", "cuda"])
def test_offset_errors(gpu, where, counts_at):
    a = torch.arange(8, dtype=torch.int32, device="cuda")
    counts = torch.full((2,), -1, dtype=torch.int32,
                        device="cuda" if counts_at == "cuda" else "cpu")
    out = torch.zeros(8, dtype=torch.int32, device="cuda")

    def off(*x):
        t = torch.tensor(x, dtype=torch.int64)
        return t.cuda() if where == "cuda" else t

    good = off(0, 4, 8)
    torch.cuda.synchronize()
    for ao, bo, oo, null, code in [
            (off(0, 5, 3), good, good, False, -1), (off(-1, 4, 8), good, good, False, -1),
            (good, off(4, 2, 8), good, False, -1), (good, good, off(0, 3, 8), False, -10),
            (good, good, off(0, 3, 8), True, -1),  # missing operand before capacity
            (off(0, 4, 1), good, off(0, 3, 8), False, -10),  # the first pair's error
            (off(0, 9, 1), good, good, False, -1), (good, good, good, False, 0)]:
        assert _call(gpu, 0, None if null else a, ao, a, bo, 2, counts, out, oo) == code
        if code:
            assert counts.cpu().tolist() == [-1, -1]
    assert counts.cpu().tolist() == [4, 4]


@pytest.mark.parametrize("counts_at", ["cuda", "host"])
@pytest.mark.parametrize("where", ["host", "cuda"])
def test_refused_split_writes_nothing(gpu, where, counts_at):
    a = torch.arange(8, dtype=torch.int32, device="cuda")
    c, d = torch.full_like(a, -7), torch.full_like(a, -7)
    counts = torch.full((4,), -1, dtype=torch.int32,
                        device="cuda" if counts_at == "cuda" else "cpu")
    i64 = ctypes.c_int64

    def off(*x):
        t = torch.tensor(x, dtype=torch.int64)
        return t.cuda() if where == "cuda" else t

    def split(ao, bo):
        return gpu.lib().jgpm_setop_split_batch(
            gpu.SPLIT_DIF_INT, _p(a), _p(ao, i64), _p(a), _p(bo, i64), 2, None, _p(counts),
            _p(c), _p(d), None)

    good = off(0, 4, 8)
    torch.cuda.synchronize()
    for ao, bo in [(off(0, 5, 3), good), (good, off(4, 2, 8)), (off(-1, 4, 8), good)]:
        assert split(ao, bo) == -1
        assert counts.tolist() == [-1] * 4 and (c == -7).all() and (d == -7).all()
    assert split(good, good) == 0
    assert counts.tolist()[0] in (0, 4)
