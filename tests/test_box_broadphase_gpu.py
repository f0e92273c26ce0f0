"""Box broadphase: the candidate list equals a brute-force search, in order, over grids whose dims
are and are not powers of two, bodies on both sides of the cell origin (columns that wrap),
scenes whose shift breaks a column, body counts around a CTA's, and with the partners kept from
the count to the emission or searched again (few candidate slots).  Integers: no tolerance."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import cuda_ok

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_ok(), reason="needs a CUDA device")]
MARGIN = np.float32(2e-3)


def _brute(x, half, scene):
    r = np.sqrt((half[:, 0] * half[:, 0] + half[:, 1] * half[:, 1]) + half[:, 2] * half[:, 2])
    ca, cb = [], []
    for i in range(len(x)):
        if x[i, 2] - r[i] < float(MARGIN) + 1e-9:
            ca.append(i), cb.append(-1)
        d = x[i] - x[i + 1:]
        rr = (r[i] + r[i + 1:]) + float(MARGIN)
        hit = np.nonzero(((d[:, 0] ** 2 + d[:, 1] ** 2) + d[:, 2] ** 2 <= rr ** 2) & (scene[i + 1:] == scene[i]))[0]
        ca += [i] * len(hit)
        cb += list(hit + i + 1)
    return np.array(ca, np.int32), np.array(cb, np.int32)


@pytest.mark.parametrize("listed", [True, False])
@pytest.mark.parametrize("n,dims,scenes", [(1, (8, 8, 8), 1), (7, (16, 16, 8), 1), (8, (9, 10, 11), 1),
                                           (9, (16, 16, 8), 3), (500, (16, 16, 8), 1), (501, (13, 16, 9), 1),
                                           (1500, (16, 16, 8), 40), (1501, (9, 8, 11), 37)])
def test_candidates_match_brute_force(me, n, dims, scenes, listed):
    rng = np.random.default_rng(n)
    dev, lib = "cuda:0", me._lib
    L = lib.load()
    side = 0.25 * (n / scenes) ** (1 / 3) + 0.2
    x = rng.uniform(-side, side, (n, 3)).astype(np.float32)
    x[:, 2] += np.float32(side / 2)
    half = rng.uniform(0.08, 0.2, (n, 3)).astype(np.float32)
    scene = np.sort(rng.integers(0, scenes, n)).astype(np.int32)
    ca, cb = _brute(x.astype(np.float64), half.astype(np.float64), scene)
    cap = max(len(ca), 1)
    if listed:
        cap = max(cap, 2 * n)
    else:
        cap = min(cap, 2 * n - 1)
    i32 = lambda k: torch.zeros(int(k), dtype=torch.int32, device=dev)
    pad = lambda a: torch.from_numpy(np.concatenate([a, np.zeros((n, 1), np.float32)], 1)).to(dev)
    xc, hf, sc, hdr = pad(x), pad(half), torch.from_numpy(scene).to(dev), i32(8)
    nbk = dims[0] * dims[1] * dims[2]
    B = dict(bucket=i32(n), start=i32(nbk + 1), cursor=i32(nbk + 1), sorted=i32(n), cand_count=i32(n + 1),
             cand_offset=i32(n + 1), cand_a=i32(cap), cand_b=i32(cap), cont_count=i32(cap + 1), cont_offset=i32(cap + 1),
             pair_flag=i32(cap + 1), pair_offset=i32(cap + 1), slot_p=i32(32 * cap), slot_n=i32(4 * cap),
             slot_f=i32(8 * cap), scan_tmp=i32(L.b2c_scan_scratch_ints(max(nbk, n, cap) + 1) + 1))
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    cell = 1.01 * (2.0 * float(np.sqrt((half.astype(np.float64) ** 2).sum(1)).max()) + float(MARGIN))
    bx = lib.Boxes(n, p(hf), None, MARGIN, cell, *dims, cap, *(p(t) for t in B.values()), p(sc) if scenes > 1 else None)
    bd = lib.Bodies(n, p(xc))
    s = torch.cuda.current_stream().cuda_stream
    lib.check(L.b2c_box_candidates(ctypes.byref(bd), ctypes.byref(bx), p(hdr), ctypes.c_void_p(s)), "candidates")
    torch.cuda.synchronize()
    total = int(B["cand_offset"][n])
    assert total == len(ca)
    m = min(total, cap)
    assert int(hdr[6]) == (64 if total > cap else 0)  # the error word: the pair overflow, where asked for
    assert np.array_equal(B["cand_a"].cpu().numpy()[:m], ca[:m]) and np.array_equal(B["cand_b"].cpu().numpy()[:m], cb[:m])
