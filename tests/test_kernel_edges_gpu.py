"""Kernels at the edges of their tiles and value ranges, against the CPU oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from bitlattice_b200 import _ops

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.view(torch.uint8).cpu().numpy()


@pytest.mark.parametrize("N,K,g", [(16, 16, 0.0137), (128, 128, 1.0), (144, 272, 3.1e-4), (64, 400, 0.77), (2064, 144, 1e-3),
                                   (256, 64, 1e-30), (256, 64, 2.5e27)])
def test_requantize_t_ties_and_edges(N, K, g):
    """W^T re-quantization with few-bit block scales and per-tensor scales of 1.0, where many quotients sit at midpoints
    between levels, tiles that are cut off on either side, scales outside the packed route's range, zero scale bytes."""
    rng = np.random.default_rng(N * K)
    codes = rng.integers(0, 256, (N, K // 2), dtype=np.uint8)
    scales = rng.integers(0x28, 0x50, (N, K // 16), dtype=np.uint8)
    scales[rng.random(scales.shape) < 0.05] = 0
    codes[: N // 2] &= 0x77 if N == 64 else 0xFF
    rc, rs = oracle.requantize_t(codes, scales, g)
    for blocked in (False, True):
        packed, sc, gout = _ops.requantize_nvfp4_t(dev(codes), dev(scales), dev(np.array([g], np.float32)), blocked=blocked)
        assert np.array_equal(host(packed), rc)
        want = oracle.to_blocked(rs) if blocked else rs
        assert np.array_equal(host(sc).reshape(want.shape), want)
        assert gout.item() == np.float32(g)


@pytest.mark.parametrize("rows,cols16", [(1, 1), (5, 4), (128, 4), (129, 8), (300, 12), (127, 6), (257, 64)])
def test_to_blocked_words_and_bytes(rows, cols16):
    s = np.random.default_rng(rows).integers(0, 256, (rows, cols16), dtype=np.uint8)
    assert np.array_equal(host(_ops.to_blocked(dev(s))), oracle.to_blocked(s).reshape(-1))
