"""Kernels at the edges of their tiles and value ranges, against the CPU oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import bitlattice_b200 as bl
from bitlattice_b200 import _C, _ops, backend

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


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_requantize_t_scales_at_any_address(shift, layout):
    """Scale buffers that start inside a word are written by bytes, and nothing beside them is."""
    N, K, g = 128, 64, 0.0137
    rng = np.random.default_rng(5)
    codes, scales = rng.integers(0, 256, (N, K // 2), dtype=np.uint8), rng.integers(0x28, 0x50, (N, K // 16), dtype=np.uint8)
    rc, rs = oracle.requantize_t(codes, scales, g)
    want = (oracle.to_blocked(rs) if layout else rs).reshape(-1)
    gd, out, gout = dev(np.array([g], np.float32)), torch.empty(K, N // 2, dtype=torch.uint8, device="cuda"), torch.empty(1, device="cuda")
    raw = torch.full((want.size + 16,), 0xEE, dtype=torch.uint8, device="cuda")
    packed, sc = dev(codes), dev(scales)
    _C.call("bl_nvfp4_requantize_t", packed.data_ptr(), sc.data_ptr(), gd.data_ptr(), N, K, out.data_ptr(), raw.data_ptr() + 8 + shift,
            gout.data_ptr(), layout, 0, torch.cuda.current_stream().cuda_stream)
    got = host(raw)
    assert np.array_equal(host(out), rc) and np.array_equal(got[8 + shift:8 + shift + want.size], want)
    assert (got[:8 + shift] == 0xEE).all() and (got[8 + shift + want.size:] == 0xEE).all()


@pytest.mark.parametrize("rows,cols16", [(1, 1), (5, 4), (128, 4), (129, 8), (300, 12), (127, 6), (257, 64)])
def test_to_blocked_words_and_bytes(rows, cols16):
    s = np.random.default_rng(rows).integers(0, 256, (rows, cols16), dtype=np.uint8)
    assert np.array_equal(host(_ops.to_blocked(dev(s))), oracle.to_blocked(s).reshape(-1))


def _sr_values(kind, shape, rng):
    if kind == "normal":
        return rng.standard_normal(shape).astype(np.float32)
    if kind == "levels":                 # on levels, midpoints and just beside them: draws against fractions of 0, 1/2, ...
        v = rng.choice(np.array([0, 0.25, 0.5, 0.75, 1, 1.25, 1.5, 2, 2.5, 3, 3.5, 4, 5, 6], np.float32), shape)
        return v * rng.choice(np.array([1, -1, 1 + 2.0 ** -8, 2.0 ** -20, 2.0 ** -130], np.float32), shape)
    return (rng.standard_normal(shape) * 10.0 ** rng.uniform(-30, 3, shape)).astype(np.float32)     # "wide"


@pytest.mark.parametrize("kind", ["normal", "levels", "wide"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_stochastic_draws_on_all_bits(kind, dtype):
    """Stochastic rounding of 2^22 elements, rows and transposed: about 60 of them draw a number whose upper 16 bits equal
    those of their position between two levels and are decided on the bits below. Per-tensor scales above, at and below
    the data's own (the last one saturates the block scales, so that values lie far beyond the last level)."""
    rng = np.random.default_rng(7)
    x = torch.from_numpy(_sr_values(kind, (2048, 2048), rng)).to(dtype)
    xf = x.float().numpy()
    g0 = np.float32(max(np.abs(xf).max() / 2688.0, 1e-12))
    for g in (g0, np.float32(g0 * 4), np.float32(g0 / 37)):
        rc, rs, _ = oracle.quantize_rows(xf, float(g), "sr", seed=11)
        packed, sc = _ops.quantize_nvfp4(x.cuda(), dev(np.array([g], np.float32)), seed=11)
        assert np.array_equal(host(packed), rc) and np.array_equal(host(sc), rs)
    H = oracle.hadamard16()
    for h in (H, None):
        bound = np.float32(g0 * 4)
        gt = oracle.global_from_bound(float(bound))
        rc, rs = oracle.quantize_t(xf, h, gt, "sr", seed=5)
        packed, sc, _ = _ops.quantize_nvfp4_t(x.cuda(), dev(h.astype(np.float32)) if h is not None else None, 5, 0,
                                              dev(np.array([bound], np.float32)))
        assert np.array_equal(host(packed), rc) and np.array_equal(host(sc), rs)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_every_gate_value(dtype):
    """Every 16-bit gate value (zeros of both signs, subnormals, infinities, NaN) through both kernels: the shared
    reciprocal gives the bits of the expression with its two plain divisions. Laid out twice, so that in-range and
    out-of-range values share vectors of eight in one and are alone in the other."""
    bits = torch.arange(1 << 16, device="cuda", dtype=torch.int32)
    order = torch.cat([bits, (bits * 40503) & 0xFFFF])
    g = order.to(torch.int16).view(dtype)
    gen = torch.Generator(device="cuda").manual_seed(3)
    u = torch.randn(g.numel(), device="cuda", generator=gen).to(dtype)
    da = torch.randn(g.numel(), device="cuda", generator=gen).to(dtype)
    gf, uf, df = g.float(), u.float(), da.float()
    d = 1.0 + torch.exp(-gf)
    silu = (gf / d).to(dtype).float()
    sig = 1.0 / d
    want = ((silu * uf).to(dtype), ((df * uf).to(dtype).float() * sig * (1.0 + gf * (1.0 - sig))).to(dtype), (df * silu).to(dtype))
    got = (_ops.swiglu_fwd(g, u), *_ops.swiglu_bwd(g, u, da))
    for a, b in zip(got, want):
        nan = b.isnan()
        assert torch.equal(a.isnan(), nan)
        assert torch.equal(a.view(torch.int16)[~nan], b.view(torch.int16)[~nan])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 48), (257, 32), (4096, 4096)])
def test_dequantize_every_code(rows, cols, dtype):
    """Level x (scale x global) rounded once to the output type, code 8 (-0) as +0, into an output that is 32-byte aligned
    and into one that is only 16-byte aligned."""
    rng = np.random.default_rng(rows + cols)
    codes = rng.integers(0, 256, (rows, cols // 2), dtype=np.uint8)
    scales = rng.integers(0, 0x7F, (rows, cols // 16), dtype=np.uint8)
    g = torch.tensor([0.0137], device="cuda")
    level = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], device="cuda")
    c = dev(codes).int()
    nib = torch.stack([c & 15, c >> 4], -1).view(rows, cols)
    s = dev(scales).view(torch.float8_e4m3fn).float() * g
    want = (level[nib] * s.repeat_interleave(16, 1)).to(dtype)
    raw = torch.zeros(rows * cols + 64, dtype=dtype, device="cuda")
    shifted = raw[16 // raw.element_size():][:rows * cols].view(rows, cols)
    packed, sc = dev(codes), dev(scales)
    _C.call("bl_nvfp4_dequantize", packed.data_ptr(), sc.data_ptr(), g.data_ptr(), rows, cols,
            shifted.data_ptr(), _C.DTYPE[dtype], 0, torch.cuda.current_stream().cuda_stream)
    for got in (_ops.dequantize(packed, sc, g, None, "nvfp4", rows, cols, dtype), shifted):
        assert torch.equal(got.contiguous().view(torch.uint8), want.view(torch.uint8))


@pytest.mark.parametrize("M", [1, 8, 9, 64, 65, 129])
@pytest.mark.parametrize("N,K", [(8, 32), (136, 288), (384, 1792), (1000, 4128)])
def test_tile_gemm_few_rows(M, N, K):
    """The tile kernel where it loads only the rows of A that exist (M <= 64) and where it loads whole tiles, k-tiles cut
    off after 1, 2 and 4 blocks and more k-tiles than stages, against the persistent kernel bit for bit."""
    gen = torch.Generator(device="cuda").manual_seed(M * N + K)
    a, b = (torch.randn(r, K, device="cuda", generator=gen).to(torch.bfloat16) for r in (M, N))
    qa, qb = (_ops.amax_quantize_nvfp4(t, -1, 0, blocked=True) for t in (a, b))
    outs = []
    try:
        for kernel in ("tile", "persistent"):
            _ops.gemm_select(kernel)
            outs.append(_ops.nvfp4_gemm(qa[0], qa[1], qa[2][1:2], qb[0], qb[1], qb[2][1:2]))
    finally:
        _ops.gemm_select("auto")
    assert torch.equal(outs[0], outs[1]) and outs[0].isfinite().all()
    assert _ops.gemm_status(0) == 0


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
@pytest.mark.parametrize("direction,dtype,lr", [("colnorm", torch.bfloat16, 3e-3), ("sign", torch.float32, 0.5),
                                                ("raw", torch.float16, 40.0)])
@pytest.mark.parametrize("rows,cols", [(1, 16), (37, 48), (300, 4112)])
def test_update_projection_edges(rows, cols, direction, dtype, lr, bits):
    """The fast update with 1 to 4 phase bits against the general route (the reference's arithmetic step by step), bit for
    bit: every code and phase, single groups, rows that end inside a block, targets beyond the last level (large lr),
    zero gradients (a group of them leaves the fast route), several steps so that rows are walked and carried over."""
    gen = torch.Generator(device="cuda").manual_seed(bits * rows + cols)
    cb = _ops.phase_container(bits)
    codes = torch.randint(0, 256, (rows, cols // 2), dtype=torch.uint8, device="cuda", generator=gen)
    scales = torch.randint(0x20, 0x48, (rows, cols // 16), dtype=torch.uint8, device="cuda", generator=gen)
    mask = sum(((1 << bits) - 1) << s for s in range(0, 8, cb))
    phase = torch.randint(0, 256, (rows, cols * cb // 8), dtype=torch.uint8, device="cuda", generator=gen) & mask
    grad = (torch.randn(rows, cols, device="cuda", generator=gen) * 1e-2).to(dtype)
    grad[:, 5] = 0 if rows == 37 else grad[:, 5]
    gs = torch.tensor([0.02], device="cuda")
    ends = []
    try:
        for route in ("auto", "general"):
            _ops.update_select(route)
            c, p, s = codes.clone(), phase.clone(), scales.clone()
            for step in (1, 2, 3):
                _ops.lattice_update(c, p, s, gs, None, grad, "nvfp4", rows, cols, lr=lr, weight_decay=0.0, phase_bits=bits,
                                    phase_cb=cb, rounding="sr", seed=77, step=step, strata=16, scale_rule="fit", trust=0.1,
                                    trust_lr=0.0, direction=direction)
            ends.append((c, p, s))
    finally:
        _ops.update_select("auto")
    for a, b in zip(*ends):
        assert torch.equal(a, b)


@pytest.mark.parametrize("seed", [-1, 7])
@pytest.mark.parametrize("rows,K,rotate,bound", [(1, 16, True, True), (17, 130, True, True), (33, 64, False, True),
                                                 (127, 192, True, False), (129, 95, True, True), (300, 1000, "other", True)])
def test_quantize_t_ragged_rows(rows, K, rotate, bound, seed):
    """Rows missing from the last block count as zeros: the bytes of the padded tensor, on the paired and the odd-width
    kernel, with the structured rotation, another matrix and none, with a bound and with the amax pass."""
    gen = torch.Generator(device="cuda").manual_seed(rows * K)
    x = torch.randn(rows, K, device="cuda", generator=gen).to(torch.bfloat16)
    padded = torch.nn.functional.pad(x, (0, 0, 0, -rows % 32))
    H = (torch.randn(16, 16, device="cuda", generator=gen) if rotate == "other"
         else backend._hadamard16(x.device, torch.float32) if rotate else None)
    g = torch.tensor([2e-3], device="cuda") if bound else None
    want = _ops.quantize_nvfp4_t(padded, H, seed, 0, g, blocked=True)
    got = _ops.quantize_nvfp4_t(x, H, seed, 0, g, blocked=True, pad_rows=32)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


@pytest.mark.parametrize("recipe", ["nvidia", "4over6"])
@pytest.mark.parametrize("rows", [1, 13, 100])
def test_ragged_rows_of_a_layer(rows, recipe):
    """A layer on a row count that is no multiple of 32, starting at an address that is no multiple of 16: outputs and both
    gradients are those of the rows padded with zeros."""
    recipe = backend.FP4_RECIPES[recipe]
    gen = torch.Generator(device="cuda").manual_seed(rows)
    w = bl.LatticeTensor.from_float(torch.randn(96, 64, device="cuda", generator=gen) * 0.02, "nvfp4", dtype=torch.bfloat16)

    def shifted(cols):
        return torch.randn(rows * cols + 1, device="cuda", generator=gen).to(torch.bfloat16)[1:].view(rows, cols)
    x, gy = shifted(64), shifted(96)
    outs = []
    for pad in (0, -rows % 32):
        backend.set_sr_seed(5)
        xi, gi = (torch.nn.functional.pad(t, (0, 0, 0, pad)) if pad else t for t in (x, gy))
        y, xt = backend.fp4_forward_saving(xi, w, None, recipe)
        gx, gw = backend.fp4_backward(gi, w, xt, True, True, recipe)
        outs.append((y[:rows], gx[:rows], gw, backend.nvfp4_linear(xi, w, None, recipe)[:rows]))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("recipe", ["fp4_all", "4over6", "quartet2"])
def test_outputs_and_draws_do_not_depend_on_grad_mode(recipe):
    """A forward pass under no_grad makes no operand for the weight gradient: same outputs, single and shared input, and
    the counter of the rounding seeds moves as it does with gradients."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    ps = [torch.nn.Parameter(bl.LatticeTensor.from_float(torch.randn(n, 128, device="cuda", generator=gen) * 0.02, "nvfp4",
                                                         dtype=torch.bfloat16)) for n in (128, 256)]
    x = torch.randn(45, 128, device="cuda", generator=gen).to(torch.bfloat16)
    seen = []
    for grad in (True, False):
        backend.set_sr_seed(3)
        backend.clear_shared()
        with torch.set_grad_enabled(grad), bl.compute(recipe):
            ys = (torch.nn.functional.linear(x, ps[0]), *bl.parallel.shared_input_linears(x, ps))
        assert all(y.requires_grad == grad for y in ys)
        seen.append((*[y.detach() for y in ys], torch.tensor(backend._seed())))
    for a, b in zip(*seen):
        assert torch.equal(a, b)


@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 48), (16, 4096), (129, 80), (1, 262144), (64, 4096), (257, 1024), (64, 4112)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("seed", [-1, 9])
def test_amax_quantize_small_and_separate(rows, cols, dtype, seed):
    """Maximum and quantization in one launch (up to 262144 values, and just above) against the two operators: codes, every
    scale byte of the tiles, padding included, and the four results of the maximum but its counter."""
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda", generator=gen) * 3).to(dtype)
    x[-1, -1] = 40.0
    if rows > 100:
        x[0] = 0.0
    am = _ops.amax_global(x)
    for blocked in (True, False):
        codes, scales = _ops.quantize_nvfp4(x, am[1:2], seed, 2, blocked=blocked)
        torch.full((1 << 20,), 0x7F, dtype=torch.uint8, device="cuda")             # stale bytes for the next allocations
        c, s, a = _ops.amax_quantize_nvfp4(x, seed, 2, blocked=blocked)
        assert torch.equal(c, codes) and torch.equal(s.view(torch.uint8), scales.view(torch.uint8))
        assert torch.equal(a[[0, 1, 3]], am[[0, 1, 3]])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [1, 7, 4099, 148 * 4 * 256 * 8 * 8 + 5, (1 << 27) + 9])
def test_amax_finds_every_position(n, dtype):
    """The maximum at the first, a middle and the last element (whole rounds of loads, the last partial round, the ragged
    tail, the grid of large tensors), a NaN ignored as before, an infinity found."""
    x = torch.full((n,), -0.5, dtype=dtype, device="cuda")
    for at in sorted({0, n // 2, max(0, n - 9), n - 1}):
        x[at] = -3.0
        assert _ops.amax_global(x)[0].item() == 3.0
        x[at] = -0.5
    x[n // 3] = float("nan")
    assert _ops.amax_global(x)[0].item() == (0.5 if n > 1 else 0.0)
    x[n // 3] = float("inf")
    assert _ops.amax_global(x)[0].item() == float("inf")


def test_host_calls_keep_their_integers_and_errors():
    """Seeds and steps of any integer-like type, taken modulo 2^64; refusals as Python exceptions of the usual types."""
    x = torch.randn(16, 64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    want = _ops.amax_quantize_nvfp4(x, 7, 3)
    for seed, step in ((np.int64(7), np.int32(3)), (7.0, 3.0), (torch.tensor(7), True + 2), (7 + (1 << 64), 3 + (5 << 32)), (7, 3 - (1 << 32))):
        for a, b in zip(_ops.amax_quantize_nvfp4(x, seed, step), want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    for pad_rows in (0, -32):
        with pytest.raises(RuntimeError, match="pad_rows"):
            _ops.quantize_nvfp4_t(x, None, pad_rows=pad_rows)
    packed, scales, am = want
    torch.cuda.set_per_process_memory_fraction(0.5)          # (the allocator refuses before it asks the device)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            _ops.dequantize(packed, scales, am[1:2], None, "nvfp4", 1 << 22, 1 << 22)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def _special_values(shape, dtype, rng):
    """Normal values, 1 % NaN of either sign and 1 % infinities, and blocks of 16 of nothing but NaN along either side."""
    v = rng.standard_normal(shape).astype(np.float32)
    at = rng.random(shape)
    v[at < 0.01] = np.nan
    v[at < 0.005] = -np.nan
    v[at > 0.99] = np.inf
    v[at > 0.995] = -np.inf
    v[3, 32:48] = np.nan
    v[64:80, 5] = np.nan
    return torch.from_numpy(v).to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_stochastic_rounding_of_nan_and_infinity(dtype):
    """A NaN takes the largest level and is ignored by every maximum, whatever its neighbours draw; an infinity is the
    largest level of its sign, or a NaN where the scale of its block is infinite as well. Rows, transposed with an even and
    an odd number of columns and rotated, and the one-launch form for small inputs."""
    rng = np.random.default_rng(19)
    x = _special_values((512, 512), dtype, rng)
    xf = x.float().numpy()
    for g in (0.0011, 0.11):
        rc, rs, _ = oracle.quantize_rows(xf, g, "sr", seed=11)
        packed, sc = _ops.quantize_nvfp4(x.cuda(), dev(np.array([g], np.float32)), seed=11)
        assert np.array_equal(host(packed), rc) and np.array_equal(host(sc), rs)
    H = oracle.hadamard16()
    for cols, h in ((512, None), (511, None), (512, H)):
        part = x[:, :cols].contiguous()
        rc, rs = oracle.quantize_t(part.float().numpy(), h, oracle.global_from_bound(0.02), "sr", seed=5)
        packed, sc, _ = _ops.quantize_nvfp4_t(part.cuda(), dev(h.astype(np.float32)) if h is not None else None, 5, 0,
                                              dev(np.array([0.02], np.float32)))
        assert np.array_equal(host(packed), rc) and np.array_equal(host(sc), rs)
    for part in (x[:40], x[:40].nan_to_num(posinf=1.0, neginf=-1.0, nan=float("nan"))):
        rc, rs, rg = oracle.quantize_rows(part.float().numpy(), None, "sr", seed=3)
        packed, sc, am = _ops.amax_quantize_nvfp4(part.cuda(), 3)
        assert am[1].item() == rg and np.array_equal(host(packed), rc) and np.array_equal(host(sc), rs)


@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("transpose", [False, True])
def test_general_stochastic_rounding_of_nan(rotate, transpose):
    """The general quantizer: NaN takes the largest level, and what shares no block (rotated: no segment of 128) with one
    keeps its code."""
    x = torch.randn(256, 256, generator=torch.Generator().manual_seed(2)).cuda()
    bad = x.clone()
    bad[7, 20] = bad[200, 131] = float("nan")
    given = torch.tensor([0.002], device="cuda")
    kw = dict(transpose=transpose, mode="sr", rotate=rotate, seed=4, rotate_seed=9 if rotate else -1, given=given)
    clean, dirty = (host(_ops.nvfp4_quantize_general(v, **kw)[0]) for v in (x, bad))
    clean, dirty = (np.stack([c & 15, c >> 4], -1).reshape(256, 256) for c in (clean, dirty))
    span = 128 if rotate else 16
    for r, c in ((20, 7), (131, 200)) if transpose else ((7, 20), (200, 131)):
        hit = dirty[r, c // span * span:][:span] if rotate else dirty[r, c:c + 1]
        assert (hit == 7).all()
        lo = c // span * span
        dirty[r, lo:lo + span] = clean[r, lo:lo + span]
    assert np.array_equal(clean, dirty)


@pytest.mark.parametrize("slice_", [0, 21, 42, 63])
def test_division_on_every_significand(slice_):
    """The packed division on all dividends by 2^17 divisors; the 64 slices together are all 2^46 pairs of significands (run
    in full when the routine changes: a minute on a B200)."""
    import ctypes
    bad = ctypes.c_uint64(1)
    _C.call("bl_selftest_division_slice", slice_, ctypes.byref(bad), 0)
    assert bad.value == 0


@pytest.mark.parametrize("g", [1e-38, 1e-30, 1e-20, 9.9e-13, 1e-12, 2.5e27, 1e37])
def test_block_scales_of_extreme_tensors(g):
    """Block maxima from a zero and 2^80 below the tensor's up to it, against per-tensor scales on both sides of the range in
    which the scales' divisions go by a shared reciprocal; rows and transposed, both roundings."""
    rng = np.random.default_rng(31)
    x = rng.standard_normal((256, 256)) * 2.0 ** rng.uniform(-80, 3, (16, 1, 16, 1)).repeat(16, 1).repeat(16, 3).reshape(256, 256) * 400.0
    x = np.clip(x * g, -3e38, 3e38).astype(np.float32)
    x[16:32, 32:48] = 0.0
    gd = dev(np.array([g], np.float32))
    for mode, seed in (("rtn", -1), ("sr", 11)):
        rc, rs, _ = oracle.quantize_rows(x, np.float32(g), mode, seed=max(seed, 0))
        packed, sc = _ops.quantize_nvfp4(dev(x), gd, seed=seed)
        assert np.array_equal(host(sc), rs) and np.array_equal(host(packed), rc)
        bound = min(np.float32(g), np.float32(1e35))
        rc, rs = oracle.quantize_t(x, None, oracle.global_from_bound(float(bound)), mode, seed=max(seed, 0))
        packed, sc, _ = _ops.quantize_nvfp4_t(dev(x), None, seed, 0, dev(np.array([bound], np.float32)))
        assert np.array_equal(host(sc), rs) and np.array_equal(host(packed), rc)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_gates_at_the_ends_of_the_shared_reciprocal(dtype):
    """Finite gates from -87 up share a warp with nothing else, so that every one of them takes the shared reciprocal; then the
    same with one gate beyond in every thousand."""
    bits = torch.arange(1 << 16, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    g = bits[(bits.float() >= -87.0) & bits.float().isfinite()]
    g = torch.cat([g, g[: -g.numel() % 256]])
    gen = torch.Generator(device="cuda").manual_seed(4)
    u, da = (torch.randn(g.numel(), device="cuda", generator=gen).to(dtype) for _ in range(2))
    mixed = g.clone()
    mixed[::1000] = torch.tensor([-87.5, -88.0, -100.0, float("inf"), float("-inf"), float("nan")], device="cuda").to(dtype).repeat(g.numel())[: mixed[::1000].numel()]
    for gate in (g, mixed):
        gf, uf, df = gate.float(), u.float(), da.float()
        d = 1.0 + torch.exp(-gf)
        silu, sig = (gf / d).to(dtype).float(), 1.0 / d
        want = ((silu * uf).to(dtype), ((df * uf).to(dtype).float() * sig * (1.0 + gf * (1.0 - sig))).to(dtype), (df * silu).to(dtype))
        for a, b in zip((_ops.swiglu_fwd(gate, u), *_ops.swiglu_bwd(gate, u, da)), want):
            nan = b.isnan()
            assert torch.equal(a.isnan(), nan) and torch.equal(a.view(torch.int16)[~nan], b.view(torch.int16)[~nan])
