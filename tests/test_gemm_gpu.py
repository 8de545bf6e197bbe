"""GPU parity of the fixed-point GEMM.

* CUDA-core route: bit-exact against the CPU oracle (same ascending-k order).
* tensor-core route: integer stage bit-exact given the kernel's own fp32
  partials; end to end within a few Q-format LSB of the oracle (different
  in-tile summation order); bitwise invariant to split-K, batch size, K-tile
  order and repeats.
* the reference's own tests (fxpr_vllm/_tests/test_gemm.py) re-stated.
"""
from __future__ import annotations

import pytest
import torch

import fxpr_vllm  # noqa: F401
from fxpr_vllm import _lib as L
from oracle import fxp_oracle as orc

pytestmark = pytest.mark.gpu

_TOL = {torch.float32: (5e-4, 5e-4), torch.float16: (1e-2, 1e-2), torch.bfloat16: (5e-2, 5e-2)}
_DTYPES = [torch.float32, torch.float16, torch.bfloat16]


def _gemm(a, b, bias=None, int_bits=32, frac_bits=16):
    return torch.ops.fxpr.gemm_fxp(a, b, bias, int_bits, frac_bits)


def _rand(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype)


# ---------------- CUDA-core route: bit-exact vs oracle -----------------------------

@pytest.mark.parametrize("dtype", _DTYPES)
@pytest.mark.parametrize("M,N,K", [(1, 1, 32), (3, 7, 16), (4, 4, 33), (130, 130, 33), (65, 200, 300)])
@pytest.mark.parametrize("int_bits", [16, 32, 64])
def test_portable_bit_exact(dtype, M, N, K, int_bits):
    a = _rand((M, K), dtype, 1, 0.5)
    b = _rand((K, N), dtype, 2, 0.5)
    bias = _rand((N,), dtype, 3)
    with L.overrides(gemm_portable=True):
        got = _gemm(a.cuda(), b.cuda(), bias.cuda(), int_bits, 16).cpu()
        got_int = torch.ops.fxpr.gemm_fxp_int(a.cuda(), b.cuda(), int_bits, 16).cpu()
    exp_int = orc.gemm_fxp(a, b, None, int_bits, 16, sequential=True, return_int=True)
    assert torch.equal(got_int.to(torch.int64), exp_int)
    exp = orc.gemm_epilogue(exp_int, bias, dtype, 16)
    assert torch.equal(got.view(torch.uint8), exp.view(torch.uint8))


@pytest.mark.parametrize("M,N,K,kt", [
    (1, 64, 17, 128), (16, 65, 300, 16), (17, 63, 129, 128), (64, 200, 520, 24), (65, 130, 260, 64), (129, 9600, 40, 64),
    (1, 132, 1025, 128), (8, 128, 600, 48), (9, 260, 2100, 64), (16, 4, 300, 16), (33, 200, 530, 64),
])
@pytest.mark.parametrize("transposed", [False, True])
def test_portable_kernel_at_tile_edges(M, N, K, kt, transposed):
    """Row tiles of 16, 64 and 128, K-tiles dealt to 1 to 8 cluster ranks, ragged chunks, both stride orders."""
    a = _rand((M, K), torch.float32, M, 0.5)
    b = _rand((K, N), torch.float32, N, 0.5)
    ga, gb = (a.t().contiguous().cuda().t(), b.t().contiguous().cuda().t()) if transposed else (a.cuda(), b.cuda())
    with L.overrides(gemm_portable=True, gemm_k_tile=kt):
        got = torch.ops.fxpr.gemm_fxp_int(ga, gb, 64, 16).cpu()
    exp = orc.gemm_fxp(a, b, None, 64, 16, sequential=True, return_int=True, k_tile=kt)
    assert torch.equal(got.to(torch.int64), exp)


def test_portable_strided_operands():
    a = _rand((40, 96), torch.float32, 4)
    w = _rand((24, 96), torch.float32, 5)  # (N, K) weight viewed as (K, N)
    with L.overrides(gemm_portable=True):
        got = _gemm(a.cuda()[::2], w.cuda().t(), None, 64, 16).cpu()
    exp = orc.gemm_fxp(a[::2], w.t(), None, 64, 16, sequential=True)
    assert torch.equal(got, exp)


# ---------------- default route: tolerance + invariance (all dtypes) ----------------

@pytest.mark.parametrize("dtype", _DTYPES)
@pytest.mark.parametrize("M,N,K", [(8, 16, 32), (4, 4, 64), (130, 130, 33), (256, 256, 256),
                                   (100, 384, 512), (300, 264, 1096)])
@pytest.mark.parametrize("use_bias", [False, True])
def test_matches_float_matmul(dtype, M, N, K, use_bias):
    a = _rand((M, K), dtype, 11, 0.5).cuda()
    b = _rand((K, N), dtype, 12, 0.5).cuda()
    bias = _rand((N,), dtype, 13).cuda() if use_bias else None
    got = _gemm(a, b, bias)
    assert got.dtype == dtype and got.shape == (M, N)
    ref = a.float() @ b.float()
    if use_bias:
        ref = ref + bias.float()
    atol, rtol = _TOL[dtype]
    assert torch.allclose(got.float(), ref.to(dtype).float(), atol=atol * max(1.0, K / 64) ** 0.5,
                          rtol=rtol)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,kt", [(128, 256, 512, 64), (200, 320, 1024, 128), (64, 4096, 1024, 64)])
def test_int_accumulators_close_to_oracle(dtype, M, N, K, kt):
    a = _rand((M, K), dtype, 21).cuda()
    b = _rand((K, N), dtype, 22, 0.05).cuda()
    with L.overrides(gemm_k_tile=kt, gemm_split_k=1):
        got = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16).cpu()
    exp = orc.gemm_fxp(a.cpu(), b.cpu(), None, 64, 16, k_tile=kt, return_int=True)
    # each K-tile's partial can differ in its last fp32 ulp -> at most one LSB per tile
    assert (got - exp).abs().max().item() <= K // kt
    assert (got - exp).abs().float().mean().item() < 0.25


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("int_bits", [32, 64])
def test_integer_stage_exact_given_kernel_partials(dtype, int_bits):
    M, N, K, kt = 150, 264, 640, 64
    a = _rand((M, K), dtype, 31, 2.0).cuda()
    b = _rand((K, N), dtype, 32, 2.0).cuda()
    a[0, :] = 3000.0  # rows that saturate a Q16.16/int32 tile and wrap the sum
    b[:, 0] = 3000.0
    with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_partials=True) as o:
        got = torch.ops.fxpr.gemm_fxp_int(a, b, int_bits, 16).cpu()
        partials = o.last_partials.cpu()
    exp = orc.gemm_int_from_partials(partials, int_bits, 16)
    assert torch.equal(got.to(torch.int64), exp)


@pytest.mark.parametrize("dtype", _DTYPES)
def test_deterministic_across_runs(dtype):
    a = _rand((200, 512), dtype, 41).cuda()
    b = _rand((512, 136), dtype, 42).cuda()
    first = _gemm(a, b)
    for _ in range(4):
        assert torch.equal(first, _gemm(a, b))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(64, 512, 2048), (300, 264, 1096), (1, 128, 4096)])
@pytest.mark.parametrize("kt", [64, 128])
def test_split_k_invariance(dtype, M, N, K, kt):
    a = _rand((M, K), dtype, 51).cuda()
    b = _rand((K, N), dtype, 52, 0.05).cuda()
    bias = _rand((N,), dtype, 53).cuda()
    outs = []
    for split in (1, 2, 4, 8, 16):
        with L.overrides(gemm_k_tile=kt, gemm_split_k=split):
            outs.append((_gemm(a, b, bias, 64, 16), torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)))
    for c, ci in outs[1:]:
        assert torch.equal(c, outs[0][0]) and torch.equal(ci, outs[0][1])
    # scratch is left clean: a second sweep gives the same bits
    with L.overrides(gemm_k_tile=kt, gemm_split_k=4):
        assert torch.equal(_gemm(a, b, bias, 64, 16), outs[0][0])


@pytest.mark.parametrize("dtype", _DTYPES)
def test_ktile_permutation_invariance(dtype):
    kt = L.BLOCK_K_BY_DTYPE[dtype]
    M, K, N = 4, kt * 4, 8
    a = _rand((M, K), dtype, 61).cuda()
    b = _rand((K, N), dtype, 62).cuda()
    tperm = torch.randperm(4)
    perm = torch.cat([torch.arange(t * kt, (t + 1) * kt) for t in tperm]).cuda()
    assert torch.equal(_gemm(a, b), _gemm(a[:, perm].contiguous(), b[perm].contiguous()))


@pytest.mark.parametrize("dtype", _DTYPES)
@pytest.mark.parametrize("K,N", [(64, 16), (512, 264)])
def test_batch_size_invariance(dtype, K, N):
    a_full = _rand((300, K), dtype, 71).cuda()
    b = _rand((K, N), dtype, 72).cuda()
    rows = [0, 3, 17, 64, 127, 299]
    refs = {m: _gemm(a_full[m:m + 1], b)[0] for m in rows}
    for batch in (1, 4, 16, 128, 300):
        out = _gemm(a_full[:batch], b)
        for m in rows:
            if m < batch:
                assert torch.equal(out[m], refs[m]), f"row {m} differs at batch={batch}"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_tensor_core_route_agrees_with_cuda_core_route(dtype):
    a = _rand((96, 512), dtype, 81).cuda()
    b = _rand((512, 128), dtype, 82, 0.1).cuda()
    tc = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
    with L.overrides(gemm_portable=True):
        cc = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
    assert (tc - cc).abs().max().item() <= 512 // L.BLOCK_K_BY_DTYPE[dtype]


def test_identity_zero_and_empty():
    a = _rand((4, 16), torch.float32, 91).cuda()
    assert torch.allclose(_gemm(a, torch.eye(16, device="cuda")), a, atol=1e-4)
    z = _gemm(torch.ones((4, 16), device="cuda"), torch.zeros((16, 4), device="cuda"))
    assert torch.equal(z, torch.zeros((4, 4), device="cuda"))
    e = _gemm(torch.empty((0, 16), device="cuda"), torch.zeros((16, 4), device="cuda"))
    assert e.shape == (0, 4)
    with pytest.raises(ValueError):
        _gemm(a, torch.eye(16, device="cuda"), None, 24, 16)


def test_epilogue_from_int_matches_oracle():
    g = torch.Generator().manual_seed(5)
    ci = torch.randint(-(2**40), 2**40, (37, 53), generator=g, dtype=torch.int64)
    bias = torch.randn(53, generator=g).to(torch.bfloat16)
    got = torch.ops.fxpr.gemm_fxp_epilogue(ci.cuda(), bias.cuda(), torch.bfloat16, 16).cpu()
    exp = orc.gemm_epilogue(ci, bias, torch.bfloat16, 16)
    assert torch.equal(got.view(torch.uint8), exp.view(torch.uint8))


def test_tp_sharding_single_gpu_equals_unsharded():
    # row-parallel layer: K sharded over "ranks", integer accumulators summed
    a = _rand((64, 4096), torch.bfloat16, 95).cuda()
    b = _rand((4096, 512), torch.bfloat16, 96, 0.02).cuda()
    full = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
    for tp in (2, 4, 8):
        ks = 4096 // tp
        acc = torch.zeros_like(full)
        for r in range(tp):
            acc += torch.ops.fxpr.gemm_fxp_int(a[:, r * ks:(r + 1) * ks], b[r * ks:(r + 1) * ks], 64, 16)
        assert torch.equal(acc, full)
    out = torch.ops.fxpr.gemm_fxp_epilogue(full, None, torch.bfloat16, 16)
    assert torch.equal(out, _gemm(a, b, None, 64, 16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("int_bits", [32, 64])
@pytest.mark.parametrize("tile,kt,split", [("n128", 64, 1), ("n128", 128, 1), ("n128", 64, 3), ("n128", 128, 2),
                                           ("pair", 64, 1), ("pair", 128, 1)])
def test_fast_epilogue_equals_plain_conversion_with_outliers(dtype, int_bits, tile, kt, split):
    """The magic-number epilogue with its exact fix-up gives the same integers as the
    tensor-core kernel that converts every partial with cvt.rni (saturating), including
    rows whose partials leave the fast range, saturate int32 or overflow the 32-bit sum."""
    from fxpr_vllm import _native as nat

    M, N, K = 300, 520, 1096
    a = _rand((M, K), dtype, 101).cuda()
    b = _rand((K, N), dtype, 102, 0.05).cuda()
    a[3, :] = 900.0
    a[M - 1, 5::7] = -3000.0
    a[M // 2, :64] = 6.0e4
    a[7, 100] = float("inf") if int_bits == 32 else 5.0e4
    # both tile shapes, whatever the default: 128 x 128, and 256 x 256 on SM pairs (unsplit K only)
    shape_flag = {"n128": nat.GEMM_TILE_N128, "pair": nat.GEMM_PAIR}[tile]
    with L.overrides(gemm_k_tile=kt, gemm_split_k=split, gemm_flags=shape_flag):
        fast_i = torch.ops.fxpr.gemm_fxp_int(a, b, int_bits, 16)
        fast_c = _gemm(a, b, None, int_bits, 16)
    with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
        exact_i = torch.ops.fxpr.gemm_fxp_int(a, b, int_bits, 16)
        exact_c = _gemm(a, b, None, int_bits, 16)
    assert torch.equal(fast_i, exact_i)
    assert torch.equal(fast_c.view(torch.int16), exact_c.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("int_bits,frac", [(16, 8), (64, 32), (32, 8)])
def test_tensor_core_route_other_q_formats(int_bits, frac):
    a = _rand((130, 512), torch.bfloat16, 111, 0.3).cuda()
    b = _rand((512, 264), torch.bfloat16, 112, 0.1).cuda()
    got = torch.ops.fxpr.gemm_fxp_int(a, b, int_bits, frac).cpu().to(torch.int64)
    exp = orc.gemm_fxp(a.cpu(), b.cpu(), None, int_bits, frac, return_int=True)
    tol = 4 if frac <= 16 else 4 * 2 ** (frac - 16)
    assert (got - exp).abs().max().item() <= tol


def test_b_given_as_transposed_weight_view():
    # weight kept (N, K) and passed as .t(): the K-major operand path, no transpose copy
    a = _rand((200, 1024), torch.bfloat16, 121).cuda()
    w = _rand((384, 1024), torch.bfloat16, 122, 0.05).cuda()
    v1 = torch.ops.fxpr.gemm_fxp_int(a, w.t(), 64, 16)
    v2 = torch.ops.fxpr.gemm_fxp_int(a, w.t().contiguous(), 64, 16)
    assert torch.equal(v1, v2)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 16, 33, 64])
@pytest.mark.parametrize("kt,split", [(64, 1), (128, 1), (64, 3), (128, 4), (64, 8), (128, 2), (64, 2)])
@pytest.mark.parametrize("int_bits", [32, 64])
def test_decode_shape_kernel_equals_wide_tile_kernel(dtype, M, kt, split, int_bits):
    """M <= 64 goes to the kernel that puts the weights on the 128-row side of the MMA.  Its
    integers and outputs must be those of the 128-row-tile kernel (and hence do not depend on
    how many rows share the launch), for both weight layouts, with bias, a ragged N and K,
    split-K and partials outside the fast conversion's range."""
    from fxpr_vllm import _native as nat

    N, K = 520, 1096
    a = _rand((M, K), dtype, 201).cuda()
    b = _rand((K, N), dtype, 202, 0.05).cuda()
    bias = _rand((N,), dtype, 203).cuda()
    a[0, 5::7] = -3000.0
    a[M - 1, :64] = 6.0e4
    bt_view = b.t().contiguous().t()               # (K, N) view of an (N, K) row-major matrix
    for bb in (b, bt_view):
        with L.overrides(gemm_k_tile=kt, gemm_split_k=split):
            sk_i = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
            sk_c = _gemm(a, bb, bias, int_bits, 16)
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_NO_SKINNY):
            wide_i = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
            wide_c = _gemm(a, bb, bias, int_bits, 16)
        assert torch.equal(sk_i, wide_i)
        assert torch.equal(sk_c.view(torch.int16), wide_c.view(torch.int16))
        if split > 1:      # 2/4/8 splits merge inside a cluster by default; the scratch-plane merge must agree
            with L.overrides(gemm_k_tile=kt, gemm_split_k=split, gemm_flags=nat.GEMM_NO_CLUSTER):
                pl_i = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
            assert torch.equal(pl_i, wide_i)
    L.check_device_status()


@pytest.mark.parametrize("M", [3, 16, 17, 32, 63])
@pytest.mark.parametrize("kt,split", [(64, 1), (128, 1), (64, 4), (128, 8), (64, 3), (128, 5)])
def test_decode_shape_row_tiles(M, kt, split):
    """Row tiles of 16, 32 and 64 at their edges, with more stages of K than the ring holds and, in the
    cluster merge, ranks with fewer rows than the others or none: the integers of the wide kernel."""
    from fxpr_vllm import _native as nat

    N, K = 392, 4168
    a = _rand((M, K), torch.bfloat16, 221).cuda()
    b = _rand((K, N), torch.bfloat16, 222, 0.05).cuda()
    a[M - 1, 700:764] = 3.0e4                      # one K-tile beyond the fast conversion's range
    with L.overrides(gemm_k_tile=kt, gemm_split_k=split):
        got = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
        best = L.gemm_fxp_argmax(a, b, None, 64, 16) if split == 1 else None
    with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_NO_SKINNY):
        want = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
        want_c = torch.ops.fxpr.gemm_fxp(a, b, None, 64, 16)
    assert torch.equal(got, want)
    if best is not None:
        assert torch.equal(best[0].view(torch.int16), want_c.view(torch.int16))
        assert torch.equal(L.argmax_from_keys(best[1]), want_c.argmax(dim=-1))
    L.check_device_status()


def test_decode_row_bits_do_not_depend_on_the_batch():
    """Row r of a 64-row launch (decode-shape kernel) equals row r of a 300-row launch."""
    a = _rand((300, 1024), torch.bfloat16, 211).cuda()
    b = _rand((1024, 384), torch.bfloat16, 212, 0.05).cuda()
    big = _gemm(a, b, None, 64, 16)
    small = _gemm(a[100:164].contiguous(), b, None, 64, 16)
    assert torch.equal(small.view(torch.int16), big[100:164].view(torch.int16))


def test_routes_agree_on_random_shapes():
    """Seeded sweep over ragged shapes: whichever kernel the dispatcher picks (decode-shape,
    128x128 tiles or 256x256 on SM pairs, cluster or plane split-K) must give the integers of the
    tensor-core kernel with plain cvt.rni conversion, for both weight layouts."""
    from fxpr_vllm import _native as nat

    g = torch.Generator().manual_seed(2024)
    for case in range(40):
        M = int(torch.randint(1, 400, (1,), generator=g))
        if case % 3 == 0:
            M = int(torch.randint(1, 65, (1,), generator=g))
        N = 8 * int(torch.randint(8, 130, (1,), generator=g))
        K = 8 * int(torch.randint(8, 300, (1,), generator=g))
        kt = (64, 128)[case % 2]
        split = (1, 2, 3, 4, 8)[case % 5]
        int_bits = (64, 32)[(case // 2) % 2]
        dtype = (torch.bfloat16, torch.float16)[(case // 4) % 2]
        a = _rand((M, K), dtype, 1000 + case).cuda()
        b = _rand((K, N), dtype, 2000 + case, 0.05).cuda()
        if case % 7 == 0:
            a[M // 2, : min(64, K)] = 3.0e4
        bb = b if case % 2 else b.t().contiguous().t()
        with L.overrides(gemm_k_tile=kt, gemm_split_k=split):
            got = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
            exp = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
        assert torch.equal(got, exp), (case, M, N, K, kt, split, int_bits, dtype)
    L.check_device_status()


def _kernels_launched(fn):
    """Names of the CUDA kernels ``fn`` launches; empty where the profiler cannot see them."""
    from torch.profiler import ProfilerActivity, profile

    fn()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.key for e in prof.key_averages()]


@pytest.mark.parametrize("M,N,K,split,flag,want", [
    (129, 128, 64, 1, "pair", "gemm_tc_pair_kernel"),           # the smallest call the two-SM kernel takes
    (128, 512, 256, 1, "pair", "gemm_tc_fast_kernel"),          # one row, column or K-tile split short of it
    (300, 120, 256, 1, "pair", "gemm_tc_fast_kernel"),
    (300, 512, 512, 2, "pair", "gemm_tc_fast_kernel"),
    (4096, 4096, 256, 0, "", "gemm_tc_pair_kernel"),            # by size
    (4096, 4096, 256, 0, "n128", "gemm_tc_fast_kernel"),
])
def test_which_kernel_takes_a_call(M, N, K, split, flag, want):
    """What the flags and the dispatch rule say about the wide kernels, seen in the launches: the comparisons
    below prove nothing if both of their sides run the same kernel."""
    from fxpr_vllm import _native as nat

    a, b = _rand((M, K), torch.bfloat16, 1).cuda(), _rand((K, N), torch.bfloat16, 2, 0.05).cuda()
    flags = {"pair": nat.GEMM_PAIR, "n128": nat.GEMM_TILE_N128, "": 0}[flag]
    kw = {"gemm_split_k": split} if split else {}
    with L.overrides(gemm_flags=flags, **kw):
        names = [n for n in _kernels_launched(lambda: _gemm(a, b, None, 64, 16)) if "gemm" in n]
    if not names:
        pytest.skip("no kernel activity from the profiler")
    assert any(want in n for n in names), names


def test_two_sm_kernel_agrees_on_random_shapes():
    """The cta_group::2 kernel (CTA pairs, 256-row tiles, unsplit K) gives the integers and outputs of the
    plain-conversion tensor-core kernel on ragged shapes: every mix of K-tile, accumulator width, io dtype,
    layout of B and bias, each with N a multiple of 16 (wide stores) and not."""
    from fxpr_vllm import _native as nat

    g = torch.Generator().manual_seed(77)
    for case in range(64):
        M = int(torch.randint(129, 900, (1,), generator=g))
        N = 16 * int(torch.randint(8, 65, (1,), generator=g)) + 8 * ((case // 32) % 2)
        K = 8 * int(torch.randint(8, 300, (1,), generator=g))
        kt = (64, 128)[case % 2]
        int_bits = (64, 32)[(case // 2) % 2]
        dtype = (torch.bfloat16, torch.float16)[(case // 4) % 2]
        a = _rand((M, K), dtype, 3000 + case).cuda()
        b = _rand((K, N), dtype, 4000 + case, 0.05).cuda()
        if case % 5 == 0:
            a[M // 2, : min(64, K)] = 3.0e4
        bb = b if (case // 8) % 2 else b.t().contiguous().t()
        bias = _rand((N,), dtype, 5000 + case).cuda() if (case // 16) % 2 else None
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_PAIR):
            got = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
            got_c = _gemm(a, bb, bias, int_bits, 16)
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
            exp = torch.ops.fxpr.gemm_fxp_int(a, bb, int_bits, 16)
            exp_c = _gemm(a, bb, bias, int_bits, 16)
        assert torch.equal(got, exp), (case, M, N, K, kt, int_bits, dtype)
        assert torch.equal(got_c.view(torch.int16), exp_c.view(torch.int16)), case
    L.check_device_status()


@pytest.mark.parametrize("M,N,K", [
    (256, 256, 128), (255, 248, 136), (257, 264, 64), (512, 512, 72), (129, 128, 64), (1025, 2056, 200),
])
@pytest.mark.parametrize("kt", [64, 128])
@pytest.mark.parametrize("kmajor", [False, True])
def test_two_sm_kernel_at_tile_edges(M, N, K, kt, kmajor):
    """256 x 256 pair tiles one short of, at and one past their edges, and the smallest the kernel takes; K of
    one, several and ragged tiles; both layouts of B; with and without bias (whose sums need not fit the
    shortcut of the wide stores)."""
    from fxpr_vllm import _native as nat

    a = _rand((M, K), torch.bfloat16, M).cuda()
    b = _rand((K, N), torch.bfloat16, N, 0.05).cuda()
    if kmajor:
        b = b.t().contiguous().t()
    bias = _rand((N,), torch.bfloat16, 7, 30.0).cuda()
    clean = a.clone()
    a[M - 1, -1] = 2.0e4                              # a partial of the last row leaves the fast range
    out = []
    for flags in (nat.GEMM_PAIR, nat.GEMM_FORCE_EXACT_TC):
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=flags):
            out.append((torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16), _gemm(a, b, None, 32, 16), _gemm(a, b, bias, 64, 16),
                        _gemm(clean, b, None, 64, 16), _gemm(clean, b, bias, 32, 16)))
    assert torch.equal(out[0][0], out[1][0])
    for got, exp in zip(out[0][1:], out[1][1:]):
        assert torch.equal(got.view(torch.int16), exp.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M,N,K,kt", [(33, 38008, 64, 64), (64, 38008, 136, 64), (64, 38016, 136, 128), (48, 76040, 712, 64),
                                      (64, 113672, 392, 128), (63, 38008, 1096, 128), (64, 38008, 3080, 64), (40, 57096, 3072, 128)])
def test_decode_shape_walk_over_large_vocabularies(M, N, K, kt):
    """More than 32 rows on more column tiles than CTAs fit the GPU: a CTA walks from tile to tile with its ring, its
    accumulators and its sums, K shorter and longer than the ring, ragged last tiles, and partials beyond the fast range
    (64-bit sums) in some tiles only, one after the other or not: the wide kernel's integers, outputs and arg-max keys."""
    from fxpr_vllm import _native as nat

    a = _rand((M, K), torch.bfloat16, 41).cuda()
    b = _rand((K, N), torch.bfloat16, 42, 0.05).cuda()
    for first in (300, 128 * 296 + 5, N - 1):                     # a CTA's first, second and last tile
        b[:, first] = 3.0e4
    bias = _rand((N,), torch.bfloat16, 43).cuda()
    with L.overrides(gemm_k_tile=kt):
        got = [torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16) for bits in (32, 64)]
        got_c = [_gemm(a, b, x, 64, 16) for x in (None, bias)]
        c, keys = L.gemm_fxp_argmax(a, b, None, 64, 16)
        act = L.gemm_silu_mul(a, b, 64, 16)
    with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_NO_SKINNY):
        for bits, x in zip((32, 64), got):
            assert torch.equal(x, torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16))
        for x, y in zip((None, bias), got_c):
            assert torch.equal(y.view(torch.int16), _gemm(a, b, x, 64, 16).view(torch.int16))
    assert torch.equal(c.view(torch.int16), got_c[0].view(torch.int16))
    assert torch.equal(L.argmax_from_keys(keys), got_c[0].argmax(dim=-1))
    assert torch.equal(act.view(torch.int16), L.silu_mul_pairs(got_c[0]).view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M", [1, 16])
@pytest.mark.parametrize("N,K,split,pad", [(1096, 4168, 0, 0), (392, 4168, 8, 0), (1800, 6000, 4, 0), (264, 520, 1, 8), (2008, 3080, 8, 0)])
@pytest.mark.parametrize("kmajor", [False, True])
def test_decode_shape_weights_off_the_sectors(M, N, K, split, pad, kmajor):
    """Up to 16 rows and weights whose rows start inside a 32-byte sector (by their stride, or by their first address):
    the whole-SM ring, with and without clusters, gives the wide kernel's integers and outputs."""
    from fxpr_vllm import _native as nat

    a = _rand((M, K), torch.bfloat16, 31).cuda()
    rows, cols = (N, K) if kmajor else (K, N)
    store = _rand((rows, cols + 2 * pad), torch.bfloat16, 32, 0.05).cuda()
    b = store[:, pad:pad + cols]
    b = b.t() if kmajor else b
    a[M - 1, 200:264] = 3.0e4                      # partials beyond the fast conversion's range in one row
    for kt in (64, 128):
        with L.overrides(gemm_k_tile=kt, gemm_split_k=split or None):
            got, got_c = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16), _gemm(a, b, None, 64, 16)
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_NO_SKINNY):
            want, want_c = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16), _gemm(a, b, None, 64, 16)
        assert torch.equal(got, want) and torch.equal(got_c.view(torch.int16), want_c.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M,N", [(129, 130), (300, 136), (256, 161), (290, 552), (417, 288)])
@pytest.mark.parametrize("big", [False, True])
def test_two_sm_kernel_output_paths(M, N, big):
    """Outputs that leave by TMA (rows on 16 bytes: boxes of 32 rows and columns, clipped at every edge), those the
    threads store (odd N), and sums beyond the shortcut's 2^22, with a bias: the plain-conversion kernel's bits."""
    from fxpr_vllm import _native as nat

    K = 256
    a = _rand((M, K), torch.bfloat16, M, 3.0 if big else 1.0).cuda()
    b = _rand((N, K), torch.bfloat16, N, 1.5 if big else 0.05).cuda().t()
    bias = _rand((N,), torch.bfloat16, 9).cuda()
    out = []
    for flags in (nat.GEMM_PAIR, nat.GEMM_FORCE_EXACT_TC):
        with L.overrides(gemm_k_tile=64, gemm_split_k=1, gemm_flags=flags):
            out.append([_gemm(a, b, x, bits, 16) for x in (None, bias) for bits in (32, 64)])
    for got, exp in zip(*out):
        assert torch.equal(got.view(torch.int16), exp.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M", [33, 62, 63, 64])
@pytest.mark.parametrize("split", [2, 5, 6, 7, 8])
@pytest.mark.parametrize("K", [896, 1064])
def test_decode_shape_cluster_merge_at_every_rank_count(M, split, K):
    """What the ranks of a merge send each other has room at every rank count: seven ranks of 64 rows receive the
    most, also where eight are asked for and there are seven K-tiles.  The unsplit integers and outputs."""
    a, b = _rand((M, K), torch.bfloat16, M).cuda(), _rand((K, 392), torch.bfloat16, split, 0.05).cuda()
    far = a.clone()
    far[M - 1, :64] = 3.0e5                            # sums beyond 32 bits in one of the splits
    out = []
    for sp in (split, 1):
        with L.overrides(gemm_k_tile=128, gemm_split_k=sp):
            out.append([torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16), torch.ops.fxpr.gemm_fxp_int(a, b, 32, 16),
                        torch.ops.fxpr.gemm_fxp_int(far, b, 64, 16), _gemm(a, b, None, 64, 16).view(torch.int16)])
    for got, exp in zip(*out):
        assert torch.equal(got, exp)
    L.check_device_status()


@pytest.mark.parametrize("M,split", [(5, 8), (16, 3), (33, 2), (64, 7), (64, 8), (80, 2), (100, 3), (128, 4)])
@pytest.mark.parametrize("wide", ["one", "some", "all"])
def test_cluster_merges_of_sums_beyond_32_bits(M, split, wide):
    """High words cross the cluster by plain loads: from one split, from some and from all of them, call after call."""
    K = 64 * 16
    a, b = _rand((M, K), torch.bfloat16, M).cuda(), _rand((K, 392), torch.bfloat16, split, 0.05).cuda()
    for t in {"one": [3], "some": [0, 1, 5], "all": range(16)}[wide]:
        a[t % M::3, 64 * t:64 * t + 64] = 3.0e5                      # partials of about 1.2e5 * 2^16
    with L.overrides(gemm_k_tile=64, gemm_split_k=1):
        exp = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
    assert exp.abs().max().item() > 1 << 32
    with L.overrides(gemm_k_tile=64, gemm_split_k=split, gemm_flags=4096):     # GEMM_MID above 64 rows
        for got in [torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16) for _ in range(20)]:
            assert torch.equal(got, exp)
    L.check_device_status()


@pytest.mark.parametrize("M,split", [(9, 8), (64, 3), (80, 2), (128, 4)])
def test_cluster_merges_wrap_32_bit_sums(M, split):
    """1040 partials of 60 * 2^16, all in the fast range: 32-bit sums wrap around in the merge, 64-bit ones do not."""
    K = 64 * 1040
    a, b = torch.ones(M, K, dtype=torch.bfloat16, device="cuda"), torch.full((K, 136), 0.9375, dtype=torch.bfloat16, device="cuda")
    with L.overrides(gemm_k_tile=64, gemm_split_k=split, gemm_flags=4096):         # GEMM_MID above 64 rows
        narrow, full = (torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16) for bits in (32, 64))
    total = 1040 * 60 << 16
    assert (full == total).all()
    assert (narrow == (total + (1 << 31)) % (1 << 32) - (1 << 31)).all()
    L.check_device_status()


@pytest.mark.parametrize("M,N", [(129, 130), (300, 136), (256, 161), (290, 552), (417, 260), (200, 129)])
@pytest.mark.parametrize("far", [False, True])
def test_two_sm_kernel_integer_outputs(M, N, far):
    """Integer sums by TMA where their rows start on 16 bytes (32 or 64 bits a column) and by rows where not, at every
    edge, with a fix-up in some warps, alone and next to the io outputs: the plain-conversion kernel's integers."""
    from fxpr_vllm import _native as nat

    K = 320
    a = _rand((M, K), torch.float16, M, 2.0).cuda()
    b = _rand((N, K), torch.float16, N, 1.0).cuda().t()
    if far:
        a[M // 2, 64:128] = 3.0e4
    lib = nat.load()
    for bits, dtype in ((32, torch.int32), (64, torch.int64)):
        with L.overrides(gemm_k_tile=64, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
            want = torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16)
            want_c = _gemm(a, b, None, bits, 16)
        with L.overrides(gemm_k_tile=64, gemm_split_k=1, gemm_flags=nat.GEMM_PAIR):
            assert torch.equal(torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16), want)
        c = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
        c_int = torch.full((M, N), -1, device="cuda", dtype=dtype)
        assert lib.fxpr_gemm(a.data_ptr(), b.data_ptr(), None, c.data_ptr(), c_int.data_ptr(), 0, M, N, K, K, 1, 1, K, N, bits, 16,
                             64, 1, nat.GEMM_PAIR, None, 0, None, None, torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(c_int, want) and torch.equal(c.view(torch.int16), want_c.view(torch.int16))
    L.check_device_status()


def _fastest_us(fn, n=5):
    times = []
    for _ in range(n):
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        fn()
        stop.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(stop) * 1e3)
    return min(times)


def test_two_sm_kernel_time_does_not_depend_on_the_size_of_the_sums():
    """Sums of 64.0 and more (16 fraction bits) are ordinary outputs of operands with a mean: they may not cost a
    multiple of small sums (2.1 to 2.3 times when they went element by element through local memory)."""
    a = _rand((4096, 4096), torch.bfloat16, 1).cuda()
    b = _rand((4096, 4096), torch.bfloat16, 2, 0.02).cuda()
    far_a, far_b = a + 0.5, b + 0.1
    for kt in (64, 128):
        with L.overrides(gemm_k_tile=kt):
            small = _fastest_us(lambda: _gemm(a, b, None, 64, 16))
            large = _fastest_us(lambda: _gemm(far_a, far_b, None, 64, 16))
        assert _gemm(far_a, far_b, None, 64, 16).float().abs().median() > 100
        assert large < 1.4 * small, (kt, small, large)


@pytest.mark.parametrize("M,N,K", [
    (65, 128, 64), (96, 256, 200), (97, 264, 1096), (128, 392, 640), (129, 520, 1096), (192, 256, 2056), (193, 1000, 328),
    (257, 384, 712), (333, 776, 456), (700, 520, 136),
])
@pytest.mark.parametrize("kt,split", [(64, 1), (128, 1), (64, 2), (128, 3), (64, 4)])
def test_medium_batch_kernel(M, N, K, kt, split):
    """Row tiles of 96 to 256 at and past their edges, ragged columns and K, one to four K-splits in a cluster (some
    with fewer rows to merge than others), both weight layouts, and partials beyond the fast conversion's range in
    some tiles only: the integers and outputs of the plain-conversion kernel."""
    from fxpr_vllm import _native as nat

    split = min(split, -(-K // kt))
    dtype = torch.float16 if N % 16 else torch.bfloat16
    a = _rand((M, K), dtype, M).cuda()
    b = _rand((K, N), dtype, N, 0.05).cuda()
    bias = _rand((N,), dtype, 7).cuda()
    far = a.clone()
    far[M - 1, :64] = 3.0e4
    for bb in (b, b.t().contiguous().t()):
        out = []
        for flags, sp in ((nat.GEMM_MID, split), (nat.GEMM_FORCE_EXACT_TC, 1)):
            with L.overrides(gemm_k_tile=kt, gemm_split_k=sp, gemm_flags=flags):
                out.append([torch.ops.fxpr.gemm_fxp_int(a, bb, 64, 16), torch.ops.fxpr.gemm_fxp_int(far, bb, 64, 16),
                            torch.ops.fxpr.gemm_fxp_int(far, bb, 32, 16), _gemm(a, bb, bias, 64, 16).view(torch.int16),
                            _gemm(far, bb, None, 64, 16).view(torch.int16)])
        for got, exp in zip(*out):
            assert torch.equal(got, exp)
    L.check_device_status()


@pytest.mark.parametrize("M,split", [(3, 1), (20, 1), (64, 4), (64, 7), (64, 16), (80, 1), (129, 3), (250, 1)])
@pytest.mark.parametrize("N", [129, 258, 391])
def test_columns_that_are_no_multiple_of_four(M, N, split):
    """Weights as an (N, K) view allow any N: the decode-shape and medium-batch kernels' scalar stores and bias guards at
    the last columns, an output whose rows start anywhere, and activations that are columns of a wider matrix."""
    from fxpr_vllm import _native as nat

    K = 1160
    wide = _rand((M, K + 24), torch.bfloat16, M).cuda()
    a = wide[:, 8:8 + K]
    b = _rand((N, K), torch.bfloat16, N, 0.05).cuda().t()
    bias = _rand((N,), torch.bfloat16, 3).cuda()
    flag = nat.GEMM_MID if M > 64 else 0
    for kt in (64, 128):
        with L.overrides(gemm_k_tile=kt, gemm_split_k=split, gemm_flags=flag):
            got = [torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16) for bits in (32, 64)] + [_gemm(a, b, x, 64, 16) for x in (None, bias)]
        with L.overrides(gemm_k_tile=kt, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
            want = [torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16) for bits in (32, 64)] + [_gemm(a, b, x, 64, 16) for x in (None, bias)]
        for x, y in zip(got, want):
            assert torch.equal(x if x.dtype != torch.bfloat16 else x.view(torch.int16), y if y.dtype != torch.bfloat16 else y.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M,N,K,split", [(16, 256, 520, 1), (64, 384, 1160, 4), (80, 384, 1160, 1), (129, 640, 1160, 3), (300, 256, 520, 1)])
def test_infinities_and_nan_in_the_newer_kernels(M, N, K, split):
    """Partials that are infinite or NaN take the fix-up: what the plain-conversion kernel makes of them."""
    from fxpr_vllm import _native as nat

    a = _rand((M, K), torch.float16, 51).cuda()
    b = _rand((K, N), torch.float16, 52, 0.05).cuda()
    a[M // 2, 70] = float("inf")
    a[0, 130] = float("-inf")
    b[300, N - 3] = float("nan")
    flags = {16: 0, 64: 0, 80: nat.GEMM_MID, 129: nat.GEMM_MID, 300: nat.GEMM_PAIR}[M]
    for bits in (32, 64):
        with L.overrides(gemm_k_tile=64, gemm_split_k=split, gemm_flags=flags):
            got, got_c = torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16), _gemm(a, b, None, bits, 16)
        with L.overrides(gemm_k_tile=64, gemm_split_k=1, gemm_flags=nat.GEMM_FORCE_EXACT_TC):
            want, want_c = torch.ops.fxpr.gemm_fxp_int(a, b, bits, 16), _gemm(a, b, None, bits, 16)
        assert torch.equal(got, want) and torch.equal(got_c.view(torch.int16), want_c.view(torch.int16))
    L.check_device_status()


@pytest.mark.parametrize("M,N,K,flag,want", [
    (80, 4096, 4096, 0, "gemm_tc_mid_kernel"), (333, 6144, 4096, 0, "gemm_tc_mid_kernel"),
    (64, 4096, 4096, 0, "gemm_tc_skinny_kernel"), (4096, 4096, 4096, 0, "gemm_tc_pair_kernel"),
    (333, 6144, 4096, 128, "gemm_tc_fast_kernel"),                # GEMM_TILE_N128
])
def test_which_kernel_a_medium_batch_takes(M, N, K, flag, want):
    a, b = _rand((M, K), torch.bfloat16, 1).cuda(), _rand((K, N), torch.bfloat16, 2, 0.05).cuda()
    with L.overrides(gemm_flags=flag):
        names = [n for n in _kernels_launched(lambda: _gemm(a, b, None, 64, 16)) if "gemm" in n]
    if not names:
        pytest.skip("no kernel activity from the profiler")
    assert any(want in n for n in names), names


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,f,K", [(64, 1792, 1024), (33, 200, 512), (1, 128, 256), (64, 4096, 2048)])
@pytest.mark.parametrize("split", [0, 1, 2, 3, 4])
def test_silu_mul_epilogue_equals_gemm_then_silu_mul(dtype, M, f, K, split):
    """The decode-shape GEMM with (gate, up) column pairs and SiLU*mul in its epilogue gives the
    bits of the plain GEMM on [gate | up] followed by the SiLU*mul kernel, for every split
    route (one CTA per tile, cluster merge, partial planes), and so does the two-kernel form on
    the paired layout that larger batches take."""
    from fxpr_vllm import _lib as L

    g = torch.Generator().manual_seed(M * 7 + f)
    a = torch.randn(M, K, generator=g).to(dtype).cuda()
    wg = (0.05 * torch.randn(K, f, generator=g)).to(dtype).cuda()
    wu = (0.05 * torch.randn(K, f, generator=g)).to(dtype).cuda()
    kw = {} if split == 0 else {"gemm_split_k": split}
    with L.overrides(gemm_k_tile=128, **kw):
        want = L.silu_mul(torch.ops.fxpr.gemm_fxp(a, torch.cat([wg, wu], dim=1).contiguous(), None, 64, 16))
        pairs = L.interleave_gate_up(wg, wu)
        got = L.gemm_silu_mul(a, pairs, 64, 16)
        two = L.silu_mul_pairs(torch.ops.fxpr.gemm_fxp(a, pairs, None, 64, 16))
    assert got.shape == (M, f)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(two.view(torch.int16), want.view(torch.int16))


def test_silu_mul_epilogue_falls_back_for_large_batches():
    from fxpr_vllm import _lib as L

    g = torch.Generator().manual_seed(3)
    a = torch.randn(200, 512, generator=g).to(torch.bfloat16).cuda()
    wg = (0.05 * torch.randn(512, 384, generator=g)).to(torch.bfloat16).cuda()
    wu = (0.05 * torch.randn(512, 384, generator=g)).to(torch.bfloat16).cuda()
    want = L.silu_mul(torch.ops.fxpr.gemm_fxp(a, torch.cat([wg, wu], dim=1).contiguous(), None, 64, 16))
    got = L.gemm_silu_mul(a, L.interleave_gate_up(wg, wu), 64, 16)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(64, 16032, 512), (33, 1000, 256), (1, 128, 128), (64, 4096, 1024)])
def test_gemm_argmax_keys_equal_argmax_of_the_logits(dtype, M, N, K):
    """The lm_head GEMM that also leaves per-row arg-max keys: same logits as ``gemm_fxp``, the
    winning column equals ``torch.argmax`` of them (first maximal column: the weights hold
    duplicated columns, so every row has ties), and the keys of two column shards combine to the
    key of the whole row."""
    from fxpr_vllm import _lib as L

    g = torch.Generator().manual_seed(N + M)
    a = torch.randn(M, K, generator=g).to(dtype).cuda()
    b = (0.05 * torch.randn(K, N, generator=g)).to(dtype)
    b[:, N // 3] = b[:, N // 2]                      # exact ties between far-apart columns
    b[:, N - 1] = b[:, 0]
    b = b.cuda()
    want = torch.ops.fxpr.gemm_fxp(a, b, None, 64, 16)
    logits, keys = L.gemm_fxp_argmax(a, b, None, 64, 16)
    assert torch.equal(logits.view(torch.int16), want.view(torch.int16))
    assert torch.equal(L.argmax_from_keys(keys), want.argmax(dim=-1))
    assert torch.equal(keys, L.argmax_keys_of(want))
    half = (N // 2 + 127) // 128 * 128 if N > 256 else N // 2
    k0 = L.gemm_fxp_argmax(a, b[:, :half].contiguous(), None, 64, 16, n_offset=0)[1]
    k1 = L.gemm_fxp_argmax(a, b[:, half:].contiguous(), None, 64, 16, n_offset=half)[1]
    assert torch.equal(L.combine_argmax_keys([k0, k1]), keys)
    big = torch.randn(100, K, generator=g).to(dtype).cuda()      # more than 64 rows: two-kernel form
    lg2, k2 = L.gemm_fxp_argmax(big, b, None, 64, 16)
    assert torch.equal(L.argmax_from_keys(k2), lg2.argmax(dim=-1))


@pytest.mark.parametrize("split", [0, 1, 4])
def test_static_weights_promise_changes_no_bit(split):
    """With FXPR_GEMM_WEIGHTS_STATIC the decode-shape kernel only moves its first weight requests
    in front of the dependency wait; the outputs are the same, also back to back in one stream
    with a kernel that writes the activations just before."""
    from fxpr_vllm import _lib as L

    g = torch.Generator().manual_seed(11)
    w = (0.05 * torch.randn(2048, 1536, generator=g)).to(torch.bfloat16).cuda()
    x0 = torch.randn(48, 2048, generator=g).cuda()
    torch.cuda.synchronize()                                # the weights are complete, as the flag promises
    kw = {} if split == 0 else {"gemm_split_k": split}
    with L.overrides(gemm_k_tile=128, **kw):
        wants = {sc: torch.ops.fxpr.gemm_fxp((x0 * sc).to(torch.bfloat16), w, None, 64, 16) for sc in (1.0, 0.5, 2.0)}
        with L.static_weights():
            for sc in (1.0, 0.5, 2.0):
                x = (x0 * sc).to(torch.bfloat16)            # written by the kernel right before the GEMM
                assert torch.equal(torch.ops.fxpr.gemm_fxp(x, w, None, 64, 16), wants[sc])
        assert torch.equal(torch.ops.fxpr.gemm_fxp(x0.to(torch.bfloat16), w, None, 64, 16), wants[1.0])


def _split_calls(n):
    """Operands of `n` products of more than 64 rows that split K through the scratch, and their results."""
    out = []
    for i in range(n):
        M, N, K = (200, 300, 65, 128)[i % 4], (512, 384, 640)[i % 3], (4096, 2048)[i % 2]
        a, b = _rand((M, K), torch.bfloat16, 300 + i).cuda(), _rand((K, N), torch.bfloat16, 400 + i, 0.05).cuda()
        with L.overrides(gemm_split_k=1):
            out.append((a, b, torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)))
    torch.cuda.synchronize()
    return out


def test_streams_that_split_k_at_the_same_time_do_not_share_scratch():
    """Split products on more streams than scratch is kept for, all in flight together, round after round."""
    streams = [torch.cuda.Stream() for _ in range(20)]
    calls = _split_calls(len(streams))
    with L.overrides(gemm_split_k=8):
        for _ in range(5):
            got = []
            for s, (a, b, _) in zip(streams, calls):
                with torch.cuda.stream(s):
                    got += [torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16) for _ in range(3)]
            torch.cuda.synchronize()
            for i, g in enumerate(got):
                assert torch.equal(g, calls[i // 3][2]), i


_CAPTURE_AFTER_WARM_UP = """
import torch, fxpr_vllm
from fxpr_vllm import warmup, _lib as L
M, N, K = %d, %d, %d
a = torch.randn(M, K, device="cuda").bfloat16()
b = torch.randn(K, N, device="cuda").bfloat16() * 0.02
warmup.warmup_gemm(b, 64, 16)
with L.overrides(gemm_k_tile=64):
    assert L.pick_split_k(M, N, K, 64, 64, 148) > 1
    small = torch.ops.fxpr.gemm_fxp_int(a[:, :256], b[:256, :256], 64, 16)     # loads the kernels
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)
    graph.replay()
    torch.cuda.synchronize()
    with L.overrides(gemm_split_k=1):
        assert torch.equal(out, torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16))
L.check_device_status()
print("captured")
"""


@pytest.mark.parametrize("M,N,K", [(65, 9600, 14336), (65, 10752, 18944)])
def test_a_split_that_a_cluster_merges_needs_no_scratch_in_a_capture(M, N, K):
    """Warmed up as a model is, a shape that was never run is captured: its planes would exceed the warmed scratch.
    In a process of its own, since scratch that other tests grew would hide it."""
    import subprocess
    import sys
    from pathlib import Path

    pkg = Path(fxpr_vllm.__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", _CAPTURE_AFTER_WARM_UP % (M, N, K)], cwd=pkg, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]


def test_a_graph_that_splits_k_does_not_share_scratch_with_eager_calls():
    (a, b, want), (a2, b2, want2) = _split_calls(2)
    with L.overrides(gemm_split_k=8):
        torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16)                  # sizes the scratch, as a warm-up does
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [torch.ops.fxpr.gemm_fxp_int(a, b, 64, 16) for _ in range(8)]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        for _ in range(5):
            with torch.cuda.stream(side):
                graph.replay()
            eager = [torch.ops.fxpr.gemm_fxp_int(a2, b2, 64, 16) for _ in range(8)]
            torch.cuda.synchronize()
            assert all(torch.equal(o, want) for o in outs)
            assert all(torch.equal(o, want2) for o in eager)
