"""Host-side logic that needs no GPU: the split policies (speed decisions only: every choice gives
the same bits) and the arg-max key arithmetic of the fused lm_head GEMM."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest
import torch

import fxpr_vllm  # noqa: F401
from fxpr_vllm import _lib as L


def _policy_program(tmp_path, body):
    """What a C++ program over csrc/host_policy.h prints (the functions that no C entry exports)."""
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    header = Path(fxpr_vllm.__file__).resolve().parent.parent / "csrc" / "host_policy.h"
    src, exe = tmp_path / "policy.cpp", tmp_path / "policy"
    src.write_text(f'#include "{header}"\n#include <chrono>\n#include <cstdio>\nusing namespace fxpr;\nint main() {{\n{body}\n}}\n')
    subprocess.run(["g++", "-O2", "-std=c++17", str(src), "-o", str(exe)], check=True, capture_output=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


def test_decode_gemm_split_policy_fills_the_sms_once():
    sms = 148
    for (n, k), want in {(4096, 4096): 4, (6144, 4096): 2, (28672, 4096): 1, (4096, 14336): 4,
                         (768, 4096): 8, (4096, 512): 1, (3584, 4096): 4, (4096, 1792): 4,
                         (128256, 4096): 1}.items():
        got = L.pick_split_k(64, n, k, 128, 64, sms)
        assert got == want, (n, k, got)
        tiles = -(-n // 128)
        assert got == 1 or tiles * got <= sms * 9 // 10          # clusters of whole-SM CTAs need headroom
        assert got == 1 or k // got >= 384
    assert L.pick_split_k(64, 4096, 4096, 128, 16, sms) == 1      # int16 accumulators never split
    assert L.pick_split_k(4096, 4096, 4096, 64, 64, sms) == 1     # the output tiles fill the GPU


def test_medium_batches_split_into_clusters():
    """65 rows and more: K-splits that a cluster merges (at most four) where those are cheaper than planes in
    scratch, none where the tiles fill the pairs, powers of two up to 16 for the CUDA-core and int16 callers' old rule."""
    sms = 148
    assert L.pick_split_k(80, 4096, 4096, 128, 64, sms) == 3      # 16 column tiles: clusters of six
    assert L.pick_split_k(80, 6144, 4096, 128, 64, sms) == 2
    assert L.pick_split_k(333, 6144, 4096, 128, 64, sms) == 1
    assert L.pick_split_k(700, 6144, 4096, 128, 64, sms) == 1
    assert L.pick_split_k(80, 4096, 4096, 128, 16, sms) == 1
    for kt in (64, 128):
        for m in (65, 100, 200, 400, 700):
            for n, k in ((768, 4096), (4096, 14336), (28672, 4096), (1064, 2376)):
                got = L.pick_split_k(m, n, k, kt, 64, sms)
                assert 1 <= got <= 16 and got <= -(-k // kt)


def test_medium_batch_plan_takes_a_handful_of_steps_and_finds_the_cheapest_row_tiles(tmp_path):
    """Every call above 64 rows makes this plan on the host: its time must not grow with the rows."""
    assert float(_policy_program(tmp_path, """
  const auto t0 = std::chrono::steady_clock::now();
  volatile int sink = 0;
  for (int i = 0; i < 1000; ++i) sink = sink + plan_mid_rows(1000000 + i, 4096, 4096, 128, 1, 148).row_tiles;
  std::printf("%f", std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count() / 1000);
""")) < 10.0                                                       # us; 98 when it walked all tile counts
    assert _policy_program(tmp_path, """
  int calls = 0, worse = 0;
  for (int64_t M = 65; M < 1500; M += 13)
    for (int64_t N : {128, 136, 768, 1000, 4096, 6144, 28672})
      for (int64_t K : {64, 512, 4096, 14336})
        for (int kt : {64, 128})
          for (int split = 1; split <= 4; ++split) {
            double least = 1e30;
            for (int64_t t = ceil_div(M, split > 1 ? 128 : 256); t <= ceil_div(M, 64); ++t)
              least = std::min(least, est_mid_us(mid_tile_rows(M, t), t, N, K, kt, split, 148));
            const MidPlan plan = plan_mid_rows(M, N, K, kt, split, 148);
            ++calls;
            worse += plan.us != least || ceil_div(M, plan.row_tiles) > (split > 1 ? 128 : 256);
          }
  std::printf("%d %d", calls, worse);
""") == "24864 0"


def test_two_planes_are_taken_where_they_measured_faster(tmp_path):
    """Calls that went to the medium-batch kernel and lost 4 to 15 % by it: two K-splits through planes."""
    for m, n, k, kt in ((200, 4096, 14336, 64), (299, 3064, 11912, 128), (402, 2016, 15704, 64), (501, 2120, 4424, 64)):
        assert L.pick_split_k(m, n, k, kt, 64, 148) == 2
        assert _policy_program(tmp_path, f'  std::printf("%d", mid_route({m}, {n}, {k}, {kt}, 2, 148));') == "0"
    assert L.pick_split_k(154, 4808, 8800, 64, 64, 148) == 3          # 48 us in a cluster of three, 54 unsplit


def test_splits_follow_the_kernel_that_runs(tmp_path):
    """The medium-batch kernel's cluster merges set the split only where that kernel may run: not above 21 fraction
    bits or in the exact-conversion kernel (planes, at most four), and not where a flag names another kernel."""
    got = _policy_program(tmp_path, """
  for (int64_t M : {80, 200, 256})
    for (int64_t N : {256, 768, 4096})
      for (auto k : {wide_kernels(16, 0), wide_kernels(32, 0), wide_kernels(16, FXPR_GEMM_FORCE_EXACT_TC),
                     wide_kernels(16, FXPR_GEMM_TILE_N128), wide_kernels(16, FXPR_GEMM_MID)})
        std::printf("%d ", pick_gemm_split_k(M, N, 4096, 128, 64, 148, k));
""").split()
    # (any kernel, 32 fraction bits, exact, 128 x 128 tiles, the medium-batch flag) by shape
    rows = [list(map(int, got[i:i + 5])) for i in range(0, len(got), 5)]
    for (m, n), (free, fine, exact, single, mid) in zip([(m, n) for m in (80, 200, 256) for n in (256, 768, 4096)], rows):
        tiles = -(-m // 128) * (n // 128)
        doubled = 1
        while doubled < 16 and tiles * doubled * 2 <= 148 and 32 // (doubled * 2) >= 4:
            doubled *= 2
        assert fine == exact == min(4, 148 // tiles) and single == doubled and mid == free <= 4, (m, n)


def test_splits_that_no_cluster_merges_stay_within_the_scratch_of_the_warm_up(tmp_path):
    """CUDA-graph capture cannot grow the scratch: whatever the policy picks needs what ``warmup_gemm`` made, or none."""
    from fxpr_vllm import _native as nat

    planes = _policy_program(tmp_path, """
  for (int64_t M : {65, 80, 96, 97, 128, 129, 200, 256, 257, 300, 384})
    for (int64_t N = 128; N <= 20000; N += N < 1500 ? 8 : 328)
      for (int64_t K : {1024, 4096, 14336, 18944, 70000})
        for (int kt : {64, 128}) {
          const int split = pick_gemm_split_k(M, N, K, kt, 64, 148);
          if (split > 1 && !mid_route(M, N, K, kt, split, 148))
            std::printf("%d %d %d\\n", (int)M, (int)N, split);
        }
""")
    shapes = {tuple(map(int, line.split())) for line in planes.splitlines()}
    assert shapes
    lib = nat.load()
    for m, n, split in shapes:
        for bits in (32, 64):
            assert lib.fxpr_gemm_scratch_bytes(m, n, bits, split) <= L.gemm_scratch_policy_bytes(148, bits), (m, n, split)


def test_decode_attention_rank_policy():
    f = L.pick_num_splits_b200
    assert f(5, 64, 1, 32, 8, 8192, 148) == 5                     # an explicit request is kept
    assert f(64, 64, 1, 32, 8, 8192, 148) == 16                   # up to the cluster limit
    assert f(0, 64, 1, 32, 8, 8192, 148) == 8                     # long contexts: ~1024 keys per rank
    assert f(0, 64, 1, 32, 8, 4096, 148) == 4
    assert f(0, 64, 1, 32, 8, 1280, 148) == 1                     # the stash still leaves 4 CTAs per SM
    assert f(0, 64, 1, 32, 8, 1408, 148) == 2
    assert f(0, 64, 1, 16, 4, 1280, 148) == 2                     # fewer clusters: fill one wave
    assert f(0, 64, 1, 8, 2, 1280, 148) == 4
    assert f(0, 64, 1, 4, 1, 1280, 148) == 8
    assert f(0, 1, 1, 32, 8, 128, 148) == 1                       # two key tiles per rank at least
    assert f(0, 16, 4096, 32, 8, 4096, 148) == 1                  # prefill with enough row blocks


def test_decode_ranks_of_small_batches_and_last_waves():
    f = L.pick_num_splits_b200
    assert f(0, 25, 1, 32, 8, 3168, 148) == 2                     # three ranks would be a full wave and eight CTAs
    assert f(0, 64, 1, 32, 8, 2048, 148) == 2                     # nearly two full waves stay
    assert f(0, 40, 1, 32, 8, 2000, 148) == 2                     # one rank would leave mixed lengths unbalanced
    assert f(0, 10, 1, 32, 32, 8192, 148) == 2
    assert f(0, 5, 1, 32, 8, 704, 148) == 5                       # two key tiles a rank
    assert f(0, 1, 1, 32, 8, 3584, 148) == 16                     # a CTA per SM
    assert f(0, 2, 1, 32, 8, 3584, 148) == 8
    assert f(0, 1, 1, 4, 1, 64, 148) == 1                         # one key tile
    for n in (1, 7, 64, 300):
        for hq, hkv in ((32, 8), (16, 4), (4, 1), (32, 32), (16, 1)):
            for keys in (16, 100, 1000, 9600, 40000):
                assert 1 <= f(0, n, 1, hq, hkv, keys, 148) <= 16


def test_sixteen_ranks_fall_back_where_the_device_cannot_place_them(tmp_path):
    """A device that cannot place a cluster of sixteen (asked of a stand-in here) gets eight ranks, not an error."""
    assert _policy_program(tmp_path, """
  for (bool can : {false, true})
    for (int ranks : {1, 8, 9, 16}) {
      int asked = 0;
      const int got = ranks_that_fit(ranks, [&](int) { ++asked; return can; });
      std::printf("%d:%d ", got, asked);
    }
""").split() == ["1:0", "8:0", "8:1", "8:1", "1:0", "8:0", "9:1", "16:1"]


def test_argmax_keys_pick_the_first_maximum_and_combine_across_shards():
    g = torch.Generator().manual_seed(0)
    for dtype in (torch.bfloat16, torch.float16):
        x = torch.randn(7, 1000, generator=g).to(dtype)
        x[:, 900] = x[:, 17]                                      # ties (bf16 has plenty anyway)
        x[0, :] = -3.0                                            # a whole row of equal negatives
        x[1, 5] = float("inf")
        keys = L.argmax_keys_of(x)
        assert torch.equal(L.argmax_from_keys(keys), x.argmax(dim=-1))
        parts = [L.argmax_keys_of(x[:, a:b].contiguous(), n_offset=a) for a, b in ((0, 384), (384, 640), (640, 1000))]
        assert torch.equal(L.combine_argmax_keys(parts), keys)
        assert torch.equal(L.combine_argmax_keys(parts[::-1]), keys)   # order-free


def test_interleave_gate_up_layout():
    wg = torch.arange(12.0).reshape(3, 4)
    wu = -torch.arange(12.0).reshape(3, 4)
    p = L.interleave_gate_up(wg, wu)
    assert p.shape == (3, 8)
    assert torch.equal(p[:, 0::2], wg) and torch.equal(p[:, 1::2], wu)


def test_default_k_tiles_are_the_reference_ones():
    # fxpr_vllm/_triton/gemm.py:26-30; one table for the operators, the C ABI and Python callers
    assert dict(L.BLOCK_K_BY_DTYPE) == {torch.float16: 128, torch.bfloat16: 128, torch.float32: 64}
    with pytest.raises(KeyError):
        L.BLOCK_K_BY_DTYPE[torch.float64]
