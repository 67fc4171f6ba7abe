"""The launched form of a schedule and the tile configurations it chooses (no GPU)."""

import pytest

from mlc_compiler_b200 import Config, kir, load_schedule
from mlc_compiler_b200.emit import matmul as M
from mlc_compiler_b200.fuse import AttentionKernel, MatmulKernel, fuse
from mlc_compiler_b200.rewrite import prepare


@pytest.mark.parametrize("stem,launches,attentions,grouped", [
    ("bert-base_b1_s128_float16", 87, 12, 12), ("bert-base_b8_s128_bfloat16", 87, 12, 12),
    ("gpt2-small_b8_s128_float16", 86, 12, 0), ("bert-base_b1_s128_float32", 111, 0, 12),
    ("gpt2-small-streamed_b1_s128_float16", 110, 0, 0)])
def test_launched_form_is_whole_and_its_arena_disjoint(stem, launches, attentions, grouped):
    work = prepare(load_schedule(stem), Config())
    f = fuse(work, Config())
    assert len(f) == launches and not any(isinstance(k, kir.ExternKernel) for k in f.kernels)
    assert sum(isinstance(k, AttentionKernel) for k in f.kernels) == attentions
    assert sum(isinstance(k, MatmulKernel) and len(k.bs) == 3 for k in f.kernels) == grouped
    assert (f.inputs, f.outputs, f.params) == (work.inputs, work.outputs, work.params)
    ready = {b for b, s in f.buffers.items() if s.kind not in ("intermediate", "output")}
    first, last = {}, {}
    for i, k in enumerate(f.kernels):
        assert set(k.reads()) <= ready, (k.name, set(k.reads()) - ready)
        ready |= set(k.writes())
        for b in [*k.reads(), *k.writes()]:
            first.setdefault(b, i)
            last[b] = i
    assert {v.buffer for v in f.outputs} <= ready
    spans = [(f.plan.offsets[b], f.plan.offsets[b] + f.buffers[b].nbytes, b) for b in first if b in f.plan.offsets]
    for i, (lo, hi, b) in enumerate(spans):
        for lo2, hi2, c in spans[:i]:
            assert hi <= lo2 or hi2 <= lo or last[b] < first[c] or last[c] < first[b], (b, c)


def test_switched_off_nothing_is_fused():
    work = prepare(load_schedule("bert-base_b1_s128_float16"), Config())
    assert fuse(work, Config(own_matmuls=False)) is work
    kept = fuse(work, Config().as_scheduled())
    assert len(kept) == len(work) and not any(isinstance(k, AttentionKernel) for k in kept.kernels)


@pytest.mark.parametrize("m", [1, 127, 128, 129, 512, 1000, 4096, 16384])
@pytest.mark.parametrize("n", [8, 64, 72, 768, 1003, 3072, 50257])
def test_tile_choices_stay_inside_the_machine(m, n):
    for k in (8, 64, 136, 768, 1032, 3072, 4096):
        for groups, z, b_mn in ((1, 1, False), (3, 1, False), (1, 12, False), (1, 12, True)):
            if b_mn and n < 64:
                continue
            c = M.choose(z, m, n, k, groups, b_mn, k % 64 == 0)
            tiles = -(-m // (128 * c.cg)) * -(-n // c.bn) * groups * z
            kb = -(-k // 64)
            assert c.smem() <= M.SMEM_MAX and c.acc * c.bn <= 512 and 2 <= c.stages
            assert c.split == 1 or (c.cg == 1 and c.bn % (8 * c.split) == 0 and c.split <= kb and c.grid == tiles * c.split)
            assert c.split > 1 or c.grid == min(tiles * c.cg, M.SM_COUNT // c.cg * c.cg)
            assert c.grid % (c.split * c.cg) == 0 and (c.epi_warps == 4 or c.bn >= 64)
            assert c.cg == 1 or not b_mn
            assert c.acc == 2 or c.split > 1 or tiles <= M.SM_COUNT // c.cg
            # how K is split does not depend on what shares the launch
            assert M.choose(z, m, n, k, 1, b_mn, k % 64 == 0, 3).split == M.choose(z, m, n, k, 3, b_mn, k % 64 == 0, 3).split
            c32 = M.choose32(z, m, n, k, groups, b_mn)
            assert c32.smem() <= M.SMEM_MAX and c32.bn % (8 * c32.split) == 0 and c32.leads * c32.bn + c32.bn <= 512


@pytest.mark.parametrize("seq", [63, 64, 65])
def test_heads_as_wide_as_the_sequence_is_long_fuse_like_others(seq):
    import kir_oracle as oracle
    import torch

    from perf import cases

    assert len(fuse(prepare(cases.encoder_schedule(2, seq, 4, 2, "float16"), Config()), Config())) == 14
    s = cases.encoder_schedule(2, seq, 4, 1, "float32")
    g = torch.Generator().manual_seed(seq)
    params = {o: torch.randn(s.buffers[b].shape, generator=g) * 0.05 for b, o in s.params.items()}
    x = [torch.randn(v.shape, generator=g) for v in s.inputs]
    want, _ = oracle.run_schedule(s, params, x)
    got, _ = oracle.run_schedule(prepare(s, Config()), params, x)
    assert torch.equal(got, want)
