"""R1/R4 and NVFP4 indexers through the C ABI: ids bit-exact (ties to the lower
block id), descriptors and scores bit-exact against the oracle's fixed
arithmetic, and the reference's own gates against its stored outputs
(benchmarks/ch4_selectors/harness.py:22-42, 116-119)."""
import ctypes
import os

import numpy as np
import pytest
import torch

import oracle
from oracle import inputs as gen
from tests.golden import cases

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


def sp():
    import sparse_attention_b200_b200 as m
    return m


def margins(scores, topk):
    s = torch.sort(scores, dim=-1, descending=True).values
    return (s[..., :topk] - s[..., 1:topk + 1]).min().item() if scores.shape[-1] > topk else float("inf")


@pytest.mark.parametrize("family", ["gaussian", "cancellation_stress", "zeros"])
@pytest.mark.parametrize("r", [1, 4])
def test_summary_selector_reference_gate(family, r):
    m = sp()
    fx = np.load(os.path.join(G, "selectors.npz"))
    q, k = cases.selector_inputs(family)
    sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=16)
    sel.run()
    torch.cuda.synchronize()
    tag = f"{family}_r{r}"
    # reference gate: ids exact, scores atol 2e-5 / rtol 3e-4
    np.testing.assert_array_equal(sel.ids.cpu().numpy(), fx[tag + "_ids"])
    np.testing.assert_allclose(sel.scores.cpu().numpy(), fx[tag + "_scores"], atol=2e-5, rtol=3e-4)
    # oracle: everything bit for bit
    qd, kd, scores, ids = oracle.summary_select(q, k, r, 16)
    assert torch.equal(sel.qd.cpu().view(torch.int16), qd.view(torch.int16))
    assert torch.equal(sel.kd.cpu().view(torch.int16), kd.view(torch.int16))
    assert torch.equal(sel.scores.cpu(), scores)
    assert torch.equal(sel.ids.cpu(), ids)
    if family == "zeros":
        assert torch.equal(sel.ids.cpu(), torch.arange(16, dtype=torch.int32).expand_as(ids))


@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, Sq, Skv, R, topk, k offset
    (1, 8, 8, 4096, 4096, 1, 8, 0.5),        # configuration 1
    (2, 16, 2, 1024, 8192, 4, 32, 0.5),      # group 8, R4, top-32 of 64
    (1, 16, 1, 512, 16384, 4, 64, 0.5),      # group 16, top-64 of 128
    (1, 4, 2, 256, 1024, 2, 8, 0.0),         # R2, top-k == all blocks
    (1, 6, 2, 256, 2048, 4, 5, 0.0),         # group 3
])
def test_summary_selector_bit_exact(shape):
    b, hq, hkv, sq, skv, r, topk, off = shape
    m = sp()
    q, k, _ = gen.make_qkv(b, hq, hkv, sq, skv, seed=17, k_block_offset=off)
    sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=topk)
    sel.prepare()
    sel.score()
    torch.cuda.synchronize()
    qd, kd, scores, ids = oracle.summary_select(q, k, r, topk)
    assert torch.equal(sel.qd.cpu().view(torch.int16), qd.view(torch.int16))
    assert torch.equal(sel.kd.cpu().view(torch.int16), kd.view(torch.int16))
    assert torch.equal(sel.scores.cpu(), scores), (sel.scores.cpu() - scores).abs().max()
    assert torch.equal(sel.ids.cpu(), ids)
    print("k-th vs (k+1)-th score margin", margins(scores, topk))
    # the fused entry gives the same ids without storing scores
    sel2 = m.SummarySelector(q.cuda(), k.cuda(), r, topk=topk, keep_scores=False)
    assert torch.equal(sel2.run().cpu(), ids)


@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, Sq, Skv, R, topk, k offset
    (1, 8, 8, 4096, 4096, 1, 8, 0.5),        # one descriptor per list, 32 blocks (row tiles)
    (2, 16, 2, 1024, 8192, 4, 32, 0.5),      # group 8, R4 (GR = 32)
    (1, 16, 1, 512, 16384, 4, 64, 0.5),      # group 16, R4 (GR = 64), top-64 of 128
    (1, 4, 2, 256, 1024, 2, 8, 0.0),         # GR = 4, top-k == all blocks
    (1, 8, 2, 384, 32768, 1, 16, 0.5),       # GR = 4, 256 blocks, query-block count not a multiple of QB
    (1, 2, 1, 256, 65536, 4, 16, 0.0),       # GR = 8, 512 blocks
    (1, 6, 2, 256, 2048, 4, 5, 0.0),         # group 3: not eligible, exact kernel behind the same entry
])
def test_summary_selector_tensor_core_path_bit_exact(shape):
    """The entry that chooses between row tiles, pre-filter and exact kernels by size, against the oracle. (That the
    pre-filter itself ran is asserted by the tests of few descriptors, long lists and the persistent form below.)"""
    b, hq, hkv, sq, skv, r, topk, off = shape
    m = sp()
    q, k, _ = gen.make_qkv(b, hq, hkv, sq, skv, seed=19, k_block_offset=off)
    sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=topk, keep_scores=False)
    ids = sel.run_fast()
    torch.cuda.synchronize()
    m.device_status()
    ref = oracle.summary_select(q, k, r, topk)[3]
    assert torch.equal(ids.cpu(), ref)
    print("lists that fell back to exact scoring:", sel.fallback_lists())


def test_summary_selector_tensor_core_path_ties_and_constant_inputs():
    """Exact ties cannot be proven safe by the pre-filter: those lists must take the
    exact fallback and still come out with the lower block id first."""
    m = sp()
    # 160 lists (more than one per SM) of 16 descriptors: the tensor-core path, not the row-tile kernel; 64 blocks > 32
    # candidates
    q = torch.zeros((1, 4, 160 * 128, 128), dtype=torch.bfloat16)
    k = torch.zeros((1, 1, 8192, 128), dtype=torch.bfloat16)
    sel = m.SummarySelector(q.cuda(), k.cuda(), 4, topk=16, keep_scores=False)
    ids = sel.run_fast().cpu()
    assert torch.equal(ids, torch.arange(16, dtype=torch.int32).expand_as(ids))
    assert sel.fallback_lists() == ids.shape[0] * ids.shape[1] * ids.shape[2]
    # the same ties through the small-problem kernel (exact everywhere: no fallback is counted)
    q, k = cases.selector_inputs("zeros", skv=8192)
    sel = m.SummarySelector(q.cuda(), k.cuda(), 4, topk=16, keep_scores=False)
    ids = sel.run_fast().cpu()
    assert torch.equal(ids, torch.arange(16, dtype=torch.int32).expand_as(ids))
    assert sel.fallback_lists() == 0
    # constant non-zero inputs: every score equal and non-zero
    qc = torch.full_like(q, 0.5)
    kc = torch.full_like(k, -0.25)
    sel = m.SummarySelector(qc.cuda(), kc.cuda(), 1, topk=16, keep_scores=False)
    ids = sel.run_fast().cpu()
    assert torch.equal(ids, torch.arange(16, dtype=torch.int32).expand_as(ids))
    # duplicated KV blocks inside the top-k: equal exact scores, lower id first
    q, k, _ = gen.make_qkv(1, 4, 1, 256, 8192, seed=23)
    k = k.clone()
    k[:, :, 5 * 128:6 * 128] = k[:, :, 2 * 128:3 * 128]
    k[:, :, 9 * 128:10 * 128] = k[:, :, 2 * 128:3 * 128]
    sel = m.SummarySelector(q.cuda(), k.cuda(), 4, topk=16, keep_scores=False)
    assert torch.equal(sel.run_fast().cpu(), oracle.summary_select(q, k, 4, 16)[3])
    # the reference's stress family
    fx = np.load(os.path.join(G, "selectors.npz"))
    for family in ("gaussian", "cancellation_stress"):
        q, k = cases.selector_inputs(family)
        for r in (1, 4):
            sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=16, keep_scores=False)
            np.testing.assert_array_equal(sel.run_fast().cpu().numpy(), fx[f"{family}_r{r}_ids"])
    m.device_status()


@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, Sq, Skv, R, topk: long lists, where several warps share a list's threshold search
    (1, 16, 1, 1024, 2176 * 128, 1, 16),      # 8 lists per CTA, 2 warps per list
    (1, 16, 1, 256, 8320 * 128, 4, 64),       # 2 lists per CTA, 8 warps per list
    (1, 16, 1, 128, 16512 * 128, 4, 32),      # 1 list per CTA, all 16 warps on it
    (1, 8, 1, 160 * 128, 2048 * 128, 1, 16),  # 16 lists per CTA: two rounds of 8, 2 warps per list
])
def test_summary_selector_tensor_core_path_long_lists(shape):
    b, hq, hkv, sq, skv, r, topk = shape
    m = sp()
    q, k, _ = gen.make_qkv(b, hq, hkv, sq, skv, seed=29, k_block_offset=0.5)
    sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=topk, keep_scores=False)
    ids = sel.run_fast()
    torch.cuda.synchronize()
    m.device_status()
    assert float(sel.aux[:b * hkv].view(torch.float32).min()) > 0     # the key abs-max only the tensor-core path writes
    ref = oracle.summary_select(q, k, r, topk)[3]
    assert torch.equal(ids.cpu(), ref)
    print("lists that fell back to exact scoring:", sel.fallback_lists())


@pytest.mark.parametrize("hkv,g,qb,nb,r,topk", [
    (8, 1, 320, 1024, 1, 8),          # one descriptor per list
    (4, 2, 320, 1024, 1, 16),         # two
    (4, 2, 320, 600, 2, 16),          # four, two of them from R
    (2, 2, 160, 700, 4, 16),          # eight
])
@pytest.mark.parametrize("near", [False, True])
def test_summary_selector_tensor_core_path_few_descriptors(hkv, g, qb, nb, r, topk, near):
    """Lists of fewer than 16 descriptors take the pre-filter where their row tiles would be more than four 64 x 64 units
    per SM; near: twenty blocks at the top are copies of one block with one token scaled (differences that the
    approximate scores cannot order). Ids equal those of the staged exact kernel, every re-scored candidate is inside
    the error bound."""
    m = sp()
    gen_ = torch.Generator(device="cuda").manual_seed(53)
    q = (torch.randn((1, hkv * g, qb * 128, 128), device="cuda", generator=gen_) + (0.5 if near else 0.0)).to(torch.bfloat16)
    k = torch.randn((1, hkv, nb, 128, 128), device="cuda", generator=gen_) * (0.2 if near else 1.0)
    k += 0.5 * torch.randn((1, hkv, nb, 1, 128), device="cuda", generator=gen_) * (0.0 if near else 1.0)
    if near:
        k[:, :, :20] = k[:, :, :1] + 1.0
        k[:, :, :20, 5] *= 1.0 + 0.01 * torch.arange(20, device="cuda").view(20, 1)
    k = k.to(torch.bfloat16).view(1, hkv, nb * 128, 128)
    fast = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    ids = fast.run_fast().clone()
    exact = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    exact.prepare()
    exact.score()
    torch.cuda.synchronize()
    m.device_status()
    assert float(fast.aux[:hkv].view(torch.float32).min()) > 0      # the key abs-max only the tensor-core path writes
    assert torch.equal(ids, exact.ids)
    violations, ratio = fast.bound_stats()
    assert violations == 0
    if near:
        assert ratio > 0                                            # some candidates were re-scored exactly
    print("lists that fell back to exact scoring:", fast.fallback_lists(), "max |approx - exact| / delta:", ratio)


@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, Sq, Skv, R, topk: the persistent form (32 query descriptors per list, at least 8 query
    # blocks), whose selection warps see a list's scores chunk by chunk, and neighbours of it that stay with
    # the one-CTA-per-unit kernel (16 / 64 descriptors per list)
    (2, 16, 2, 44 * 128, 133 * 128, 4, 32),     # 8 lists per unit, last unit half empty, partial last key tile, one chunk
    (1, 8, 1, 24 * 128, 3000 * 128, 4, 48),     # 94 key tiles: 12 chunks of 8, 3 units
    (2, 32, 1, 16 * 128, 2100 * 128, 1, 16),    # group 32, R1: a chunk is two key tiles, 9 chunks
    (1, 16, 1, 160 * 128, 520 * 128, 2, 150),   # group 16, R2, 187 + 16 candidates: more than a chunk holds
    (3, 8, 1, 56 * 128, 64 * 128, 4, 60),       # all blocks are candidates (64 < 60 + 16)
    (1, 16, 1, 40 * 128, 2100 * 128, 1, 16),    # 16 descriptors per list: two warps per list, slices of 1056 and 1044
                                                # blocks (a remainder below 32 once left part of a warp out of a vote)
    (1, 16, 1, 12 * 128, 2100 * 128, 4, 64),    # 64 descriptors per list
])
def test_summary_selector_persistent_form_bit_exact(shape):
    b, hq, hkv, sq, skv, r, topk = shape
    m = sp()
    q, k, _ = gen.make_qkv(b, hq, hkv, sq, skv, seed=31, k_block_offset=0.5)
    q, k = q.cuda(), k.cuda()
    fast = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    ids = fast.run_fast().clone()
    exact = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    exact.prepare()
    exact.score()
    torch.cuda.synchronize()
    m.device_status()
    assert float(fast.aux[:b * hkv].view(torch.float32).min()) > 0     # the key abs-max only the tensor-core path writes
    assert torch.equal(ids, exact.ids)
    violations, ratio = fast.bound_stats()
    assert violations == 0
    print("lists that fell back to exact scoring:", fast.fallback_lists(), "max |approx - exact| / delta:", ratio)


@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, Sq, KV blocks, R, topk: lists far longer than shared memory could hold as a whole
    (1, 8, 1, 8 * 128, 32768, 4, 64),        # 4 Mi tokens: 1024 key tiles, 64 chunks per unit
    (1, 8, 1, 24 * 128, 20001, 4, 128),      # odd block count, 176 candidates
    (2, 32, 1, 9 * 128, 6000, 1, 16),        # group 32 with R1, last unit holds one list
])
def test_summary_selector_persistent_form_very_long_lists(shape):
    b, hq, hkv, sq, nt, r, topk = shape
    m = sp()
    g = torch.Generator(device="cuda").manual_seed(nt)
    q = torch.randn((b, hq, sq, 128), device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn((b, hkv, nt * 128, 128), device="cuda", generator=g).to(torch.bfloat16)
    fast = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    ids = fast.run_fast().clone()
    exact = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    exact.prepare()
    exact.score()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(ids, exact.ids)
    assert fast.bound_stats()[0] == 0


@pytest.mark.parametrize("order", ["ascending", "descending", "plateaus"])
def test_summary_selector_persistent_form_adversarial_score_order(order):
    """Scores that grow with the block index make every chunk beat everything seen before it (the pool of the
    streaming selection overflows and is cut back again and again); falling scores make the first chunk
    final; plateaus of exactly equal scores put ties on the threshold. Ids must equal the exact kernel's."""
    m = sp()
    b, hq, hkv, sq, skv, r, topk = 1, 8, 1, 24 * 128, 2304 * 128, 4, 32     # more than 2048 blocks: not a small problem
    nt = skv // 128
    g = torch.Generator().manual_seed(41)
    q = (torch.rand((b, hq, sq, 128), generator=g) + 0.5)
    ramp = torch.arange(nt, dtype=torch.float32) / nt
    if order == "descending":
        ramp = 1.0 - ramp
    if order == "plateaus":
        ramp = torch.floor(ramp * 16) / 16
    k = (0.25 + ramp).repeat_interleave(128)[None, None, :, None].expand(b, hkv, skv, 128).clone()
    if order != "plateaus":
        k = k + 0.001 * torch.randn((b, hkv, skv, 128), generator=g)
    q, k = q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda()
    fast = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    ids = fast.run_fast().clone()
    exact = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    exact.prepare()
    exact.score()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(ids, exact.ids)
    assert fast.bound_stats()[0] == 0
    print(order, "lists that fell back to exact scoring:", fast.fallback_lists())


@pytest.mark.parametrize("r,nt", [(1, 2112), (4, 64)])       # four descriptors per list: row tiles up to 2048 blocks
def test_summary_selector_tensor_core_path_near_ties(r, nt):
    """A cluster of almost equal blocks at the top of every list (copies of one block, some
    exact, some with one feature nudged): their approximate scores cannot order them, so the
    pre-filter must re-score exactly these and still agree with the oracle id for id, while
    the well separated blocks below them are ordered without exact scores."""
    m = sp()
    g = torch.Generator().manual_seed(77)
    q = (torch.randn((1, 4, 160 * 128, 128), generator=g) + 0.5).to(torch.bfloat16)   # 160 lists: not a small problem
    k = (0.2 * torch.randn((1, 1, nt * 128, 128), generator=g)).to(torch.bfloat16)
    base = (k[:, :, :128].float() + 1.0).to(torch.bfloat16)
    for blk in range(20):
        k[:, :, blk * 128:(blk + 1) * 128] = base
        if blk % 3:                                  # every third copy stays an exact duplicate of block 0
            k[0, 0, blk * 128:(blk + 1) * 128, blk] = (base[0, 0, :, blk].float() * (1.0 + 0.01 * blk)).to(torch.bfloat16)
    sel = m.SummarySelector(q.cuda(), k.cuda(), r, topk=32, keep_scores=False)
    ids = sel.run_fast().cpu()
    m.device_status()
    ref = oracle.summary_select(q, k, r, 32)[3]
    assert torch.equal(ids, ref)
    assert set(ids[0, 0, 0, :20].tolist()) == set(range(20))
    assert float(sel.aux[:1].view(torch.float32)) > 0     # the key abs-max only the tensor-core path writes
    assert sel.bound_stats()[0] == 0 and sel.bound_stats()[1] > 0     # candidates were re-scored, inside the bound
    assert sel.fallback_lists() <= 8                 # the near ties are settled by re-scoring, not by the fallback
    print("lists that fell back to exact scoring:", sel.fallback_lists())


@pytest.mark.parametrize("b,hkv,g,sq,skv,r,topk", [
    (2, 1, 16, 4096, 16384, 1, 16),      # the reference's selector benchmark shape: 16 query descriptors per list
    (2, 1, 16, 4096, 4096, 4, 16),       # 64 query descriptors, 4 key representatives per block
    (1, 2, 8, 1024, 2048 + 128, 2, 8),   # 16 descriptors, a block count that is no multiple of the chunk
    (1, 1, 1, 512, 8192, 1, 32),         # MHA: padded query descriptors
    (1, 4, 4, 256, 1024, 4, 8),
])
def test_small_problem_selector_equals_the_exact_kernels(b, hkv, g, sq, skv, r, topk):
    """The row-tile kernel for small problems (taken by run() and run_fast()) against the
    staged exact kernels (prepare() + score()): descriptors, scores and ids bit for bit,
    and ids against the CPU oracle."""
    m = sp()
    q, k, _ = gen.make_qkv(b, hkv * g, hkv, sq, skv, seed=31, k_block_offset=0.5)
    qc, kc = q.cuda(), k.cuda()
    staged = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    staged.prepare()
    staged.score()
    fused = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    fused.run()
    fast = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=False)
    fast.aux.fill_(7)
    fast.run_fast()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(fused.kd.view(torch.int16), staged.kd.view(torch.int16))
    assert torch.equal(fused.qd.view(torch.int16), staged.qd.view(torch.int16))
    assert torch.equal(fused.scores, staged.scores)
    assert torch.equal(fused.ids, staged.ids)
    assert torch.equal(fast.ids, staged.ids)
    assert fast.fallback_lists() == 0
    ref = oracle.summary_select(q, k, r, topk)[3]
    assert torch.equal(staged.ids.cpu(), ref)


@pytest.mark.parametrize("b,hkv,g,qb,nb,r,topk", [
    (1, 8, 1, 33, 32, 1, 8),        # one descriptor per list: 64 lists in a row tile, the second tile nearly empty
    (2, 3, 2, 40, 300, 1, 40),      # two per list; more than 256 blocks: threshold search
    (1, 2, 3, 21, 65, 1, 65),       # three per list padded to four, every block selected
    (1, 1, 3, 7, 129, 4, 129),      # twelve padded to sixteen, one key chunk more than a multiple, k > 128
    (1, 1, 5, 3, 2048, 1, 64),      # the largest block count, chunks for a whole cluster
    (1, 1, 16, 30, 70, 2, 1),       # 32 per list, two representatives, k = 1
    (3, 1, 12, 60, 33, 4, 12),      # 48 padded to 64: a list fills the row tile; not a power of two, any size
    (1, 1, 1, 70, 512, 1, 256),     # k > 128, sorted: several lists per CTA in one batch
    (1, 4, 1, 64, 300, 1, 140),     # more than one batch of lists per CTA, padded to 512
    (1, 1, 4, 20, 1025, 1, 700),    # padded to 2048
    (1, 1, 1, 40, 2048, 1, 2048),   # the largest block count, every block
    (1, 2, 3, 150, 200, 1, 129),    # at most 256 blocks, too many lists for counting
    (1, 1, 1, 1000, 300, 1, 5),     # many lists of one descriptor: four to a thread
    (1, 1, 2, 500, 301, 1, 7),      # two to a thread
    (1, 2, 1, 16, 128, 1, 8),       # few lists spread over small row tiles: one row per thread
    (1, 1, 3, 5, 20, 4, 3),         # the same, three chunks for four CTAs of a cluster
])
@pytest.mark.parametrize("ties", [False, True])
def test_row_tile_selector_equals_the_exact_kernels(b, hkv, g, qb, nb, r, topk, ties):
    """Lists of 1 to 64 descriptors packed into row tiles of 64, shared by 1 to 8 CTAs: ids and scores bit for bit
    against the staged exact kernels; with every third key block a copy of block 0 (equal scores, lower id first)."""
    m = sp()
    q, k, _ = gen.make_qkv(b, hkv * g, hkv, qb * 128, nb * 128, seed=37, k_block_offset=0.5)
    if ties:
        k = k.clone()
        for blk in range(0, nb, 3):
            k[:, :, blk * 128:(blk + 1) * 128] = k[:, :, :128]
    qc, kc = q.cuda(), k.cuda()
    staged = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    staged.prepare()
    staged.score()
    fused = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    fused.run()
    fast = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=False)
    fast.run_fast()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(fused.scores, staged.scores)
    assert torch.equal(fused.ids, staged.ids)
    assert torch.equal(fast.ids, staged.ids)


@pytest.mark.parametrize("keys", [64, 65, 127, 128, 129, 193])
@pytest.mark.parametrize("g,qb", [(64, 20), (2, 700), (1, 1500)])     # one, 32 and 64 lists to a tile of 64 rows
def test_row_tiles_at_the_edges_of_a_key_chunk(g, qb, keys):
    """Two groups of 64 keys in a chunk, the second one full, ragged or empty; four, two and one rows of a thread to a
    list: scores and ids bit for bit against the staged exact kernels."""
    m = sp()
    q, k, _ = gen.make_qkv(1, g, 1, qb * 128, keys * 128, seed=53, k_block_offset=0.5)
    qc, kc = q.cuda(), k.cuda()
    staged = m.SummarySelector(qc, kc, 1, topk=9, keep_scores=True)
    staged.prepare()
    staged.score()
    fused = m.SummarySelector(qc, kc, 1, topk=9, keep_scores=True)
    fused.run()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(fused.scores, staged.scores)
    assert torch.equal(fused.ids, staged.ids)


@pytest.mark.parametrize("hkv,g,qb,nb,r,topk", [
    (1, 12, 3, 24, 4, 16),      # 64 rows, one list to a tile, two CTAs with a chunk of 64 keys each
    (1, 32, 9, 75, 2, 75),      # four CTAs
    (1, 6, 58, 172, 4, 16),     # two lists to a tile
    (4, 8, 226, 41, 4, 41),     # more CTAs than fit at once
    (1, 16, 160, 1024, 1, 16),  # clusters of eight, a little more than a round
    (2, 1, 1131, 38, 4, 16),    # sixteen lists to a tile, one CTA each
])
def test_row_tiles_with_one_group_of_keys_to_a_chunk(hkv, g, qb, nb, r, topk):
    """Problems whose 64-row tiles go through 64 keys at a time, or did with another estimate: scores and ids bit for bit
    against the staged exact kernels."""
    m = sp()
    q, k, _ = gen.make_qkv(1, hkv * g, hkv, qb * 128, nb * 128, seed=59, k_block_offset=0.5)
    qc, kc = q.cuda(), k.cuda()
    staged = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    staged.prepare()
    staged.score()
    fused = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    fused.run()
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(fused.scores, staged.scores)
    assert torch.equal(fused.ids, staged.ids)


@pytest.mark.parametrize("b,hkv,g,qb,nb,r,topk", [
    (1, 2, 1, 80, 33, 1, 33),        # 160 lists of one descriptor, every block selected
    (1, 1, 2, 150, 300, 2, 40),      # four descriptors, threshold search
    (1, 1, 3, 152, 40, 1, 40),       # group of three: no tensor-core form
    (2, 1, 16, 8, 40, 4, 40),        # 64 descriptors, few lists
    (1, 1, 1, 4, 600, 1, 600),       # k > 128 of more than 256 blocks
])
def test_selector_with_nan_keys_and_queries_equals_the_exact_kernel(b, hkv, g, qb, nb, r, topk):
    """A NaN product never is a maximum: a block without any other product scores -inf and keeps an id of its own,
    whichever kernel scores it."""
    m = sp()
    q, k, _ = gen.make_qkv(b, hkv * g, hkv, qb * 128, nb * 128, seed=43, k_block_offset=0.5)
    k = k.clone()
    for blk in (0, 3, nb - 1):
        k[:, :, blk * 128:(blk + 1) * 128] = float("nan")           # no descriptor of the block is a number
    k[:, :, 5 * 128 + 7, 3] = float("nan")                          # one of its R descriptors is not
    q = q.clone()
    q[:, 0, 128] = float("nan")                                     # one head (R = 1: the whole row) of the second list
    qc, kc = q.cuda(), k.cuda()
    staged = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    staged.prepare()
    staged.score()
    fused = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=True)
    fused.run()
    fast = m.SummarySelector(qc, kc, r, topk=topk, keep_scores=False)
    fast.run_fast()
    torch.cuda.synchronize()
    m.device_status()
    assert not staged.scores.isnan().any()
    assert torch.isneginf(staged.scores[:, :, 0, 0]).all()
    assert torch.equal(fused.scores, staged.scores)
    assert torch.equal(fused.ids, staged.ids)
    assert torch.equal(fast.ids, staged.ids)
    assert all(len(set(row)) == topk for row in fused.ids.flatten(0, 2).tolist())


def test_summary_selector_duplicate_scores_tie_to_lower_id():
    """Duplicate KV blocks give exactly equal scores: the lower id must come first."""
    m = sp()
    q, k, _ = gen.make_qkv(1, 4, 1, 256, 2048, seed=23)
    k = k.clone()
    k[:, :, 5 * 128:6 * 128] = k[:, :, 2 * 128:3 * 128]
    k[:, :, 9 * 128:10 * 128] = k[:, :, 2 * 128:3 * 128]
    sel = m.SummarySelector(q.cuda(), k.cuda(), 4, topk=16)
    ids = sel.run().cpu()
    _, _, scores, ref = oracle.summary_select(q, k, 4, 16)
    assert torch.equal(ids, ref)
    pos = {int(v): i for i, v in enumerate(ids[0, 0, 0].tolist())}
    assert pos[2] + 1 == pos[5] and pos[5] + 1 == pos[9]


@pytest.mark.parametrize("family", ["row_scales_2^+-12", "cancellation_amplitude_64", "near_subnormal", "gaussian_long"])
def test_summary_tensor_core_bound_holds_on_stress_inputs(family):
    """Bit-exact ids of the tensor-core selector rest on |tcgen05 bf16 MMA score - canonical fp32 score| <=
    delta = 2^-14 * (bound on the sum of |q_d k_d|). Inputs that stress it: token rows scaled by powers of
    two between 2^-12 and 2^12 (descriptors of wildly different magnitude inside one list), the
    reference's cancellation_stress family at amplitude 64 (large terms that cancel), values next to
    the bf16 subnormal range, and long gaussian lists. The kernel compares both scores of every
    re-scored candidate: no violation may be counted, the largest observed difference must stay under
    a quarter of the bound, and the ids must equal the exact kernel's."""
    m = sp()
    b, hq, hkv, sq, skv, r, topk = 1, 8, 1, 160 * 128, 32768, 4, 32      # 160 lists: more than one per SM, so the tensor-core path runs
    g = torch.Generator().manual_seed(len(family))
    q = torch.randn((b, hq, sq, 128), generator=g)
    k = torch.randn((b, hkv, skv, 128), generator=g)
    if family == "row_scales_2^+-12":
        q = q * torch.exp2(torch.randint(-12, 13, (b, hq, sq, 1), generator=g).float())
        k = k * torch.exp2(torch.randint(-12, 13, (b, hkv, skv, 1), generator=g).float())
    elif family == "cancellation_amplitude_64":
        # benchmarks/ch4_selectors/reference.py:12-21: a large common component with alternating sign + small noise
        sign = torch.where(torch.arange(128) % 2 == 0, 1.0, -1.0)
        q = 64.0 * sign + 0.01 * q
        k = 64.0 + 0.01 * k
    elif family == "near_subnormal":
        q = q * 2.0 ** -60
        k = k * 2.0 ** -62
    # every KV block gets an identical twin in the second half of the sequence: all candidates come in exact
    # ties, so every one of them is re-scored and checked (lists whose ties straddle the candidate cut take
    # the exact fallback, as they must)
    k[:, :, skv // 2:] = k[:, :, :skv // 2]
    q, k = q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda()
    fast = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    ids = fast.run_fast().clone()
    exact = m.SummarySelector(q, k, r, topk=topk, keep_scores=False)
    exact.prepare()
    exact.score()
    torch.cuda.synchronize()
    m.device_status()
    violations, ratio = fast.bound_stats()
    print(f"{family}: fallback lists {fast.fallback_lists()}, violations {violations}, max |approx - exact| / delta {ratio:.3g}")
    assert torch.equal(ids, exact.ids)
    assert violations == 0
    assert ratio <= 0.25
    if family != "cancellation_amplitude_64":    # there bf16 rounds the noise away: every score is exactly 0 on both paths
        assert ratio > 0                         # > 0: candidates were re-scored, i.e. the check did run


def test_fp4_reference_gate_and_bit_exact():
    m = sp()
    fx = np.load(os.path.join(G, "fp4.npz"))
    qp, qs, kp, ks, b, lq, lkv = cases.fp4_case()
    inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=b, len_q=lq, len_kv=lkv)
    scores = m.fp4_block_scores(inputs)
    ids = m.tile_topk(scores, batch_size=b, len_q=lq, topk=16)
    torch.cuda.synchronize()
    # reference gate: scores rtol 1e-4 / atol 1e-3, ids exact
    np.testing.assert_allclose(scores.cpu().numpy(), fx["scores"], rtol=1e-4, atol=1e-3)
    np.testing.assert_array_equal(ids.cpu().numpy(), fx["ids"])
    # oracle: bit for bit
    ref = oracle.fp4_scores(qp, qs, kp, ks, b, lq, lkv)
    assert torch.equal(scores.cpu(), ref)
    # fused indexer: same ids, tile scores = max over the query tile
    tile = torch.empty((b, qp.shape[1], lq // 128, lkv // 128), device="cuda")
    ids2 = m.fp4_indexer(inputs, topk=16, tile_scores=tile)
    assert torch.equal(ids2.cpu(), ids.cpu())
    assert torch.equal(tile.cpu(), oracle.fp4_tile_scores(ref, b, lq))
    # top-k of other sizes
    for kk in (1, 5, 16):
        got = m.tile_topk(scores, batch_size=b, len_q=lq, topk=kk)
        assert torch.equal(got.cpu(), oracle.fp4_select(ref, b, lq, kk))


def test_nvfp4_quantiser_and_quantised_indexer():
    """bf16 -> NVFP4 (parity unpinned by the reference: checked against the stated
    rule in the oracle), then the configuration-4 flow at a small size:
    quantise Q (group mean) and K, score, top-k, KV-centric attention."""
    m = sp()
    b, hq, hkv, n, topk = 1, 16, 2, 1024, 4
    q, k, v = gen.make_qkv(b, hq, hkv, n, n, seed=41, k_block_offset=0.5)
    q[0, 0, 0, :16] = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0,
                                    -0.25, -0.75, -1.25, -1.75, -2.5, -3.5, -5.0, -6.0]).to(torch.bfloat16)
    qc, qs = m.quantize_queries(q.cuda(), hkv)
    kc, ks = m.quantize_keys(k.cuda())
    torch.cuda.synchronize()
    rqc, rqs = oracle.quantize_queries(q, hkv)
    rkc, rks = oracle.quantize_keys(k)
    assert torch.equal(qs.cpu().view(torch.uint8), rqs.view(torch.uint8))
    assert torch.equal(ks.cpu().view(torch.uint8), rks.view(torch.uint8))
    assert torch.equal(qc.cpu(), rqc) and torch.equal(kc.cpu(), rkc)
    inputs = m.prepare_fp4_inputs(qc, kc, qs, ks, batch_size=b, len_q=n, len_kv=n)
    ids = m.fp4_indexer(inputs, topk=topk)
    ref_scores = oracle.fp4_scores(rqc, rqs, rkc, rks, b, n, n)
    ref_ids = oracle.fp4_select(ref_scores, b, n, topk)
    assert torch.equal(ids.cpu(), ref_ids)
    out, lse = m.kv_centric_attention(q.cuda(), k.cuda(), v.cuda(), ids, nseg=2)
    ref_o, ref_l = oracle.gather_attention(q, k, v, ref_ids)
    d = (out.float().cpu() - ref_o).abs()
    assert d.max() <= 2e-2 and d.mean() <= 2e-3
    assert torch.all((lse.cpu() - ref_l).abs() <= 1e-3 * ref_l.abs().clamp_min(1.0))
    o2, sel2 = m.indexed_attention(q.cuda(), k.cuda(), v.cuda(), inputs, topk=topk)
    assert torch.equal(sel2.cpu(), ref_ids)
    assert (o2.float().cpu() - ref_o).abs().max() <= 2e-2
    m.device_status()


def test_fp4_tensor_core_path_bit_exact():
    """Tensor-core pre-filter + exact re-scoring must give the ids of the exact scorer."""
    m = sp()
    # random codes (the reference's synthetic family), one shared key head, 16 pages: all pages are candidates
    qp, qs, kp, ks, b, lq, lkv = cases.fp4_case()
    inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=b, len_q=lq, len_kv=lkv)
    ids, _ = m.fp4_indexer_fast(inputs, topk=16)
    fx = np.load(os.path.join(G, "fp4.npz"))
    np.testing.assert_array_equal(ids.cpu().numpy(), fx["ids"])
    # eight times more pages than candidates (the tensor-core path is taken only then), per-head
    # key pages, top-4 and top-24
    for (hidx, hk, lq, lkv, topk, seed) in [(2, 2, 256, 32768, 4, 5), (1, 1, 256, 49152, 24, 6)]:
        g = torch.Generator().manual_seed(seed)
        pages = lkv // 128
        qp = torch.randint(256, (lq, hidx, 64), dtype=torch.uint8, generator=g)
        kp = torch.randint(256, (pages, hk, 128, 64), dtype=torch.uint8, generator=g)
        choices = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.5, 2.0])
        qs = choices[torch.randint(7, (lq, hidx, 8), generator=g)].to(torch.float8_e4m3fn)
        ks = choices[torch.randint(7, (pages, hk, 128, 8), generator=g)].to(torch.float8_e4m3fn)
        inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=1, len_q=lq, len_kv=lkv)
        fn = m.lib().sparse_b200_indexer_fp4_workspace_bytes
        fn.restype = ctypes.c_int64
        need = fn(1, hidx, hk, lq, lkv)
        ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
        ids, ws = m.fp4_indexer_fast(inputs, topk=topk, workspace=ws)
        torch.cuda.synchronize()
        m.device_status()
        assert ws[:4].view(torch.int32).item() > 0         # CTAs of the tensor-core kernel: only that path counts them
        ref = oracle.fp4_select(oracle.fp4_scores(qp, qs, kp, ks, 1, lq, lkv), 1, lq, topk)
        assert torch.equal(ids.cpu(), ref)
        assert torch.equal(ids.cpu(), m.fp4_indexer(inputs, topk=topk).cpu())
        print("fallback tiles:", int(ws[4:8].view(torch.int32).item()))
    # quantised real data (configuration-4 flow) and exact ties (all-zero keys): lower id first
    q, k, _ = gen.make_qkv(1, 16, 2, 256, 32768, seed=43, k_block_offset=0.5)
    qc, qsc = m.quantize_queries(q.cuda(), 2)
    kc, ksc = m.quantize_keys(k.cuda())
    inputs = m.prepare_fp4_inputs(qc, kc, qsc, ksc, batch_size=1, len_q=256, len_kv=32768)
    ids, _ = m.fp4_indexer_fast(inputs, topk=8)
    assert torch.equal(ids.cpu(), m.fp4_indexer(inputs, topk=8).cpu())
    kc.zero_()
    ids, ws = m.fp4_indexer_fast(inputs, topk=8)
    assert torch.equal(ids.cpu(), torch.arange(8, dtype=torch.int32).expand_as(ids.cpu()))
    assert int(ws[4:8].view(torch.int32).item()) == ids.shape[1] * ids.shape[2]
    m.device_status()


@pytest.mark.parametrize("pages", [10672, 10673, 12001, 16304, 16384])
def test_fp4_selection_of_long_lists(pages):
    """Six pages in flight up to 10672 pages, four beyond; one CTA to an SM again beyond 16304: ids of the exact scorer."""
    m = sp()
    g = torch.Generator(device="cuda").manual_seed(pages)
    choices = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.5, 2.0], device="cuda")
    qp = torch.randint(256, (256, 2, 64), dtype=torch.uint8, generator=g, device="cuda")
    kp = torch.randint(256, (pages, 1, 128, 64), dtype=torch.uint8, generator=g, device="cuda")
    qs = choices[torch.randint(7, (256, 2, 8), generator=g, device="cuda")].to(torch.float8_e4m3fn)
    ks = choices[torch.randint(7, (pages, 1, 128, 8), generator=g, device="cuda")].to(torch.float8_e4m3fn)
    inputs = m.prepare_fp4_inputs(qp, kp, qs, ks, batch_size=1, len_q=256, len_kv=pages * 128)
    ids, ws = m.fp4_indexer_fast(inputs, topk=32)
    torch.cuda.synchronize()
    m.device_status()
    assert ws[:4].view(torch.int32).item() == 4          # CTAs of the tensor-core kernel
    assert torch.equal(ids, m.fp4_indexer(inputs, topk=32))


def _fast_path_tile_scores(ws, b, hidx, hk, lq, lkv):
    """Tile scores the fast entry left in its workspace: 256 bytes of statistics, then the scores."""
    n = b * hidx * (lq // 128) * (lkv // 128)
    return ws[256:256 + 4 * n].view(torch.float32).view(b, hidx, lq // 128, lkv // 128)


@pytest.mark.parametrize("case", ["random_codes", "shared_key_head", "zero_keys", "one_page", "many_pages_per_cta"])
def test_fp4_pruned_tile_scores_bit_exact(case):
    """Few pages per list: the fast entry computes exact tile scores by pruning each
    (query tile, page) pair with tensor-core values. Scores must equal those of the scorer that
    evaluates every element, bit for bit, and the ids those of the oracle."""
    m = sp()
    hidx, hk, lq, lkv, topk, seed = {"random_codes": (2, 2, 512, 4096, 16, 11), "shared_key_head": (4, 1, 256, 2048, 8, 12),
                                     "zero_keys": (1, 1, 256, 1024, 4, 13), "one_page": (1, 1, 128, 128, 1, 14),
                                     # 320 lists of 256 pages: one CTA per list, the warps agree on each pair's maximum
                                     "many_pages_per_cta": (4, 1, 10240, 32768, 64, 15)}[case]
    b = 2 if case == "random_codes" else 1
    g = torch.Generator().manual_seed(seed)
    pages = b * lkv // 128
    qp = torch.randint(256, (b * lq, hidx, 64), dtype=torch.uint8, generator=g)
    kp = torch.randint(256, (pages, hk, 128, 64), dtype=torch.uint8, generator=g)
    if case == "zero_keys":
        kp.zero_()
    choices = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.5, 2.0])
    qs = choices[torch.randint(7, (b * lq, hidx, 8), generator=g)].to(torch.float8_e4m3fn)
    ks = choices[torch.randint(7, (pages, hk, 128, 8), generator=g)].to(torch.float8_e4m3fn)
    inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=b, len_q=lq, len_kv=lkv)
    ids, ws = m.fp4_indexer_fast(inputs, topk=topk)
    exact_scores = torch.empty((b, hidx, lq // 128, lkv // 128), dtype=torch.float32, device="cuda")
    exact_ids = m.fp4_indexer(inputs, topk=topk, tile_scores=exact_scores)
    torch.cuda.synchronize()
    m.device_status()
    assert ws[:4].view(torch.int32).item() > 0            # CTAs of the pruning kernel: only that path counts them
    pruned = _fast_path_tile_scores(ws, b, hidx, hk, lq, lkv)
    assert torch.equal(pruned.view(torch.int32), exact_scores.view(torch.int32))
    assert torch.equal(ids, exact_ids)
    if case != "many_pages_per_cta":             # too large for the CPU oracle: the exact GPU scorer above stands in
        ref = oracle.fp4_select(oracle.fp4_scores(qp, qs, kp, ks, b, lq, lkv), b, lq, topk)
        assert torch.equal(ids.cpu(), ref)


def _long_run_inputs(m, pages, zero, seed=21):
    """160 lists of `pages` pages, one CTA of the pruning scorer per 3072 of them; pages `zero` all equal."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    choices = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.5, 2.0], device="cuda")

    def scales(*shape):
        return choices[torch.randint(7, shape, generator=g, device="cuda")].to(torch.float8_e4m3fn)
    qp = torch.randint(256, (2048, 10, 64), dtype=torch.uint8, generator=g, device="cuda")
    kp = torch.randint(256, (pages, 1, 128, 64), dtype=torch.uint8, generator=g, device="cuda")
    kp[list(zero)] = 0
    return m.prepare_fp4_inputs(qp, kp, scales(2048, 10, 8), scales(pages, 1, 128, 8), batch_size=1, len_q=2048,
                                len_kv=pages * 128)


@pytest.mark.parametrize("pages,topk,zero", [
    (24, 8, (0, 1, 2, 3, 12, 13, 14)),    # each queues its 1024 groups; ordinary pages behind them
    (40, 16, tuple(range(7, 40))),        # padding: only the first pages differ
    (2500, 200, ()),                      # more pages than the queue has room for
    (3100, 250, (1549, 1550, 3099)),      # more than one CTA takes
    (18300, 200, ()),                     # the results of all of a list's pages would not fit a CTA's shared memory
])
def test_fp4_pruned_scores_of_long_runs(pages, topk, zero):
    """The queue of the pruning scorer fills up, is emptied and fills up again: scores bit for bit those of the scorer that
    evaluates every element, the same ids."""
    m = sp()
    inputs = _long_run_inputs(m, pages, zero)
    ids, ws = m.fp4_indexer_fast(inputs, topk=topk)
    exact_scores = torch.empty((1, 10, 16, pages), dtype=torch.float32, device="cuda")
    exact_ids = m.fp4_indexer(inputs, topk=topk, tile_scores=exact_scores)
    torch.cuda.synchronize()
    m.device_status()
    assert ws[:4].view(torch.int32).item() == 160 * ((pages + 3071) // 3072)      # CTAs of the pruning kernel
    assert ws[12:16].view(torch.int32).item() == 0                                 # no bound was violated
    pruned = _fast_path_tile_scores(ws, 1, 10, 1, 2048, pages * 128)
    assert torch.equal(pruned.view(torch.int32), exact_scores.view(torch.int32))
    assert torch.equal(ids, exact_ids)


def test_fp4_pruning_full_queue_costs_little():
    """Neither a long run nor pages of equal scores make the pages behind them dear. An ordinary page takes about 1 us of the
    160 lists together, one that is evaluated in full 110 to 160 us: 2500 pages stay within twice the time per page of 1000
    (500 pages in full would take 55 ms), and six all-equal pages among 1000, in full themselves, take about as long as the
    other 994, which in full would take 100 times that."""
    m = sp()

    def us(pages, zero=()):
        inputs = _long_run_inputs(m, pages, zero)
        _, ws = m.fp4_indexer_fast(inputs, topk=160)
        best = float("inf")
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            m.fp4_indexer_fast(inputs, topk=160, workspace=ws)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best
    plain = us(1000)
    assert us(2500) < 2 * 2.5 * plain
    assert us(1000, (0, 1, 2, 500, 501, 502)) < 4 * plain


def _varlen_case(seed, hq, hk, q_lens, k_lens, shuffle_pages=True):
    g = torch.Generator().manual_seed(seed)
    total_q = sum(q_lens)
    pages_per = [(k + 127) // 128 for k in k_lens]
    total_pages = sum(pages_per) + 3                       # a few pages nobody owns
    qp = torch.randint(256, (total_q, hq, 64), dtype=torch.uint8, generator=g)
    kp = torch.randint(256, (total_pages, hk, 128, 64), dtype=torch.uint8, generator=g)
    choices = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.5, 2.0])
    qs = choices[torch.randint(7, (total_q, hq, 8), generator=g)].to(torch.float8_e4m3fn)
    ks = choices[torch.randint(7, (total_pages, hk, 128, 8), generator=g)].to(torch.float8_e4m3fn)
    perm = torch.randperm(total_pages, generator=g) if shuffle_pages else torch.arange(total_pages)
    kv_indices = perm[:sum(pages_per)].to(torch.int32)
    cu = lambda xs: torch.tensor([0] + list(np.cumsum(xs)), dtype=torch.int32)
    return qp, qs, kp, ks, cu(q_lens), cu(k_lens), cu(pages_per), kv_indices


@pytest.mark.parametrize("causal", [False, True])
def test_fp4_scores_ragged_paged_causal(causal):
    """Ragged requests over a shuffled page table (lengths that are no multiples of 128, a request
    with more queries than keys, GQA 4:1, a single-token decode request), optionally causal, with
    and without an explicit causal offset: bit-exact against the oracle, -inf outside."""
    m = sp()
    q_lens, k_lens = [200, 128, 1, 300, 77], [1000, 128, 517, 260, 64]
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(11, 4, 1, q_lens, k_lens)
    offsets = [None] + ([torch.tensor([800, 0, 516, -50, 10], dtype=torch.int32)] if causal else [])
    for qo in offsets:
        ref = oracle.fp4_scores_varlen(qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx, max(k_lens), causal=causal,
                                       qo_offset=qo)
        out = m.fp4_block_scores_varlen(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), cu_q.cuda(), cu_k.cuda(),
                                        cu_p.cuda(), max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens),
                                        kv_indices=kv_idx.cuda(), causal=causal,
                                        qo_offset=None if qo is None else qo.cuda())
        torch.cuda.synchronize()
        m.device_status()
        assert out.shape == ref.shape
        assert torch.equal(out.cpu(), ref)
    # a dense, unshuffled batch equals the dense scorer bit for bit
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(12, 2, 2, [256, 256], [512, 512], shuffle_pages=False)
    if not causal:
        kp, ks = kp[:8].contiguous(), ks[:8].contiguous()
        inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=2, len_q=256, len_kv=512)
        dense = m.fp4_block_scores(inputs)
        ragged = m.fp4_block_scores_varlen(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), cu_q.cuda(), cu_k.cuda(),
                                           cu_p.cuda(), max_seqlen_q=256, max_seqlen_k=512, kv_indices=kv_idx.cuda())
        assert torch.equal(dense, ragged)


@pytest.mark.parametrize("heads", [(16, 1), (8, 2), (32, 1), (3, 3)])
@pytest.mark.parametrize("causal", [False, True])
def test_fp4_scores_decode_batches(heads, causal):
    """Decode batches (at most 8 new queries per request): the packed form of the scorer, rows =
    (group head, query) pairs, for group sizes 16 (the reference's decode case), 4, 32 (two blocks of
    16 heads) and 1 (not packed). Bit-exact against the oracle, -inf outside."""
    m = sp()
    hq, hk = heads
    q_lens, k_lens = [1, 8, 3, 5], [1000, 517, 128, 2048]
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(51 + hq, hq, hk, q_lens, k_lens)
    ref = oracle.fp4_scores_varlen(qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx, max(k_lens), causal=causal)
    out = m.fp4_block_scores_varlen(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), cu_q.cuda(), cu_k.cuda(), cu_p.cuda(),
                                    max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(),
                                    causal=causal)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(out.cpu(), ref)
    # the same requests declared as a prefill batch (max_seqlen_q = 128) take the unpacked form: same scores
    out2 = m.fp4_block_scores_varlen(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), cu_q.cuda(), cu_k.cuda(), cu_p.cuda(),
                                     max_seqlen_q=128, max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal)
    assert torch.equal(out2, out)


def _assert_within_reference_gate(mine, exact, what):
    """Finite scores within the reference's own gate (rtol 1e-4, atol 1e-3,
    benchmarks/ch4_selectors/harness.py:33-42), identical -inf pattern."""
    assert mine.shape == exact.shape, what
    assert torch.equal(torch.isinf(mine), torch.isinf(exact)), what
    fin = torch.isfinite(exact)
    np.testing.assert_allclose(mine[fin].numpy(), exact[fin].numpy(), rtol=1e-4, atol=1e-3, err_msg=what)


@pytest.mark.parametrize("causal", [False, True])
def test_fp4_scores_on_the_tensor_cores_ragged_decode_dense(causal):
    """The NVFP4-MMA scorer (per-query page scores straight off tcgen05 block-scaled MMAs, query tile as the M
    operand) against the exact scorer: ragged prefill batch with explicit causal offsets, decode batches of
    several group sizes (packed rows), an out-of-range page-table entry, and a dense batch."""
    m = sp()
    q_lens, k_lens = [200, 128, 1, 300, 77], [1000, 128, 517, 260, 64]
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(11, 4, 1, q_lens, k_lens)
    kv_bad = kv_idx.clone()
    kv_bad[2] = 10 ** 6                                     # page 2 of request 0 does not exist: stays -inf
    offsets = [None] + ([torch.tensor([800, 0, 516, -50, 10], dtype=torch.int32)] if causal else [])
    dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
    for table in (kv_idx, kv_bad):
        for qo in offsets:
            kw = dict(max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=table.cuda(), causal=causal,
                      qo_offset=None if qo is None else qo.cuda())
            exact = m.fp4_block_scores_varlen(*dev, **kw)
            fast = m.fp4_block_scores_varlen(*dev, exact=False, **kw)
            torch.cuda.synchronize()
            m.device_status()
            _assert_within_reference_gate(fast.cpu(), exact.cpu(), f"ragged causal={causal}")
    for hq, hk in ((16, 1), (8, 2), (32, 1), (3, 3)):
        q_lens, k_lens = [1, 8, 3, 5], [1000, 517, 128, 2048]
        qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(51 + hq, hq, hk, q_lens, k_lens)
        dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
        kw = dict(max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal)
        exact = m.fp4_block_scores_varlen(*dev, **kw)
        fast = m.fp4_block_scores_varlen(*dev, exact=False, **kw)
        torch.cuda.synchronize()
        m.device_status()
        _assert_within_reference_gate(fast.cpu(), exact.cpu(), f"decode Hq{hq}/Hk{hk} causal={causal}")
    if not causal:
        qp, qs, kp, ks, b, lq, lkv = cases.fp4_case()
        inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=b, len_q=lq, len_kv=lkv)
        _assert_within_reference_gate(m.fp4_block_scores(inputs, exact=False).cpu(), m.fp4_block_scores(inputs).cpu(), "dense")
        fx = np.load(os.path.join(G, "fp4.npz"))
        np.testing.assert_allclose(m.fp4_block_scores(inputs, exact=False).cpu().numpy(), fx["scores"], rtol=1e-4, atol=1e-3)
        m.device_status()


@pytest.mark.parametrize("causal", [False, True])
def test_fp4_varlen_scores_against_the_reference_scorer(causal):
    """Pins the ragged / paged / causal contract to the reference's own kernel: the vendored MiniMax
    MSA scorer (indexers/fp4/vendor_minimax_msa/fp4_indexer_interface.py:745-1056, copied unmodified
    into the git-ignored baseline/_ref/fp4 by baseline/build_reference_kernels.py) on the same ragged
    batch, public scale layout. Its scores come from NVFP4 MMAs in the tensor core's own accumulation
    order, so they are compared with the reference's own gate tolerance (rtol 1e-4, atol 1e-3,
    benchmarks/ch4_selectors/harness.py:33-42); the -inf pattern must be identical. The CPU oracle is
    held to the same comparison, which is what pins it."""
    vendor = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "baseline", "_ref", "fp4",
                          "vendor_minimax_msa")
    if not os.path.isdir(vendor):
        pytest.skip("reference sources not present under baseline/_ref/fp4 (python baseline/build_reference_kernels.py --ref ...)")
    import sys
    sys.path.insert(0, vendor)
    try:
        from fp4_indexer_interface import fp4_indexer_block_scores
    except Exception as e:                                  # nvidia-cutlass-dsl missing or unusable here
        pytest.skip(f"the vendored scorer does not import: {type(e).__name__}: {e}")
    finally:
        sys.path.remove(vendor)
    m = sp()
    cases = [((4, 1), [200, 128, 300, 77], [1000, 128, 260, 64]),      # prefill-like, ragged
             ((16, 1), [1, 8, 3, 5], [1000, 517, 128, 2048])]         # decode, group 16 (its packed-Q kernel)
    for (hq, hk), q_lens, k_lens in cases:
        qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(61 + hq, hq, hk, q_lens, k_lens)
        dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
        theirs = fp4_indexer_block_scores(dev[0], dev[1], dev[2], dev[3], dev[4], dev[5], dev[6],
                                          max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(),
                                          fp4_format="nvfp4", causal=causal, scale_layout="public")
        ours = m.fp4_block_scores_varlen(dev[0], dev[1], dev[2], dev[3], dev[4], dev[5], dev[6], max_seqlen_q=max(q_lens),
                                         max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal)
        torch.cuda.synchronize()
        fast = m.fp4_block_scores_varlen(dev[0], dev[1], dev[2], dev[3], dev[4], dev[5], dev[6], max_seqlen_q=max(q_lens),
                                         max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal, exact=False)
        torch.cuda.synchronize()
        ref = oracle.fp4_scores_varlen(qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx, max(k_lens), causal=causal)
        assert theirs.shape == ours.shape == ref.shape
        for name, mine in (("kernel", ours.cpu()), ("tensor-core kernel", fast.cpu()), ("oracle", ref)):
            t = theirs.cpu()
            assert torch.equal(torch.isinf(t), torch.isinf(mine)), name
            fin = torch.isfinite(t)
            np.testing.assert_allclose(mine[fin].numpy(), t[fin].numpy(), rtol=1e-4, atol=1e-3, err_msg=name)
    m.device_status()


@pytest.mark.parametrize("requests,hq,hk,q_hi,k_hi,causal,offsets", [
    (1, 1, 1, 1, 100, False, False),           # one page: one CTA has a run, the others none
    (3, 6, 2, 300, 700, True, False),          # heads of a group and query tiles follow each other within a run
    (70, 3, 3, 40, 900, True, True),           # more requests than a warp has lanes, some of them empty
    (45, 40, 2, 8, 1500, True, False),         # packed rows, two blocks of heads per KV head
    (33, 16, 1, 5, 6000, False, False),        # packed, more than 32 pages per item
    (2, 2, 1, 4500, 5200, True, True),         # more than 32 query tiles
])
def test_fp4_varlen_runs_of_pages(requests, hq, hk, q_hi, k_hi, causal, offsets):
    """The tensor-core scorer cuts the pages of all (request, tile, head) items into equal runs on the device: against the
    exact scorer, which takes item by item. Same -inf pattern; finite scores within the bound on the tensor core's sums,
    2^-18 of (largest L1 norm of a query) x (largest key element), at most 128 * 6 * 6 * the largest scales."""
    m = sp()
    rng = np.random.RandomState(requests * 31 + hq)
    q_lens = [int(x) for x in rng.randint(1, q_hi + 1, requests)]
    k_lens = [int(x) for x in rng.randint(1, k_hi + 1, requests)]
    if requests > 2:
        q_lens[1] = 0                          # nothing to score
        k_lens[2] = 1
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(5 + requests, hq, hk, q_lens, k_lens)
    if requests > 1:
        kv_idx[0] = kp.shape[0] + 3            # out of range: that page stays -inf
    dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
    kw = dict(max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal)
    if offsets:
        kw["qo_offset"] = torch.from_numpy(rng.randint(-100, 600, requests).astype(np.int32)).cuda()
    exact = m.fp4_block_scores_varlen(*dev, **kw)
    for _ in range(2):
        fast = m.fp4_block_scores_varlen(*dev, exact=False, **kw)
        torch.cuda.synchronize()
        m.device_status()
        assert torch.equal(torch.isinf(exact), torch.isinf(fast))
        fin = torch.isfinite(exact)
        scale = max(float(qs.float().max()) * float(ks.float().max()), 1.0)
        assert (exact[fin] - fast[fin]).abs().max().item() <= 128 * 36 * scale * 2.0 ** -18


@pytest.mark.parametrize("requests,hq,hk,q_hi,causal", [
    (224, 16, 1, 8, True),                     # one request to a thread of the CTA that looks for its run
    (225, 4, 2, 150, True),                    # two
    (1000, 16, 1, 1, False),
    (7400, 2, 2, 3, True),                     # more than a warp has lanes
])
def test_fp4_varlen_runs_of_many_requests(requests, hq, hk, q_hi, causal):
    """As test_fp4_varlen_runs_of_pages, by the number of requests; many of them empty or without a visible page."""
    m = sp()
    rng = np.random.RandomState(requests)
    q_lens = [int(x) for x in rng.randint(0, q_hi + 1, requests)]
    k_lens = [int(x) for x in rng.randint(0, 400, requests)]
    q_lens[0] = q_lens[-1] = q_hi
    k_lens[0] = k_lens[-1] = 390
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(requests, hq, hk, q_lens, k_lens)
    dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
    kw = dict(max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), kv_indices=kv_idx.cuda(), causal=causal)
    exact = m.fp4_block_scores_varlen(*dev, **kw)
    fast = m.fp4_block_scores_varlen(*dev, exact=False, **kw)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(torch.isinf(exact), torch.isinf(fast))
    fin = torch.isfinite(exact)
    scale = max(float(qs.float().max()) * float(ks.float().max()), 1.0)
    assert fin.any() and (exact[fin] - fast[fin]).abs().max().item() <= 128 * 36 * scale * 2.0 ** -18


@pytest.mark.parametrize("requests,hq,hk,q_hi,k_hi,causal", [
    (1, 16, 1, 1, 200, True),                  # one CTA
    (5, 40, 2, 8, 1500, True),                 # two blocks of heads to a KV head, shares of two pages, the last ones empty
    (9, 6, 3, 300, 700, True),                 # query tiles and heads; requests shorter than the longest
    (37, 16, 1, 1, 4000, False),               # 592 CTAs: the last size of a launch without runs
    (38, 16, 1, 1, 4000, False),               # 608: the first with runs
    (2368, 16, 1, 3, 500, True),               # one item to a request, few pages: as many CTAs as requests
    (2369, 16, 1, 3, 500, True),               # and one more
])
def test_fp4_varlen_shares_of_an_item(requests, hq, hk, q_hi, k_hi, causal):
    """Launches whose CTAs take shares of an item's pages, and those next to them that take runs, against the exact scorer
    (bound as in test_fp4_varlen_runs_of_pages)."""
    m = sp()
    rng = np.random.RandomState(requests)
    q_lens = [int(x) for x in rng.randint(0 if requests > 4 else 1, q_hi + 1, requests)]
    k_lens = [int(x) for x in rng.randint(1, k_hi + 1, requests)]
    q_lens[-1], k_lens[-1] = q_hi, k_hi
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(requests + 1, hq, hk, q_lens, k_lens)
    dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
    kw = dict(max_seqlen_q=q_hi, max_seqlen_k=k_hi, kv_indices=kv_idx.cuda(), causal=causal)
    exact = m.fp4_block_scores_varlen(*dev, **kw)
    fast = m.fp4_block_scores_varlen(*dev, exact=False, **kw)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(torch.isinf(exact), torch.isinf(fast))
    fin = torch.isfinite(exact)
    scale = max(float(qs.float().max()) * float(ks.float().max()), 1.0)
    assert fin.any() and (exact[fin] - fast[fin]).abs().max().item() <= 128 * 36 * scale * 2.0 ** -18


def test_fp4_varlen_start_up_with_many_requests():
    """A CTA finds its run of pages without a walk over all requests: 16384 requests of one page each take no more than six
    times what the same pages take as 64 requests (2.6 measured, more than 10 with a walk over all requests by one warp)."""
    m = sp()

    def us(requests, pages):
        q_lens, k_lens = [1] * requests, [128 * pages] * requests
        qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(3, 16, 1, q_lens, k_lens)
        dev = [t.cuda() for t in (qp, kp, qs, ks, cu_q, cu_k, cu_p)]
        kw = dict(max_seqlen_q=1, max_seqlen_k=128 * pages, kv_indices=kv_idx.cuda(), causal=True, exact=False)
        best = float("inf")
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            m.fp4_block_scores_varlen(*dev, **kw)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best
    few, many = us(64, 256), us(16384, 1)
    print(f"64 requests {few:.1f} us, 16384 requests {many:.1f} us")
    assert many <= 6 * few


def test_fp4_scores_varlen_inconsistent_lengths_stay_in_bounds():
    """max_seqlen_k smaller than one request's key length, a page table shorter than the key
    length claims, and cu_seqlens_q that runs past total_q: the kernel must skip what does not fit.
    The output (sized from max_seqlen_k) sits inside a larger poisoned buffer, so a write outside it,
    or into another head's rows for pages past the output's page axis, shows up."""
    m = sp()
    q_lens, k_lens = [130, 64], [700, 256]
    qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx = _varlen_case(21, 2, 1, q_lens, k_lens)
    short = 384                                            # 3 pages of output; request 0 has 6 pages of keys
    hq, total_q = 2, sum(q_lens)
    tiles = (short + 127) // 128
    ref_full = oracle.fp4_scores_varlen(qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx, max(k_lens))
    L = m.lib()
    guard = 4096
    buf = torch.full((guard + hq * tiles * total_q + guard,), 12345.0, device="cuda")
    out = buf[guard:guard + hq * tiles * total_q]
    args = [t.cuda() for t in (qp, qs, kp, ks, cu_q, cu_k, cu_p, kv_idx)]
    from sparse_attention_b200_b200 import _lib
    rc = L.sparse_b200_fp4_scores_varlen(*[_lib.ptr(t) for t in args], None, _lib.ptr(out), 2, hq, 1, total_q,
                                         int(kp.shape[0]), max(q_lens), short, 0, _lib.current_stream())
    assert rc == 0
    torch.cuda.synchronize()
    m.device_status()
    assert torch.all(buf[:guard] == 12345.0) and torch.all(buf[-guard:] == 12345.0)
    got = out.view(hq, tiles, total_q).cpu()
    assert torch.equal(got[:, :, :q_lens[0]], ref_full[:, :tiles, :q_lens[0]])      # the pages that fit are right
    assert torch.equal(got[:, :2, q_lens[0]:], ref_full[:, :2, q_lens[0]:])
    # a page table that ends before the key length says, and queries claimed past total_q
    cu_p_short = cu_p.clone()
    cu_p_short[1:] -= 2                                    # request 0 now owns 4 pages for 700 keys
    cu_q_long = cu_q.clone()
    cu_q_long[-1] += 500
    buf.fill_(12345.0)
    rc = L.sparse_b200_fp4_scores_varlen(_lib.ptr(args[0]), _lib.ptr(args[1]), _lib.ptr(args[2]), _lib.ptr(args[3]),
                                         _lib.ptr(cu_q_long.cuda()), _lib.ptr(args[5]), _lib.ptr(cu_p_short.cuda()),
                                         _lib.ptr(args[7]), None, _lib.ptr(out), 2, hq, 1, total_q, int(kp.shape[0]),
                                         max(q_lens) + 500, short, 0, _lib.current_stream())
    assert rc == 0
    torch.cuda.synchronize()
    m.device_status()
    assert torch.all(buf[:guard] == 12345.0) and torch.all(buf[-guard:] == 12345.0)


def test_indexer_then_attention_config1():
    """Configuration 1 end to end: R1 picks top-8 of 32, Q-centric attention,
    against the masked-attention oracle."""
    m = sp()
    q, k, v = gen.make_qkv(1, 8, 8, 4096, 4096, seed=17, k_block_offset=0.5)
    sel = m.SummarySelector(q.cuda(), k.cuda(), 1, topk=8)
    ids = sel.run()
    ref_ids = oracle.summary_select(q, k, 1, 8)[3]
    assert torch.equal(ids.cpu(), ref_ids)
    out, lse = m.attention(q.cuda(), k.cuda(), v.cuda(), ids, return_lse=True)
    ref_o, ref_l = oracle.masked_attention(q, k, v, ref_ids)
    d = (out.float().cpu() - ref_o).abs()
    assert d.max() <= 2e-2 and d.mean() <= 2e-3
    assert torch.all((lse.cpu() - ref_l).abs() <= 1e-3 * ref_l.abs().clamp_min(1.0))


@pytest.mark.parametrize("sq", [1024, 80 * 128])      # 16 lists: the small-problem selector; 160 lists: the persistent one
def test_indexer_attention_pipeline_in_a_cuda_graph(sq):
    """Indexer -> attention as one call, captured once and replayed after the inputs changed:
    new exact ids and a correct output must come out of the replay (the reference's gate,
    benchmarks/ch4_selectors/harness.py:105-111)."""
    m = sp()
    q, k, v = gen.make_qkv(1, 16, 2, sq, 8192, seed=61, k_block_offset=0.5)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    sel = m.SummarySelector(qc, kc, 4, topk=16, keep_scores=False)
    out = torch.empty_like(qc)
    lse = torch.empty(qc.shape[:3], device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        m.summary_indexed_attention_out(sel, vc, out, lse)           # eager call first
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        m.summary_indexed_attention_out(sel, vc, out, lse)
    torch.cuda.synchronize()
    for shift in (0, 128, 384):
        with torch.cuda.stream(stream):
            qc.copy_(q.cuda().roll(shift, dims=2))
            sel.ids.fill_(-1)
            out.fill_(float("nan"))
            graph.replay()
        stream.synchronize()
        ref_ids = oracle.summary_select(qc.cpu(), k, 4, 16)[3]
        assert torch.equal(sel.ids.cpu(), ref_ids)
        ref_o, ref_l = oracle.gather_attention(qc.cpu(), k, v, ref_ids)
        d = (out.float().cpu() - ref_o).abs()
        assert d.max() <= 2e-2 and d.mean() <= 2e-3
        assert torch.all((lse.cpu() - ref_l).abs() <= 1e-3 * ref_l.abs().clamp_min(1.0))
    m.device_status()


def _fp4_stats(ws):
    """(tiles on the exact path, bound violations, largest |tensor-core value - exact| / bound)."""
    w = ws[:20].cpu()
    return int(w[4:8].view(torch.int32)), int(w[12:16].view(torch.int32)), float(w[16:20].view(torch.float32))


@pytest.mark.parametrize("family", ["full_scale_range", "huge_and_tiny_groups", "largest_codes"])
@pytest.mark.parametrize("lkv", [4096, 32768])
def test_fp4_tensor_core_bound_holds_on_stress_inputs(family, lkv):
    """The NVFP4 MMA accumulates the eight scaled group sums of a dot in its own order and
    precision; bit-exact ids rest on |tensor-core value - canonical value| <= delta. Inputs that
    stress that: scales over the whole e4m3 range (2^-9 .. 448, a spread of 2^17 between the
    groups of one vector), vectors whose groups alternate between the largest and the smallest
    scales (cancellation of large terms), and all codes at +-6. The kernels compare both values
    wherever they have them: no violation may be counted, the largest observed difference must
    stay under a quarter of the bound, and the ids must equal the exact scorer's (4096 keys: the
    pruning path; 32768 keys: the page pre-filter)."""
    m = sp()
    hidx, lq, topk = 2, 256, 8
    g = torch.Generator().manual_seed({"full_scale_range": 31, "huge_and_tiny_groups": 32, "largest_codes": 33}[family] + lkv)
    pages = lkv // 128
    qp = torch.randint(256, (lq, hidx, 64), dtype=torch.uint8, generator=g)
    kp = torch.randint(256, (pages, hidx, 128, 64), dtype=torch.uint8, generator=g)
    if family == "largest_codes":            # magnitude code 7 (= 6.0) everywhere, random signs
        qp, kp = qp | 0x77, kp | 0x77
    if family == "huge_and_tiny_groups":
        big, small = 0x7E, 0x01              # 448 and 2^-9
        pat = torch.tensor([big, small] * 4, dtype=torch.uint8)
        qs = pat.expand(lq, hidx, 8).clone()
        ks = torch.where(torch.rand((pages, hidx, 128, 1), generator=g) < 0.5, pat, pat.flip(0)).contiguous()
    else:
        qs = torch.randint(0, 0x7F, (lq, hidx, 8), generator=g).to(torch.uint8)
        ks = torch.randint(0, 0x7F, (pages, hidx, 128, 8), generator=g).to(torch.uint8)
    qs, ks = qs.view(torch.float8_e4m3fn), ks.view(torch.float8_e4m3fn)
    inputs = m.prepare_fp4_inputs(qp.cuda(), kp.cuda(), qs.cuda(), ks.cuda(), batch_size=1, len_q=lq, len_kv=lkv)
    ids, ws = m.fp4_indexer_fast(inputs, topk=topk)
    exact = m.fp4_indexer(inputs, topk=topk)
    torch.cuda.synchronize()
    m.device_status()
    fallbacks, violations, ratio = _fp4_stats(ws)
    print(f"{family}/{lkv}: exact-path tiles {fallbacks}, violations {violations}, max |approx - exact| / delta {ratio:.3g}")
    assert torch.equal(ids, exact)
    assert violations == 0
    assert ratio <= 0.25
    if lkv == 4096:
        ref = oracle.fp4_select(oracle.fp4_scores(qp, qs, kp, ks, 1, lq, lkv), 1, lq, topk)
        assert torch.equal(ids.cpu(), ref)


def test_fp4_pipeline_one_call_in_a_cuda_graph():
    """quantise -> NVFP4 indexer -> top-k -> attention as ONE C call with caller-owned buffers,
    captured once and replayed after the inputs changed (the reference's gate,
    benchmarks/ch4_selectors/harness.py:105-111): exact ids, output within tolerance."""
    m = sp()
    b, hq, hkv, sq, skv, topk = 1, 8, 2, 256, 32768, 8
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=71, k_block_offset=0.5)
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    pipe = m.Fp4Pipeline(qc, kc, vc, topk=topk)
    out = torch.empty_like(qc)
    lse = torch.empty(qc.shape[:3], device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        pipe.run(out, lse)                                   # eager call first
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        pipe.run(out, lse)
    torch.cuda.synchronize()
    rkc, rks = oracle.quantize_keys(k)
    for shift in (0, 128):
        with torch.cuda.stream(stream):
            qc.copy_(q.cuda().roll(shift, dims=2))
            pipe.ids.fill_(-1)
            out.fill_(float("nan"))
            graph.replay()
        stream.synchronize()
        qh = qc.cpu()
        rqc, rqs = oracle.quantize_queries(qh, hkv)
        ref_ids = oracle.fp4_select(oracle.fp4_scores(rqc, rqs, rkc, rks, b, sq, skv), b, sq, topk)
        assert torch.equal(pipe.ids.cpu(), ref_ids)
        ref_o, ref_l = oracle.gather_attention(qh, k, v, ref_ids)
        d = (out.float().cpu() - ref_o).abs()
        assert d.max() <= 2e-2 and d.mean() <= 2e-3
        assert torch.all((lse.cpu() - ref_l).abs() <= 1e-3 * ref_l.abs().clamp_min(1.0))
        assert pipe.stats()[1] == 0
    # prepared inputs (the reference's form of the call): same ids through the same entry
    inputs = m.prepare_fp4_inputs(pipe.qc, pipe.kc, pipe.qs, pipe.ks, batch_size=b, len_q=sq, len_kv=skv)
    o2, ids2 = m.indexed_attention(qc, kc, vc, inputs, topk=topk)
    assert torch.equal(ids2, pipe.ids) and torch.equal(o2, out)
    m.device_status()


def test_rejected_indexer_inputs():
    m = sp()
    q, k, _ = gen.make_qkv(1, 4, 2, 256, 512, seed=1)
    with pytest.raises(ValueError):
        m.SummarySelector(q.cuda(), k.cuda(), 3)
    with pytest.raises(ValueError):
        m.SummarySelector(q.cuda(), k.cuda(), 1, topk=5)
    with pytest.raises(ValueError):
        m.SummarySelector(q.float().cuda(), k.cuda(), 1, topk=2)
    scores = torch.zeros((1, 4, 256), device="cuda")
    with pytest.raises(RuntimeError):
        m.tile_topk(scores, batch_size=1, len_q=256, topk=5)
    with pytest.raises(RuntimeError):
        m.tile_topk(scores.double(), batch_size=1, len_q=256, topk=2)
