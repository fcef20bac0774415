"""Q-centric kernel through the C ABI against the CPU oracle (B200 only).

Tolerances: O max-abs 2e-2 and mean-abs 2e-3 against the fp32 oracle, LSE
within 1e-3 relative (and inside the reference's own atol 0.002 / rtol 0.0002,
attention/kv_centric/validate_gpu.py:12-13). Cases follow the reference gate
list (attention/q_centric/progression_validation.py:82-104)."""
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


def check(out, lse, ref_o, ref_l, o_max=2e-2, o_mean=2e-3):
    o = out.float().cpu()
    assert torch.isfinite(o).all()
    d = (o - ref_o).abs()
    assert d.max().item() <= o_max, d.max().item()
    assert d.mean().item() <= o_mean, d.mean().item()
    if lse is not None:
        l = lse.cpu()
        fin = torch.isfinite(ref_l)
        assert torch.equal(torch.isinf(l) & (l < 0), ~fin)
        err = (l[fin] - ref_l[fin]).abs()
        assert torch.all(err <= 1e-3 * ref_l[fin].abs().clamp_min(1.0))
        assert torch.all(err <= 0.002 + 0.0002 * ref_l[fin].abs())
    return d.max().item()


def run(q, k, v, ids, counts=None):
    m = sp()
    out = torch.full(q.shape, float("nan"), dtype=torch.bfloat16, device="cuda")
    lse = torch.full(q.shape[:3], float("nan"), device="cuda")
    m.attention_out(q.cuda(), k.cuda(), v.cuda(), ids.cuda(), out,
                    None if counts is None else counts.cuda(), lse)
    torch.cuda.synchronize()
    m.device_status()
    return out, lse


CASES = [
    # (B, Hq, Hkv, Sq, Skv), topk, pattern, scale
    ((1, 2, 2, 256, 128), 1, "independent", 1.0),
    ((1, 2, 2, 512, 512), 2, "reverse", 0.25),
    ((2, 4, 2, 256, 512), 3, "unsorted", 1.0),
    ((1, 8, 2, 512, 2048), 16, "reverse", 1.0),
    ((1, 16, 2, 512, 4096), 16, "unsorted", 2.0),
    ((1, 32, 2, 256, 4096), 16, "independent", 4.0),
    ((1, 2, 2, 512, 4096), 32, "reverse", 1.0),
    ((1, 4, 2, 128, 128), 1, "independent", 1.0),
    ((1, 8, 2, 384, 512), 3, "reverse", 1.0),
    ((1, 3, 3, 384, 512), 4, "unsorted", 1.0),      # odd tile count, MHA
    ((1, 6, 2, 256, 1024), 5, "unsorted", 1.0),     # odd group size 3
    ((2, 16, 16, 2048, 2048), 16, "independent", 1.0),
    ((2, 16, 1, 1024, 8192), 16, "paired", 1.0),
]


@pytest.mark.parametrize("shape,topk,pattern,scale", CASES)
def test_against_oracle(shape, topk, pattern, scale):
    b, hq, hkv, sq, skv = shape
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=1700 + topk, scale=scale)
    ids = gen.make_ids(b, hkv, sq // 128, skv // 128, topk, 2300 + topk, pattern)
    ref_o, ref_l = oracle.gather_attention(q, k, v, ids)
    out, lse = run(q, k, v, ids)
    check(out, lse, ref_o, ref_l)


def test_golden_fixtures():
    """Directly against the reference's stored outputs."""
    fx = np.load(os.path.join(G, "attention_masked.npz"))
    q, k, v, ids = cases.attention_masked_case()
    out, lse = run(q, k, v, ids)
    check(out, lse, torch.from_numpy(fx["o"]), torch.from_numpy(fx["lse"]))
    fx = np.load(os.path.join(G, "attention_gather.npz"))
    for i, (q, k, v, ids) in enumerate(cases.attention_gather_cases()):
        out, _ = run(q, k, v, ids)
        check(out, None, torch.from_numpy(fx[f"o{i}"]), None)


def test_config1_shape():
    """B=1, Hq=Hkv=8, N=4096, top-8, K with per-block offsets, masked oracle."""
    q, k, v = gen.make_qkv(1, 8, 8, 4096, 4096, seed=17, k_block_offset=0.5)
    ids = gen.make_ids(1, 8, 32, 32, 8, 1017, "unsorted")
    ref_o, ref_l = oracle.masked_attention(q, k, v, ids)
    out, lse = run(q, k, v, ids)
    check(out, lse, ref_o, ref_l)


def test_counts_and_empty_lists():
    q, k, v = gen.make_qkv(1, 4, 2, 512, 512, seed=5)
    ids = gen.make_ids(1, 2, 4, 4, 3, 6, "unsorted")
    counts = torch.tensor([[[3, 0, 1, 2], [2, 3, 0, 1]]], dtype=torch.int32)
    for hq in (4, 2):   # pair mode and split mode
        qq = q[:, :hq].contiguous()
        ref_o, ref_l = oracle.gather_attention(qq, k, v, ids, counts)
        out, lse = run(qq, k, v, ids, counts)
        check(out, lse, ref_o, ref_l)
        assert torch.all(out[0, :, 128:256][: hq // 2] == 0)


def test_analytic_cases():
    """validate_gpu.py:49-73: constant V gives the constant; zero Q gives the
    uniform softmax with LSE = ln(#keys); selecting every block equals dense."""
    q, k, v = gen.make_qkv(1, 16, 1, 256, 2048, seed=42)
    ids = gen.make_ids(1, 1, 2, 16, 16, 43, "unsorted")      # all 16 blocks
    vc = torch.full_like(v, 3.0)
    out, lse = run(q, k, vc, ids)
    assert torch.allclose(out.float().cpu(), torch.full(q.shape, 3.0), atol=2e-2)
    out, lse = run(torch.zeros_like(q), k, v, ids)
    assert torch.allclose(lse.cpu(), torch.full(q.shape[:3], float(np.log(2048.0))), atol=1e-3)
    assert torch.allclose(out.float().cpu(), v.float().mean(dim=2, keepdim=True).expand(1, 16, 256, 128)
                          .contiguous(), atol=2e-2)
    dense = torch.softmax(q.float() @ k.float().transpose(-1, -2) / 128 ** 0.5, -1) @ v.float()
    out, _ = run(q, k, v, ids)
    check(out, None, dense, None)


def test_out_api_repeat_bitwise_and_nondefault_stream():
    m = sp()
    q, k, v = gen.make_qkv(2, 16, 2, 1024, 4096, seed=601)
    ids = gen.make_ids(2, 2, 8, 32, 16, 601, "unsorted")
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    a = m.attention(qc, kc, vc, ic)
    b = torch.full_like(qc, float("nan"))
    m.attention_out(qc, kc, vc, ic, b)
    assert torch.equal(a, b)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        c = m.attention(qc, kc, vc, ic)
    stream.synchronize()
    assert torch.equal(a, c)
    m.device_status()


def test_cuda_graph_replay_with_mutated_inputs():
    """progression_validation.py:118-140."""
    m = sp()
    q, k, v = gen.make_qkv(2, 16, 2, 1024, 4096, seed=601)
    ids = gen.make_ids(2, 2, 8, 32, 16, 601, "unsorted")
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    out = torch.empty_like(qc)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for _ in range(3):
            m.attention_out(qc, kc, vc, ic, out)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        m.attention_out(qc, kc, vc, ic, out)
        m.attention_out(qc, kc, vc, ic, out)
    torch.cuda.synchronize()
    for seed in (607, 613):
        with torch.cuda.stream(stream):
            qc.mul_(-0.75)
            vc.add_(0.0625)
            ic.copy_(gen.make_ids(2, 2, 8, 32, 16, seed, "unsorted"))
            out.fill_(float("nan"))
            graph.replay()
        stream.synchronize()
        ref_o, _ = oracle.gather_attention(qc.cpu(), kc.cpu(), vc.cpu(), ic.cpu())
        check(out, None, ref_o, None)
    m.device_status()


def test_rejected_inputs():
    """progression_validation.py:141-161."""
    m = sp()
    q, k, v = gen.make_qkv(1, 4, 2, 256, 512, seed=9)
    ids = gen.make_ids(1, 2, 2, 4, 2, 9)
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    bad = [
        (qc, kc[:, :0], vc[:, :0], ic[:, :0]),
        (qc, kc, vc, ic[..., :0]),
        (qc.float(), kc, vc, ic),
        (qc.detach().requires_grad_(), kc, vc, ic),
        (qc, kc, vc, ic.repeat_interleave(2, dim=1)),
        (qc, kc, vc, ic.long()),
        (qc[:, :, :, :64], kc, vc, ic),
    ]
    for args in bad:
        with pytest.raises(RuntimeError):
            m.attention(*args)
    out = torch.empty_like(qc)
    with pytest.raises(RuntimeError):
        m.attention_out(qc, kc, vc, ic, qc)
    with pytest.raises(RuntimeError):
        m.attention_out(qc, kc, vc, ic, out[:, :, :128])
    # top-k larger than the number of KV blocks
    with pytest.raises(RuntimeError):
        m.attention(qc, kc, vc, torch.zeros((1, 2, 2, 5), dtype=torch.int32, device="cuda"))


def test_partial_segments_merge_to_whole():
    """KV-range segments through the partial entry point + oracle merge."""
    m = sp()
    q, k, v = gen.make_qkv(1, 8, 2, 512, 2048, seed=77)
    ids = gen.make_ids(1, 2, 4, 16, 8, 78, "unsorted")
    ref_o, ref_l = oracle.gather_attention(q, k, v, ids)
    seg_ids, seg_counts = oracle.split_kv_segments(ids, 16, 4)
    for dtype in (torch.float32, torch.bfloat16):
        partial = torch.full((4, 1, 8, 512, 128), float("nan"), dtype=dtype, device="cuda")
        plse = torch.full((4, 1, 8, 512), float("nan"), device="cuda")
        m.attention_partial_out(q.cuda(), k.cuda(), v.cuda(), seg_ids.cuda(), seg_counts.cuda(), partial, plse)
        torch.cuda.synchronize()
        m.device_status()
        po = partial.float().cpu().permute(1, 2, 3, 0, 4)
        pl = plse.cpu().permute(1, 2, 3, 0)
        o, l = oracle.combine_partials(po, pl)
        d = (o - ref_o).abs()
        assert d.max() <= 2e-2 and d.mean() <= 2e-3
        assert torch.all((l - ref_l).abs() <= 1e-3 * ref_l.abs().clamp_min(1.0))


def test_host_pipeline_matches_device_path():
    """Pinned host buffers in and out, chunks pipelined over three streams."""
    m = sp()
    q, k, v = gen.make_qkv(2, 8, 4, 512, 1024, seed=91)
    ids = gen.make_ids(2, 4, 4, 8, 3, 92, "unsorted")
    ref_o, ref_l = oracle.gather_attention(q, k, v, ids)
    hq_, hk_, hv_, hi_ = (t.pin_memory() for t in (q, k, v, ids))
    ho = torch.full(q.shape, float("nan"), dtype=torch.bfloat16).pin_memory()
    hl = torch.full(q.shape[:3], float("nan")).pin_memory()
    pipe = m.HostPipeline(2, 8, 4, 512, 1024, 3, "cuda:0", chunks=3)
    for _ in range(2):                      # second call reuses the staging buffers
        ho.fill_(float("nan"))
        pipe.run(hq_, hk_, hv_, hi_, ho, hl).synchronize()
        check(ho, hl, ref_o, ref_l)
    m.device_status()
    # fewer groups than chunks: a group's heads are split over chunks (K, V and the lists travel with
    # the first one), staged through caller-owned device buffers; changed inputs on the second call
    q, k, v = gen.make_qkv(1, 8, 1, 512, 1024, seed=93)
    ids = gen.make_ids(1, 1, 4, 8, 3, 94)
    hq_, hk_, hv_, hi_ = (t.clone().pin_memory() for t in (q, k, v, ids))
    ho = torch.empty(q.shape, dtype=torch.bfloat16).pin_memory()
    hl = torch.empty(q.shape[:3]).pin_memory()
    bufs = (torch.empty_like(q, device="cuda"), torch.empty_like(k, device="cuda"), torch.empty_like(v, device="cuda"),
            torch.empty_like(ids, device="cuda"), torch.empty_like(q, device="cuda"),
            torch.empty(q.shape[:3], device="cuda"))
    pipe = m.HostPipeline(1, 8, 1, 512, 1024, 3, "cuda:0", chunks=4, buffers=bufs)
    assert pipe.chunks == 4
    for shift in (0, 1):
        hk_.copy_(k.roll(shift * 128, dims=2))
        hv_.copy_(v.roll(shift * 128, dims=2))
        ref_o, ref_l = oracle.gather_attention(q, hk_.clone(), hv_.clone(), ids)
        ho.fill_(float("nan"))
        pipe.run(hq_, hk_, hv_, hi_, ho, hl).synchronize()
        check(ho, hl, ref_o, ref_l)
    t0 = pipe.run(hq_, hk_, hv_, hi_, ho, hl, copy_only=True)
    t0.synchronize()
    m.device_status()


@pytest.mark.parametrize("shape,topk,counts_kind", [
    ((2, 16, 1, 4096, 2048), 16, "full"),      # the reference's shape: 512 items = 3 rounds + 68 -> two pieces each
    ((1, 8, 2, 40 * 128, 4096), 16, "ragged"),      # 160 items: 1 round + 12 -> four pieces each, ragged counts
    ((1, 3, 3, 51 * 256, 2048), 8, "full"),    # split mode (group 1): 153 items, 5 left over, two pieces of four blocks
])
def test_balanced_last_round_matches_the_plain_call(shape, topk, counts_kind):
    """With a workspace the kernel cuts the items of a last, partly filled round into pieces and merges their
    partials: same result as the plain call up to the bf16 rounding of the partials, LSE to fp32 rounding, and
    inside the oracle tolerance; rows outside the last round are bit-identical."""
    m = sp()
    b, hq, hkv, sq, skv = shape
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=11, k_block_offset=0.5)
    ids = gen.make_ids(b, hkv, sq // 128, skv // 128, topk, 3, "unsorted")
    counts = None
    if counts_kind == "ragged":
        g = torch.Generator().manual_seed(4)
        counts = torch.randint(0, topk + 1, (b, hkv, sq // 128), generator=g, dtype=torch.int32)
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    cc = None if counts is None else counts.cuda()
    plain = torch.full(q.shape, float("nan"), dtype=torch.bfloat16, device="cuda")
    plain_lse = torch.full(q.shape[:3], float("nan"), device="cuda")
    m.attention_out(qc, kc, vc, ic, plain, cc, plain_lse, balance=False)
    bal = torch.full_like(plain, float("nan"))
    bal_lse = torch.full_like(plain_lse, float("nan"))
    m.attention_out(qc, kc, vc, ic, bal, cc, bal_lse, balance=True)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.isfinite(bal.float()).all()
    diff = (bal.float() - plain.float()).abs()
    changed = (diff > 0).reshape(b, hq, sq // 128, -1).any(-1)    # (head, query block) tiles that went through the merge
    assert 0 < int(changed.sum()) <= changed.numel() // 2         # the last round only
    assert diff.max().item() <= 2.0 ** -6 * max(1.0, plain.float().abs().max().item())
    fin = torch.isfinite(plain_lse)
    assert torch.equal(torch.isfinite(bal_lse), fin)
    assert torch.all((bal_lse[fin] - plain_lse[fin]).abs() <= 2e-6 * plain_lse[fin].abs().clamp_min(1.0))
    ref_o, ref_l = oracle.gather_attention(q, k, v, ids, counts)
    check(bal, bal_lse, ref_o, ref_l)


@pytest.mark.parametrize("shape,topk,counts_kind", [
    ((1, 2, 1, 128, 8192), 64, None),          # one pair item: 16 pieces of 4 blocks
    ((1, 3, 1, 384, 2048), 16, None),          # split mode, odd number of query blocks: a stream without a tile
    ((2, 1, 1, 384, 4096), 16, "ragged"),      # lists of 0 to 16 blocks: with counts the plain launch
    ((1, 4, 2, 2304, 2304), 18, "ragged"),     # 36 items, the same
    ((1, 8, 1, 2304, 4096), 32, None),         # 72 items: two pieces
    ((1, 8, 1, 2304, 1024), 8, None),          # 72 items, not worth a split: the plain launch
])
@pytest.mark.parametrize("nan", [False, True])
def test_launch_of_less_than_a_round_matches_the_plain_call(shape, topk, counts_kind, nan):
    """With a workspace, no counts and at most half as many items as SMs, every item is cut into pieces with fp32
    partials (which launches are split, and the weights of the pieces, are asserted by the next test): same result as the plain call up to the rounding of the bf16 probabilities and outputs, LSE to fp32 rounding, inside the
    oracle tolerance; rows that are NaN without the split stay NaN."""
    m = sp()
    b, hq, hkv, sq, skv = shape
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=13, k_block_offset=0.5)
    ids = gen.make_ids(b, hkv, sq // 128, skv // 128, topk, 5, "unsorted")
    counts = None
    if counts_kind == "ragged":
        counts = (torch.arange(b * hkv * (sq // 128)) * 7 % (topk + 1)).to(torch.int32).reshape(b, hkv, sq // 128)
    if nan:
        q = q.clone()
        q[:, 0, 5] = float("nan")
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    cc = None if counts is None else counts.cuda()
    plain = torch.full(q.shape, 7.0, dtype=torch.bfloat16, device="cuda")
    plain_lse = torch.full(q.shape[:3], 7.0, device="cuda")
    m.attention_out(qc, kc, vc, ic, plain, cc, plain_lse, balance=False)
    split = torch.full_like(plain, 9.0)
    split_lse = torch.full_like(plain_lse, 9.0)
    m.attention_out(qc, kc, vc, ic, split, cc, split_lse, balance=True)
    torch.cuda.synchronize()
    m.device_status()
    assert torch.equal(split.isnan(), plain.isnan()) and torch.equal(split_lse.isnan(), plain_lse.isnan())
    fin = torch.isfinite(plain.float())
    diff = (split.float() - plain.float())[fin].abs()
    # Both calls round every probability to bf16 (relative error 2^-9 each, relative to different running maxima) and
    # the output once: |difference| <= 2 * 2^-9 * (sum p |v| + |o|) <= 2^-8 * (max |v| + |o|).
    assert torch.all(diff <= 2.0 ** -8 * (v.float().abs().max().item() + plain.float()[fin].abs()))
    lfin = torch.isfinite(plain_lse)
    assert torch.equal(torch.isneginf(split_lse), torch.isneginf(plain_lse))
    assert torch.all((split_lse[lfin] - plain_lse[lfin]).abs() <= 2e-6 * plain_lse[lfin].abs().clamp_min(1.0))
    if not nan:
        ref_o, ref_l = oracle.gather_attention(q, k, v, ids, counts)
        check(split, split_lse, ref_o, ref_l)


@pytest.mark.parametrize("shape,topk,counts_kind,pieces", [
    ((1, 2, 1, 128, 8192), 64, None, True),          # one pair item: 16 pieces of 4 blocks
    ((1, 3, 1, 384, 2048), 16, None, True),          # split mode, odd number of query blocks: a stream without a tile
    ((1, 4, 2, 2304, 2304), 18, None, True),         # 36 items: four pieces, not all of the same length
    ((1, 8, 1, 2304, 4096), 32, None, True),         # 72 items: two pieces
    ((2, 1, 1, 384, 4096), 16, "ragged", False),     # counts, empty lists among them: the plain launch
    ((1, 8, 1, 2304, 1024), 8, None, False),         # 72 items, not worth a split: the plain launch
])
def test_pieces_of_small_launches_have_their_weights(shape, topk, counts_kind, pieces):
    """Every key block's values have a mean of their own, so that a wrong weight of a piece shows: the error of a tile
    against the fp32 oracle is that of the plain call. A launch that is not split has the plain call's bits."""
    m = sp()
    b, hq, hkv, sq, skv = shape
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=13, k_block_offset=0.5)
    means = torch.randn((b, hkv, skv // 128, 1, 128), generator=torch.Generator().manual_seed(29)) * 4.0
    v = (v.float().view(b, hkv, skv // 128, 128, 128) + means).view(b, hkv, skv, 128).to(torch.bfloat16)
    ids = gen.make_ids(b, hkv, sq // 128, skv // 128, topk, 5, "unsorted")
    counts = None
    if counts_kind == "ragged":
        counts = (torch.arange(b * hkv * (sq // 128)) * 7 % (topk + 1)).to(torch.int32).reshape(b, hkv, sq // 128)
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    cc = None if counts is None else counts.cuda()
    plain, split = torch.empty_like(qc), torch.empty_like(qc)
    m.attention_out(qc, kc, vc, ic, plain, cc, balance=False)
    m.attention_out(qc, kc, vc, ic, split, cc, balance=True)
    torch.cuda.synchronize()
    m.device_status()
    # every 128-row tile goes through the merge, or none does
    differs = (split != plain).reshape(b, hq, sq // 128, -1).any(-1)
    assert torch.equal(differs, torch.full_like(differs, pieces))
    ref, _ = oracle.gather_attention(q, k, v, ids, counts)

    def rms(x):
        return x.reshape(b, hq, sq // 128, -1).square().mean(-1).sqrt()
    plain_err, split_err = rms(plain.float().cpu() - ref), rms(split.float().cpu() - ref)
    # Both calls round every probability to bf16 once (against different running maxima) and the output once; partials
    # and weights are fp32. So the errors are of one size, 1.25 for the sampling of a tile's 16384 values; one piece of
    # 16 left out is 200 times that. The output's rounding is 2^-9 / sqrt(3) of it, the probabilities' about a fifth.
    assert torch.all(split_err <= 1.25 * plain_err)
    assert torch.all(plain_err <= 2.0 ** -8 * rms(ref))


@pytest.mark.parametrize("shape,topk", [
    ((1, 6, 3, 128, 8192), 64),           # three pair items in 16 pieces of four blocks each
    ((1, 3, 1, 384, 2048), 16),           # split mode, a stream without a tile
    ((1, 10, 5, 4096, 2048), 16),         # one round and twelve items: the pieces of a balanced last round
])
def test_blocks_of_minus_infinite_scores_have_no_weight(shape, topk):
    """Keys whose scores are all -inf (first feature -inf against a positive query feature) take no part in the softmax,
    wherever they stand: as the whole of a piece of a list, as its first block, as any other. A row with no other keys
    is NaN with LSE -inf, split or not."""
    m = sp()
    b, hq, hkv, sq, skv = shape
    q, k, v = gen.make_qkv(b, hq, hkv, sq, skv, seed=17, k_block_offset=0.5)
    nt, qt = skv // 128, sq // 128
    q, k = q.clone(), k.clone()
    q[..., 0] = 1.0
    masked = torch.zeros(nt, dtype=torch.bool)
    masked[: nt // 4] = True              # ascending lists: whole pieces at the start ...
    masked[nt // 2::3] = True             # ... and blocks here and there
    k.view(b, hkv, nt, 128, 128)[:, :, masked, :, 0] = -float("inf")
    ids = torch.arange(topk, dtype=torch.int32).mul(nt).div(topk, rounding_mode="floor").expand(b, hkv, qt, topk).contiguous()
    ids[:, 0, 0] = ids[:, -1, -1] = torch.where(masked)[0][:1].int()     # lists of masked blocks only
    kept = ~masked[ids.long()]
    counts = kept.sum(-1).to(torch.int32)
    kept_ids = torch.zeros_like(ids)
    for i in range(b):
        for h in range(hkv):
            for t in range(qt):
                live = ids[i, h, t][kept[i, h, t]]
                kept_ids[i, h, t, :len(live)] = live
    ref_o, ref_l = oracle.gather_attention(q, k, v, kept_ids, counts)
    none = (counts == 0).repeat_interleave(hq // hkv, 1).repeat_interleave(128, 2)
    assert none.any() and not none.all()
    qc, kc, vc, ic = q.cuda(), k.cuda(), v.cuda(), ids.cuda()
    for balance in (False, True):
        out = torch.full(q.shape, 7.0, dtype=torch.bfloat16, device="cuda")
        lse = torch.full(q.shape[:3], 7.0, device="cuda")
        m.attention_out(qc, kc, vc, ic, out, None, lse, balance=balance)
        torch.cuda.synchronize()
        m.device_status()
        assert out.cpu()[none].isnan().all() and torch.isneginf(lse.cpu()[none]).all()
        check(out.cpu()[~none], lse.cpu()[~none], ref_o[~none], ref_l[~none])


def test_small_launch_with_counts_is_not_split():
    """How much of a list is live stands on the device: with counts a launch of less than a round runs as the plain
    call does, bit for bit, and the same lists without counts are split (other bits somewhere)."""
    m = sp()
    q, k, v = (t.cuda() for t in gen.make_qkv(1, 4, 2, 384, 8192, seed=19, k_block_offset=0.5))
    ids = gen.make_ids(1, 2, 3, 64, 64, 5, "unsorted").cuda()
    for counts in (torch.full((1, 2, 3), 2, dtype=torch.int32, device="cuda"), None):
        plain, out = torch.empty_like(q), torch.empty_like(q)
        m.attention_out(q, k, v, ids, plain, counts, balance=False)
        m.attention_out(q, k, v, ids, out, counts)
        assert torch.equal(plain, out) == (counts is not None)
    m.device_status()


@pytest.mark.parametrize("items,topk,split", [(74, 20, False), (74, 24, False), (74, 32, True), (37, 16, True), (37, 13, False), (1, 64, True)])
def test_small_launch_split_rule(items, topk, split):
    """Both sides of the line where the blocks saved outweigh partials and merge, which cost more with more items: a
    launch that is not split has the bits of the plain call."""
    m = sp()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are for 148 SMs")
    q, k, v = (t.cuda() for t in gen.make_qkv(1, 2 * items, items, 128, topk * 128, seed=23, k_block_offset=0.5))
    ids = gen.make_ids(1, items, 1, topk, topk, 7, "unsorted").cuda()
    plain, out = torch.empty_like(q), torch.empty_like(q)
    m.attention_out(q, k, v, ids, plain, balance=False)
    m.attention_out(q, k, v, ids, out)
    assert torch.equal(plain, out) != split
    m.device_status()


def test_split_calls_share_no_scratch():
    """Two graphs captured one after the other on the same stream and replayed at the same time on two, with launches
    that are split into pieces: every output stays that of the plain call. (32 CTAs each: both graphs fit the GPU.)"""
    m = sp()
    b, hq, hkv, sq, skv, topk, calls = 1, 4, 2, 128, 8192, 64, 20
    graphs, want, outs, keep = [], [], [], []
    for seed in (1, 2):
        q, k, v = (t.cuda() for t in gen.make_qkv(b, hq, hkv, sq, skv, seed=seed, k_block_offset=0.5))
        ids = gen.make_ids(b, hkv, 1, skv // 128, topk, seed, "unsorted").cuda()
        plain = torch.empty_like(q)
        m.attention_out(q, k, v, ids, plain, balance=False)
        out = torch.empty((calls, *q.shape), dtype=q.dtype, device="cuda")
        m.attention_out(q, k, v, ids, out[0])
        torch.cuda.synchronize()
        assert not torch.equal(out[0], plain)            # the call is split: other bits
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for i in range(calls):
                m.attention_out(q, k, v, ids, out[i])
        graphs.append(g)
        want.append(out[0].clone())
        outs.append(out)
        keep.append((q, k, v, ids))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(10):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        for out, w in zip(outs, want):
            assert torch.equal(out, w.expand_as(out))
    m.device_status()


def test_a_waiting_attention_call_leaves_the_idle_sms_to_other_streams():
    """Stream 1 runs one long work item (one SM) and then a call that fills the GPU; stream 2 a short call. The second
    call of stream 1 may be set up under the first one's tail, but must not hold the other SMs while that runs: the
    short call is done long before the long item."""
    m = sp()

    def call(hkv, nb, topk, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = torch.randn((1, 2 * hkv, 128, 128), device="cuda", generator=g).to(torch.bfloat16)
        k = torch.randn((1, hkv, nb * 128, 128), device="cuda", generator=g).to(torch.bfloat16)
        v = torch.randn((1, hkv, nb * 128, 128), device="cuda", generator=g).to(torch.bfloat16)
        ids = torch.arange(topk, dtype=torch.int32, device="cuda").expand(1, hkv, 1, topk).contiguous()
        out = torch.empty_like(q)
        return lambda: m.attention_out(q, k, v, ids, out, balance=False)

    long_item, filling, short = call(1, 2048, 2048, 1), call(148, 2, 2, 2), call(148, 2, 2, 3)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):                          # once to warm up
        start, end1, end2 = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        torch.cuda.synchronize()
        with torch.cuda.stream(s1):
            start.record()
            long_item()
            filling()
            end1.record()
        with torch.cuda.stream(s2):
            short()
            end2.record()
        torch.cuda.synchronize()
    whole, other = start.elapsed_time(end1), start.elapsed_time(end2)
    assert whole > 2.0                          # 2048 blocks at 1.7 us
    assert other < 0.5 * whole, (other, whole)
    m.device_status()
