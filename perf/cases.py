"""The work a user of this framework has it do, as cases that can be timed and compared.

A case names an operation of the public interface and its sizes:

  attention        block-sparse attention over given lists (attention_out)
  indexed_summary  R1 / R2 / R4 selection, then attention over the selected blocks (one call)
  select_summary   R1 / R2 / R4 selection alone
  fp4_select       bf16 q and k -> NVFP4 index vectors -> top-k block lists
  fp4_pipeline     quantise, NVFP4 selection and attention as one call
  kv_centric       KV-centric attention over block lists: segments, partials, merge
  kv_tokens        KV-centric attention over per-token lists: reverse index, partials, merge
  fp4_scores       NVFP4 page scores of a ragged batch over a paged key cache

`qb` and `nb` are query and key blocks of 128 tokens. Everything random is drawn on the GPU from the
seed; request lengths are part of the case."""
import math
import random

import torch

import sparse_attention_b200_b200 as sp

BLOCK, D = 128, 128


def listed():
    return [
        # the smallest call: a short odd-sized sequence, a group of three heads, lists of different lengths
        dict(name="attention_ragged", op="attention", b=1, hkv=4, group=3, qb=9, nb=23, topk=7, ragged=True, sort=False),
        # a 4 Ki prompt with every head its own lists: selection and attention of one layer, latency and launches count
        dict(name="r1_indexed_attention_4k", op="indexed_summary", b=1, hkv=8, group=1, qb=32, nb=32, r=1, topk=8),
        # a 4 Ki chunk of queries of 16 heads over one shared 16 Ki key head (chunked prefill, two requests)
        dict(name="attention_gqa_16k", op="attention", b=2, hkv=1, group=16, qb=32, nb=128, topk=16, ragged=False, sort=True),
        # a whole 32 Ki sequence of a 32-head model without grouping
        dict(name="attention_mha_32k", op="attention", b=1, hkv=32, group=1, qb=256, nb=256, topk=16, ragged=False, sort=True),
        # the R4 selector alone on that chunk: what stands between two layers' kernels
        dict(name="r4_select_16k", op="select_summary", b=2, hkv=1, group=16, qb=32, nb=128, r=4, topk=16),
        # one KV-head group of the 1 Mi-token model: the share of one GPU of eight, selection and attention
        dict(name="r4_indexed_attention_1m", op="indexed_summary", b=1, hkv=1, group=8, qb=8192, nb=8192, r=4, topk=64),
        # the NVFP4 indexer of the 128 Ki-token model (quantisation included)
        dict(name="fp4_select_131k", op="fp4_select", b=1, hkv=4, group=16, qb=1024, nb=1024, topk=64),
        # NVFP4 selection and attention of the 4 Ki chunk over 16 Ki keys as one call
        dict(name="fp4_pipeline_16k", op="fp4_pipeline", b=2, hkv=1, group=16, qb=32, nb=128, topk=16),
        # the attention of the 128 Ki-token model by KV ranges with a merge
        dict(name="kv_centric_131k", op="kv_centric", b=1, hkv=4, group=16, qb=1024, nb=1024, topk=64),
        # per-token lists: eight 4 Ki sequences, 16 heads on one key head
        dict(name="kv_tokens_4k", op="kv_tokens", b=8, hkv=1, group=16, sq=4096, nb=32, topk=16, q_token_major=False,
             partial_f32=False),
        # serving: a batch of ragged prefill requests over a paged cache, causal
        dict(name="fp4_scores_prefill", op="fp4_scores", requests=8, hk=1, group=2, q_lo=512, q_hi=4096, k_lo=4096,
             k_hi=16384, causal=True, lengths=7),
        # serving: a decode batch, a few new tokens for each of 64 long requests
        dict(name="fp4_scores_decode", op="fp4_scores", requests=64, hk=1, group=16, q_lo=1, q_hi=8, k_lo=8192,
             k_hi=32768, causal=True, lengths=7),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    while True:
        op = rng.choice(["attention", "attention", "indexed_summary", "indexed_summary", "select_summary", "fp4_select",
                         "fp4_pipeline", "kv_centric", "kv_tokens", "fp4_scores"])
        if op == "fp4_scores":
            decode = rng.random() < 0.5
            q_hi = rng.randint(1, 8) if decode else _log(rng, 16, 4096)
            k_hi = _log(rng, 512, 32768)
            case = dict(op=op, requests=_log(rng, 1, 128 if decode else 16), hk=rng.choice([1, 1, 2]),
                        group=rng.choice([1, 2, 4, 8, 16]), q_lo=max(1, q_hi // 8), q_hi=q_hi, k_lo=max(1, k_hi // 4),
                        k_hi=k_hi, causal=rng.random() < 0.7, lengths=rng.randrange(1 << 20))
        elif op == "kv_tokens":
            group = rng.choice([1, 2, 4, 8, 16, 16])
            nb = _log(rng, 2, 256)
            case = dict(op=op, b=_log(rng, 1, 8), hkv=rng.choice([1, 1, 2, 4]), group=group, sq=_log(rng, 17, 8192), nb=nb,
                        topk=_log(rng, 1, min(nb, 16)), q_token_major=group >= 8 and rng.random() < 0.3,
                        partial_f32=rng.random() < 0.2)
        else:
            summary = op in ("indexed_summary", "select_summary")
            most = 8192 if summary else 1024
            nb = _log(rng, 4, most)
            case = dict(op=op, b=rng.choice([1, 1, 2, 3]), hkv=rng.choice([1, 1, 2, 3, 4, 8]),
                        group=rng.choice([1, 2, 3, 4, 8, 16]), qb=_log(rng, 1, most), nb=nb)
            if summary:
                case["r"] = rng.choice([1, 2, 4, 4])
            case["topk"] = _log(rng, min(4, nb), min(nb, 64))
            if op == "attention":
                case.update(ragged=rng.random() < 0.3, sort=rng.random() < 0.5)
            if summary and case["group"] * case["r"] > 64:
                continue
        w = work(case)
        # no drawn case is larger than the largest listed one of its kind
        flops, bytes_ = {"attention": (1.2e12, 3e9), "indexed_summary": (4e13, 5e9), "select_summary": (5e11, 3e9),
                         "fp4_select": (1.8e13, 6e9), "fp4_pipeline": (1e13, 3e9), "kv_centric": (3.6e13, 5e9),
                         "kv_tokens": (5.6e11, 1e9), "fp4_scores": (2e11, 4e8)}[op]
        if w["flops"] <= flops and w["bytes"] <= bytes_:
            return case


def _lengths(case):
    r = random.Random(case["lengths"])
    q = [r.randint(case["q_lo"], case["q_hi"]) for _ in range(case["requests"])]
    k = [max(n, r.randint(case["k_lo"], case["k_hi"])) for n in q]
    return q, k


def _normal(shape, gen):
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(generator=gen)


def _qkv(case, gen, values=True):
    """q, k, v ~ N(0, 1); every key block has a mean of its own ~ N(0, 0.5), which is what a block indexer looks for."""
    b, hkv, hq, nb = case["b"], case["hkv"], case["hkv"] * case["group"], case["nb"]
    q = _normal((b, hq, case.get("sq", case.get("qb", 0) * BLOCK), D), gen)
    k = _normal((b, hkv, nb, BLOCK, D), gen)
    k += 0.5 * _normal((b, hkv, nb, 1, D), gen)
    return q, k.view(b, hkv, nb * BLOCK, D), _normal((b, hkv, nb * BLOCK, D), gen) if values else None


def _lists(shape, nb, topk, sort, gen):
    """Distinct key blocks of every list, in random order (as a scorer ranks them) or ascending."""
    rows = math.prod(shape)
    ids = torch.empty((rows, topk), dtype=torch.int32, device="cuda")
    step = max(1, (1 << 26) // nb)
    for i in range(0, rows, step):
        n = min(step, rows - i)
        ids[i:i + n] = torch.rand((n, nb), device="cuda", generator=gen).topk(topk, dim=1).indices
    if sort:
        ids = ids.sort(dim=1).values
    return ids.view(*shape, topk)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, s = case["op"], {"op": case["op"]}
    if op == "fp4_scores":
        q_lens, k_lens = _lengths(case)
        hk, hq = case["hk"], case["hk"] * case["group"]
        pages = [-(-n // BLOCK) for n in k_lens]
        total_q, total_pages = sum(q_lens), sum(pages)

        def cumulated(lengths):
            return torch.tensor([0] + lengths, device="cuda").cumsum(0).to(torch.int32)
        s["q"] = torch.randint(256, (total_q, hq, 64), dtype=torch.uint8, device="cuda", generator=gen)
        s["k"] = torch.randint(256, (total_pages, hk, BLOCK, 64), dtype=torch.uint8, device="cuda", generator=gen)
        s["q_scale"] = (torch.rand((total_q, hq, 8), device="cuda", generator=gen) + 0.5).to(torch.float8_e4m3fn)
        s["k_scale"] = (torch.rand((total_pages, hk, BLOCK, 8), device="cuda", generator=gen) + 0.5).to(torch.float8_e4m3fn)
        s["cu"] = cumulated(q_lens), cumulated(k_lens), cumulated(pages)
        s["options"] = dict(max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens), causal=case["causal"], exact=False,
                            kv_indices=torch.randperm(total_pages, device="cuda", generator=gen).to(torch.int32))
        return s
    q, k, v = _qkv(case, gen, values=op not in ("select_summary", "fp4_select"))
    s.update(q=q, k=k, v=v)
    b, hkv, nb, topk = case["b"], case["hkv"], case["nb"], case["topk"]
    if op in ("attention", "indexed_summary", "fp4_pipeline"):
        s["out"] = torch.empty_like(q)
    if op == "attention":
        s["lse"] = torch.empty(q.shape[:3], dtype=torch.float32, device="cuda")
        s["ids"] = _lists((b, hkv, case["qb"]), nb, topk, case["sort"], gen)
        s["counts"] = torch.randint(1, topk + 1, (b, hkv, case["qb"]), dtype=torch.int32, device="cuda",
                                    generator=gen) if case["ragged"] else None
    elif op in ("indexed_summary", "select_summary"):
        s["selector"] = sp.SummarySelector(q, k, case["r"], topk=topk, keep_scores=False)
    elif op == "fp4_select":
        s["ids"] = torch.empty((b, hkv, case["qb"], topk), dtype=torch.int32, device="cuda")
        s["workspace"] = None                           # made by the first pass and kept
    elif op == "fp4_pipeline":
        s["lse"] = torch.empty(q.shape[:3], dtype=torch.float32, device="cuda")
        s["pipeline"] = sp.Fp4Pipeline(q, k, v, topk=topk)
    elif op == "kv_centric":
        s["operator"] = sp.Prepared(q, k, v, _lists((b, hkv, case["qb"]), nb, topk, False, gen))
    elif op == "kv_tokens":
        ids = _lists((b, hkv, case["sq"]), nb, topk, False, gen)
        if case["q_token_major"]:
            q = q.transpose(1, 2).contiguous()
        s["operator"] = sp.PreparedTokens(q, k, v, ids, q_token_major=case["q_token_major"],
                                          partial_f32=case["partial_f32"])
    return s


def run(s):
    op = s["op"]
    if op == "attention":
        sp.attention_out(s["q"], s["k"], s["v"], s["ids"], s["out"], counts=s["counts"], lse=s["lse"])
        return s["out"], s["lse"]
    if op == "indexed_summary":
        sp.summary_indexed_attention_out(s["selector"], s["v"], s["out"])
        return s["out"], s["selector"].ids
    if op == "select_summary":
        return s["selector"].run()
    if op == "fp4_select":
        q, k = s["q"], s["k"]
        hkv = k.shape[1]
        (qc, qs), (kc, ks) = sp.quantize_queries(q, hkv), sp.quantize_keys(k)
        inputs = sp.prepare_fp4_inputs(qc, kc, qs, ks, batch_size=q.shape[0], len_q=q.shape[2], len_kv=k.shape[2])
        ids, s["workspace"] = sp.fp4_indexer_fast(inputs, selected=s["ids"], workspace=s["workspace"])
        return ids
    if op == "fp4_pipeline":
        s["pipeline"].run(s["out"], s["lse"])
        return s["out"], s["lse"], s["pipeline"].ids
    if op in ("kv_centric", "kv_tokens"):
        return s["operator"].run()
    cu_q, cu_k, cu_pages = s["cu"]
    return sp.fp4_block_scores_varlen(s["q"], s["k"], s["q_scale"], s["k_scale"], cu_q, cu_k, cu_pages, **s["options"])


def work(case):
    op = case["op"]
    if op == "fp4_scores":
        q_lens, k_lens = _lengths(case)
        hk, hq = case["hk"], case["hk"] * case["group"]
        pages = sum(-(-n // BLOCK) for n in k_lens)
        tiles = -(-max(k_lens) // BLOCK)
        # causal: the last query of a request sees all of its keys
        pairs = sum(q * k - (q * (q - 1) // 2 if case["causal"] else 0) for q, k in zip(q_lens, k_lens))
        return {"bytes": 72 * (sum(q_lens) * hq + pages * BLOCK * hk) + 4 * hq * tiles * sum(q_lens),
                "flops": 2.0 * D * hq * pairs}
    b, hkv, hq, nb, topk = case["b"], case["hkv"], case["hkv"] * case["group"], case["nb"], case["topk"]
    sq = case.get("sq", case.get("qb", 0) * BLOCK)
    lists = b * hkv * (sq if op == "kv_tokens" else sq // BLOCK)
    q_bytes, key_bytes, id_bytes = 2 * D * b * hq * sq, 2 * D * b * hkv * nb * BLOCK, 4 * lists * topk
    live = (topk + 1) / 2 if case.get("ragged") else topk      # ragged counts are uniform in 1..topk
    attention = 4.0 * b * hq * sq * live * BLOCK * D
    lse_bytes = 4 * b * hq * sq
    if op == "select_summary":
        return {"bytes": q_bytes + key_bytes + id_bytes, "flops": 2.0 * b * hq * case["qb"] * nb * case["r"] ** 2 * D}
    if op == "indexed_summary":
        return {"bytes": 2 * q_bytes + 2 * key_bytes + id_bytes,
                "flops": attention + 2.0 * b * hq * case["qb"] * nb * case["r"] ** 2 * D}
    if op == "fp4_select":
        return {"bytes": q_bytes + key_bytes + id_bytes, "flops": 2.0 * b * hkv * sq * nb * BLOCK * D}
    # blocks that no list names need not be read
    used = min(1.0, lists * live / (b * hkv * nb))
    bytes_ = 2 * q_bytes + 2 * key_bytes * used + id_bytes + lse_bytes
    if op == "fp4_pipeline":
        return {"bytes": 2 * q_bytes + key_bytes * (1 + used) + id_bytes + lse_bytes,
                "flops": attention + 2.0 * b * hkv * sq * nb * BLOCK * D}
    return {"bytes": bytes_, "flops": attention}


def tolerance(case):
    if case["op"] in ("select_summary", "fp4_select"):
        return "exact"                                  # block ids: ties go to the lower id
    if case["op"] == "fp4_scores":
        return {"rel": 1e-6, "max": 1e-5}               # exact group sums, added in fp32
    return {"rel": 1e-2, "max": 7e-2, "differ": 0.0}    # bf16 probabilities, partials and outputs


def _attend(q, k, v, blocks, keep):
    """softmax(q k^T / sqrt(D)) v of one list in 64 bits: q [g, n, D], k and v [nb, BLOCK, D], blocks [m], keep
    [n, m * BLOCK] or None -> (o, lse)."""
    kk, vv = (t[blocks].reshape(-1, D).double() for t in (k, v))
    s = q.double() @ kk.T / math.sqrt(D)
    if keep is not None:
        s = s.masked_fill(~keep, -math.inf)
    lse = s.logsumexp(-1)
    return torch.exp(s - lse[..., None]) @ vv, lse


def _exact_scores(s, case):
    """Page scores of the ragged batch: decoded e2m1 codes and e4m3 scales, products and sums in 64 bits."""
    table = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    table = torch.cat([table, -table])

    def decode(codes, scales):
        pairs = torch.stack([codes & 15, codes >> 4], -1).flatten(-2)
        return table[pairs.long()] * scales.to(torch.float64).repeat_interleave(16, -1)
    q_lens, k_lens = _lengths(case)
    hq, tiles, pages = case["hk"] * case["group"], -(-max(k_lens) // BLOCK), s["options"]["kv_indices"]
    out = torch.full((hq, tiles, sum(q_lens)), -math.inf, dtype=torch.float64, device="cuda")
    q0 = p0 = 0
    for n, m in zip(q_lens, k_lens):
        np_ = -(-m // BLOCK)
        own = pages[p0:p0 + np_].long()
        last = torch.arange(n, device="cuda") + (m - n if case["causal"] else m)      # last visible key of a query
        for h in range(hq):
            qd = decode(s["q"][q0:q0 + n, h], s["q_scale"][q0:q0 + n, h])
            kd = decode(s["k"][own, h // case["group"]], s["k_scale"][own, h // case["group"]]).reshape(-1, D)
            x = qd @ kd.T
            col = torch.arange(np_ * BLOCK, device="cuda")
            x = x.masked_fill((col[None] >= m) | (col[None] > last[:, None]), -math.inf)
            out[h, :np_, q0:q0 + n] = x.view(n, np_, BLOCK).amax(-1).T
        q0, p0 = q0 + n, p0 + np_
    return out


def exact(case, seed):
    """The outputs of run() in 64 bits; None where the path selects its blocks itself (the ids are compared as they
    are) and where it would take long."""
    op = case["op"]
    if op not in ("attention", "kv_centric", "kv_tokens", "fp4_scores") or work(case)["flops"] > 5e12:
        return None
    s = prepare(case, seed)
    if op == "fp4_scores":
        return _exact_scores(s, case)
    b, hkv, g, nb = case["b"], case["hkv"], case["group"], case["nb"]
    source = s["operator"] if op != "attention" else None
    q, k, v = (source.q, source.k, source.v) if source else (s["q"], s["k"], s["v"])
    ids, counts = (source.selected, None) if source else (s["ids"], s["counts"])
    if case.get("q_token_major"):
        q = q.transpose(1, 2)
    sq = q.shape[2]
    step = BLOCK
    if op == "kv_tokens":
        if 4.0 * b * hkv * g * sq * nb * BLOCK * D > 5e12:
            return None
        step = max(1, (1 << 27) // (g * nb * BLOCK))
    out = torch.empty((b, hkv * g, sq, D), dtype=torch.float64, device="cuda")
    lse = torch.empty((b, hkv * g, sq), dtype=torch.float64, device="cuda")
    everything = torch.arange(nb, device="cuda")
    lists = ids.long()
    live = counts.tolist() if counts is not None else None
    for i in range(b):
        for h in range(hkv):
            heads = slice(h * g, (h + 1) * g)
            ki, vi = (t[i, h].view(nb, BLOCK, D) for t in (k, v))
            for t in range(0, sq, step):
                rows = slice(t, min(t + step, sq))
                if op == "kv_tokens":
                    mark = torch.zeros((rows.stop - t, nb), dtype=torch.bool, device="cuda")
                    mark.scatter_(1, lists[i, h, rows], True)
                    blocks, keep = everything, mark.repeat_interleave(BLOCK, 1)
                else:
                    blocks, keep = lists[i, h, t // BLOCK], None
                    if live:
                        blocks = blocks[:live[i][h][t // BLOCK]]
                out[i, heads, rows], lse[i, heads, rows] = _attend(q[i, heads, rows], ki, vi, blocks, keep)
    return out, lse
