"""Numerics of every sm_100a kernel against the plain PyTorch fp32 reference of the same op."""
import math

import numpy as np
import pytest
import torch

from pie_b200 import ops
from pie_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def close(a, b, atol, rtol=2e-2):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    assert bool((err <= tol).all()), f"max err {err.max().item():.4g} (allowed {tol.max().item():.4g})"


def test_embed_and_shard():
    table = bf(1000, 256)
    tok = torch.randint(0, 1000, (77,), device=DEV, dtype=torch.int32)
    assert torch.equal(ops.embed(tok, table), ref.embed(tok, table))
    shard = table[250:500].contiguous()
    assert torch.equal(ops.embed(tok, shard, vocab_start=250), ref.embed(tok, shard, 250))


@pytest.mark.parametrize("hidden", [256, 2048, 4096, 5120, 8192])
def test_rmsnorm(hidden):
    x, w = bf(33, hidden, seed=1), bf(hidden, seed=2) + 1
    close(ops.rmsnorm(x, w, 1e-5), ref.rmsnorm(x, w, 1e-5), 2e-2)
    res, res2 = bf(33, hidden, seed=3), None
    res2 = res.clone()
    y = ops.add_rmsnorm(x, res, w, 1e-5)
    y2 = ref.add_rmsnorm(x, res2, w, 1e-5)
    close(res, res2, 1e-2)
    close(y, y2, 3e-2)


def test_swiglu():
    gu = bf(50, 2 * 1408, seed=4)
    close(ops.swiglu(gu), ref.swiglu(gu), 2e-2)


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_glu_interleaved(act):
    gu = bf(50, 2 * 1408, seed=4) * 3
    close(ops.glu_interleaved(gu, act), ref.glu_interleaved(gu.float(), act).to(gu.dtype), 2e-2)
    assert ops.glu_interleaved(gu[:0], act).shape == (0, 1408)


@pytest.mark.parametrize("d,hq,hkv,norm", [(128, 8, 2, False), (64, 4, 2, True), (256, 4, 1, False)])
def test_qk_norm_rope_kvwrite_with_projection_bias(d, hq, hkv, norm):
    """The projection bias added inside the kernel equals adding it to the packed rows first."""
    n, page, pages = 33, 16, 8
    qkv = bf(n, (hq + 2 * hkv) * d, seed=5)
    bias = bf((hq + 2 * hkv) * d, seed=9)
    pos = torch.randint(0, 5000, (n,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages * page, device=DEV)[:n].to(torch.int32)
    inv = ref.rope_inv_freq(d, 500000.0, None, DEV)
    qn = (bf(d, seed=6) + 1) if norm else None
    kn = (bf(d, seed=7) + 1) if norm else None
    kv_a = torch.zeros(pages, 2, hkv, page, d, dtype=torch.bfloat16, device=DEV)
    kv_b = torch.zeros_like(kv_a)
    qa = ops.qk_norm_rope_kvwrite(qkv, pos, slots, inv, qn, kn, kv_a, hq, hkv, d, page, 1e-6, bias=bias)
    qb = ops.qk_norm_rope_kvwrite(qkv + bias, pos, slots, inv, qn, kn, kv_b, hq, hkv, d, page, 1e-6)
    assert torch.equal(qa, qb) and torch.equal(kv_a, kv_b)


@pytest.mark.parametrize("d,hq,hkv,norm", [(128, 8, 2, False), (128, 8, 2, True), (64, 4, 2, True)])
def test_qk_norm_rope_kvwrite(d, hq, hkv, norm):
    n, page, pages = 41, 16, 12
    qkv = bf(n, (hq + 2 * hkv) * d, seed=5)
    pos = torch.randint(0, 5000, (n,), device=DEV, dtype=torch.int32)
    perm = torch.randperm(pages * page, device=DEV)[:n].to(torch.int32)
    perm[3] = -1
    inv = ref.rope_inv_freq(d, 500000.0, None, DEV)
    qn = (bf(d, seed=6) + 1) if norm else None
    kn = (bf(d, seed=7) + 1) if norm else None
    kv1 = torch.zeros(pages, 2, hkv, page, d, dtype=torch.bfloat16, device=DEV)
    kv2 = kv1.clone()
    q1 = ops.qk_norm_rope_kvwrite(qkv, pos, perm, inv, qn, kn, kv1, hq, hkv, d, page, 1e-6)
    q2 = ref.qk_norm_rope_kvwrite(qkv, pos, perm, inv, qn, kn, kv2, hq, hkv, d, page, 1e-6)
    close(q1, q2, 3e-2)
    close(kv1, kv2, 3e-2)


def test_gather_copy_pages():
    x = bf(100, 512, seed=8)
    idx = torch.randint(0, 100, (37,), device=DEV, dtype=torch.int32)
    assert torch.equal(ops.gather_rows(x, idx), x[idx.long()])
    kv = bf(3, 10, 2, 2, 16, 64, seed=9)
    want = kv.clone()
    src = torch.tensor([1, 4], device=DEV, dtype=torch.int32)
    dst = torch.tensor([7, 2], device=DEV, dtype=torch.int32)
    want[:, dst.long()] = want[:, src.long()]
    ops.copy_pages(kv, src, dst)
    assert torch.equal(kv, want)


def test_brle_expand():
    rng = np.random.default_rng(0)
    rows, nbits = [], 1000
    for _ in range(9):
        runs, tot = [], 0
        while tot < nbits:
            r = int(rng.integers(0, 90))
            runs.append(r)
            tot += r
        rows.append(runs)
    rows.append([0, nbits])
    rows.append([nbits])
    rows.append([5, 3])      # short vector: tail is zeros
    got = ops.brle_expand(rows, nbits, DEV).cpu()
    want = ops.brle_expand(rows, nbits, "cpu")
    assert torch.equal(got, want)


def test_brle_expand_ragged_equals_row_by_row():
    rng = np.random.default_rng(1)
    rows, bits = [], []
    for nbits in (1, 31, 32, 33, 700, 64, 5000, 17):
        for _ in range(3):
            runs, tot = [], 0
            while tot < nbits:
                r = int(rng.integers(0, 90))
                runs.append(r)
                tot += r
            rows.append(runs)
            bits.append(nbits)
    rows.append([4, 2])          # short row: the tail is zeros
    bits.append(100)
    got, offs = ops.brle_expand_ragged(rows, bits, DEV)
    assert offs[-1] == got.numel() == sum((b + 31) // 32 for b in bits)
    for i, (r, b) in enumerate(zip(rows, bits)):
        want = ops.brle_expand([r], b, "cpu").reshape(-1)
        assert torch.equal(got[offs[i]:offs[i + 1]].cpu(), want), (i, b)
    cpu, offs2 = ops.brle_expand_ragged(rows, bits, "cpu")
    assert torch.equal(cpu, got.cpu()) and np.array_equal(offs, offs2)


def make_paged(nreq, kv_lens, hkv, d, page, seed=0, extra_pages=5):
    npages = [-(-int(k) // page) for k in kv_lens]
    total = sum(npages) + extra_pages
    kv = bf(total, 2, hkv, page, d, seed=seed)
    perm = torch.randperm(total)[: sum(npages)].numpy().astype(np.int32)
    indptr = np.zeros(nreq + 1, dtype=np.int32)
    indptr[1:] = np.cumsum(npages)
    return kv, perm, indptr


@pytest.mark.parametrize("d,hq,hkv", [(128, 32, 8), (128, 8, 1), (64, 4, 2), (128, 16, 16), (128, 16, 1)])
def test_paged_decode_attention(d, hq, hkv):
    page = 16
    kv_lens = np.array([1, 15, 16, 17, 300, 1000, 2305, 64], dtype=np.int32)
    r = len(kv_lens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=11)
    q = bf(r, hq, d, seed=12)
    item_req, st, en, iptr = ops.plan_decode_items(kv_lens, hkv, target_ctas=64, min_chunk=256)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    max_items = len(item_req) + 3
    plan = ops.DecodePlan(t(pages), t(indptr), t(item_req), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(max_items, hq, d), device=DEV),
                          max_items, r, 64, page)
    scale = 1 / math.sqrt(d)
    out = ops.paged_decode_attention(q, kv, plan, scale)
    qo = np.arange(r + 1, dtype=np.int32)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale)
    close(out, want, 2e-2)


@pytest.mark.parametrize("d,hq,hkv,softcap,window", [(256, 8, 4, 0.0, -1), (256, 8, 1, 0.0, 100), (256, 16, 16, 0.0, -1), (256, 8, 2, 1.5, -1),
                                                     (128, 32, 8, 1.5, -1), (128, 16, 8, 2.0, 100), (64, 4, 2, 1.5, -1)])
def test_paged_decode_attention_head_dim_256_and_softcap(d, hq, hkv, softcap, window):
    """head_dim 256 (Gemma sizes) and soft-capped scores (softmax over cap * tanh(s / cap), Gemma-2), alone and together."""
    page = 16
    kv_lens = np.array([1, 15, 16, 17, 300, 1000, 2305, 64], dtype=np.int32)
    r = len(kv_lens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=11)
    q = bf(r, hq, d, seed=12)
    item_req, st, en, iptr = ops.plan_decode_items(kv_lens, hkv, target_ctas=64, min_chunk=256, window_left=window)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    max_items = len(item_req) + 3
    plan = ops.DecodePlan(t(pages), t(indptr), t(item_req), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(max_items, hq, d), device=DEV),
                          max_items, r, 64, page, window_left=window)
    scale = 1 / math.sqrt(d)
    out = ops.paged_decode_attention(q, kv, plan, scale, softcap=softcap)
    qo = np.arange(r + 1, dtype=np.int32)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale, window_left=window,
                               softcap=softcap)
    close(out, want, 2e-2)
    if softcap:     # the cap changes the result: the test would not pass without it
        plain = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale, window_left=window)
        assert (plain.float() - want.float()).abs().max() > 0.05


@pytest.mark.parametrize("d,hq,hkv,softcap,rows", [(256, 8, 4, 0.0, 64), (256, 4, 4, 0.0, 64), (256, 8, 1, 1.5, 64), (128, 32, 8, 1.5, 64),
                                                   (64, 4, 2, 2.0, 64), (128, 32, 8, 1.5, 256), (128, 32, 16, 2.0, 256), (128, 8, 1, 1.5, 256),
                                                   (64, 16, 2, 2.0, 256)])
@pytest.mark.parametrize("mode", ["causal", "custom", "window"])
def test_paged_prefill_attention_head_dim_256_and_softcap(d, hq, hkv, softcap, rows, mode):
    """head_dim 256 on the 64-row kernel (the tcgen05 kernel stops at 128); soft-capped scores on both kernels (the
    tcgen05 one in its two-tile form)."""
    page = 16
    assert ops.prefill_tile_rows(hq, hkv, d, page, softcap=bool(softcap)) == (64 if d == 256 else 256)
    qlens = np.array([1, 5, 64, 130, 17, 700], dtype=np.int32)
    prev = np.array([40, 0, 0, 200, 31, 333], dtype=np.int32)
    kv_lens = qlens + prev
    r = len(qlens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=21)
    qo = np.zeros(r + 1, dtype=np.int32)
    qo[1:] = np.cumsum(qlens)
    q = bf(int(qo[-1]), hq, d, seed=22)
    masks, window = None, -1
    if mode == "custom":
        rng = np.random.default_rng(5)
        masks = []
        for i in range(r):
            m = rng.random((qlens[i], kv_lens[i])) < 0.6
            m[:, 0] = True
            masks.append(m if i != 2 else None)
    if mode == "window":
        window = 37
    plan = ops.build_prefill_plan(ops.AttnBatch(qo, indptr, pages, kv_lens, masks, window), hq // hkv, page, DEV, tile_rows=rows)
    scale = 1 / math.sqrt(d)
    lse = torch.empty(int(qo[-1]), hq, device=DEV)
    out = ops.paged_prefill_attention(q, kv, plan, scale, lse_out=lse, softcap=softcap)
    ops.check_kernel_status(DEV)
    tmasks = None if masks is None else [None if m is None else torch.from_numpy(m) for m in masks]
    want, want_lse = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale,
                                         masks=tmasks, window_left=window, return_lse=True, softcap=softcap)
    close(out, want, 2e-2)
    close(lse, want_lse, 2e-2)


@pytest.mark.parametrize("d,hq,hkv", [(128, 32, 8), (128, 4, 1), (64, 16, 2), (128, 16, 16), (128, 16, 1)])
def test_paged_decode_attention_shared_prefix(d, hq, hkv):
    """Forks of one context share their leading pages: the cascade plan reads those pages once per
    tile of members and must give what the plain per-request plan gives."""
    page = 16
    rng = np.random.default_rng(5)
    tables, kv_lens = [], []
    nxt = 0
    for g, (members, shared_pages) in enumerate([(8, 40), (3, 17), (11, 64)]):
        shared = list(range(nxt, nxt + shared_pages))
        nxt += shared_pages
        for b in range(members):
            own_n = int(rng.integers(1, 9))
            tables.append(shared + list(range(nxt, nxt + own_n)))
            nxt += own_n
            kv_lens.append(shared_pages * page + (own_n - 1) * page + int(rng.integers(1, page + 1)))
    for n in (1, 3, 70):                                   # requests that share nothing
        tables.append(list(range(nxt, nxt + n)))
        nxt += n
        kv_lens.append((n - 1) * page + int(rng.integers(1, page + 1)))
    order = rng.permutation(len(tables))
    tables, kv_lens = [tables[i] for i in order], np.array([kv_lens[i] for i in order], dtype=np.int32)
    r = len(tables)
    phys = rng.permutation(nxt + 7)[:nxt].astype(np.int32)          # logical -> physical page ids
    indptr = np.zeros(r + 1, dtype=np.int32)
    indptr[1:] = np.cumsum([len(t) for t in tables])
    pages = np.concatenate([phys[np.array(t)] for t in tables]).astype(np.int32)
    kv = bf(nxt + 7, 2, hkv, page, d, seed=71)
    q = bf(r, hq, d, seed=72)
    groups = ops.find_shared_prefixes(kv_lens, indptr, pages, page, min_shared_tokens=64)
    assert sorted(len(m) for m, _ in groups) == [3, 8, 11]
    assert sorted(st for _, st in groups) == [17 * page, 40 * page, 64 * page]
    cp = ops.plan_decode_cascade(kv_lens, groups, hkv, hq // hkv, target_ctas=64, max_items=4096, min_chunk=256)
    if hq // hkv == 16:               # one request's heads fill the 16-row tile: no shared items to make
        assert cp is None
        return
    assert cp is not None and cp.shared_tokens > 0
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    max_items = int(cp.req_slot_indptr[-1]) + 5
    status = ops.kernel_status(DEV)
    status.zero_()
    plan = ops.DecodePlan(t(pages), t(indptr), t(cp.item_req), t(cp.item_start), t(cp.item_end), t(cp.req_slot_indptr),
                          torch.tensor([len(cp.item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(max_items, hq, d), device=DEV), max_items, r, 64, page,
                          item_slot=t(cp.item_slot), item_tile=t(cp.item_tile), tile_members=t(cp.tile_members))
    scale = 1 / math.sqrt(d)
    out = ops.paged_decode_attention(q, kv, plan, scale)
    torch.cuda.synchronize()
    assert int(status[0].item()) == 0
    qo = np.arange(r + 1, dtype=np.int32)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale)
    close(out, want, 2e-2)
    # attention sinks merge the same way over shared and unshared slots
    sinks = torch.linspace(-1.0, 2.0, hq, device=DEV)
    sl2 = (sinks * 1.4426950408889634).float().contiguous()
    out = ops.paged_decode_attention(q, kv, plan, scale, sinks_log2=sl2)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale, sinks=sinks)
    close(out, want, 2e-2)


def test_paged_decode_attention_clamps_work_count():
    """A work count in device memory larger than the scratch was sized for (a stale value on a graph
    replay, an embedder's mistake) must not write past the scratch: the kernel drops the extra items,
    reports PIE_ERR_BOUNDS and the requests whose items are all covered still come out right."""
    d, hq, hkv, page = 128, 32, 8, 16
    kv_lens = np.array([300, 17, 1000, 2305], dtype=np.int32)
    r = len(kv_lens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=61)
    q = bf(r, hq, d, seed=62)
    item_req, st, en, iptr = ops.plan_decode_items(kv_lens, hkv, target_ctas=64, min_chunk=256)
    covered = int(iptr[2])                       # every item of requests 0 and 1
    assert covered < len(item_req) and iptr[3] > covered + 1
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    need = ops.decode_scratch_floats(covered, hq, d)
    big = torch.full((need + 65536,), 777.0, device=DEV)
    status = ops.kernel_status(DEV)
    status.zero_()
    plan = ops.DecodePlan(t(pages), t(indptr), t(item_req), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV), big, covered, r, 64, page)
    scale = 1 / math.sqrt(d)
    out = ops.paged_decode_attention(q, kv, plan, scale)
    torch.cuda.synchronize()
    assert int(status[0].item()) == 5               # PIE_ERR_BOUNDS
    with pytest.raises(ops._lib.KernelLibraryError):
        ops.check_kernel_status(DEV)
    assert int(status[0].item()) == 0
    assert bool((big[need:] == 777.0).all())     # nothing written past the scratch
    qo = np.arange(r + 1, dtype=np.int32)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale)
    close(out[:2], want[:2], 2e-2)
    # an item that names a request outside the batch is skipped and reported as well
    bad = item_req.copy()
    bad[-1] = r + 5
    plan = ops.DecodePlan(t(pages), t(indptr), t(bad), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(len(item_req), hq, d), device=DEV),
                          len(item_req), r, 64, page)
    out = ops.paged_decode_attention(q, kv, plan, scale)
    torch.cuda.synchronize()
    assert int(status[0].item()) == 5
    status.zero_()
    close(out[:3], want[:3], 2e-2)


@pytest.mark.parametrize("d,hq,hkv", [(128, 32, 8), (64, 16, 2)])
def test_attention_sinks_and_per_call_window(d, hq, hkv):
    """Per-head sink logits in the softmax denominator (decode: single-item and merged requests;
    prefill: both kernels) and a window given per call over a plan that covers the whole range."""
    page = 16
    sinks = torch.linspace(-2.0, 3.0, hq, device=DEV)
    sl2 = (sinks * 1.4426950408889634).float().contiguous()
    scale = 1 / math.sqrt(d)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    # decode
    kv_lens = np.array([1, 17, 300, 2305, 64], dtype=np.int32)
    r = len(kv_lens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=51)
    q = bf(r, hq, d, seed=52)
    item_req, st, en, iptr = ops.plan_decode_items(kv_lens, hkv, target_ctas=64, min_chunk=256)
    max_items = len(item_req) + 3
    plan = ops.DecodePlan(t(pages), t(indptr), t(item_req), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(max_items, hq, d), device=DEV), max_items, r, 64, page)
    qo = np.arange(r + 1, dtype=np.int32)
    for window in (-1, 40):
        out = ops.paged_decode_attention(q, kv, plan, scale, window_left=window, sinks_log2=sl2)
        want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale,
                                   window_left=window, sinks=sinks)
        close(out, want, 2e-2)
    # prefill
    qlens = np.array([5, 130, 300], dtype=np.int32)
    kv_lens = qlens + np.array([40, 0, 77], dtype=np.int32)
    kv, pages, indptr = make_paged(3, kv_lens, hkv, d, page, seed=53)
    qo = np.zeros(4, dtype=np.int32)
    qo[1:] = np.cumsum(qlens)
    q = bf(int(qo[-1]), hq, d, seed=54)
    batch = ops.AttnBatch(qo, indptr, pages, kv_lens, None, -1)
    for rows in [64, 128, 256]:
        plan = ops.build_prefill_plan(batch, hq // hkv, page, DEV, tile_rows=rows)
        for window in (-1, 33):
            out = ops.paged_prefill_attention(q, kv, plan, scale, window_left=window, sinks_log2=sl2)
            want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale,
                                       window_left=window, sinks=sinks)
            close(out, want, 2e-2)
    ops.check_kernel_status(DEV)


@pytest.mark.parametrize("window", [0, 15, 16, 100, 1000])
def test_paged_decode_attention_sliding_window(window):
    """Decode attention over the last window + 1 keys only: the plan starts at the 16-token boundary
    below the first visible key and the kernel masks the keys under it."""
    d, hq, hkv, page = 128, 32, 8, 16
    kv_lens = np.array([1, 15, 16, 17, 300, 1000, 2305, 64], dtype=np.int32)
    r = len(kv_lens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=13)
    q = bf(r, hq, d, seed=14)
    item_req, st, en, iptr = ops.plan_decode_items(kv_lens, hkv, target_ctas=64, min_chunk=256, window_left=window)
    assert (st % 16 == 0).all() and (en[iptr[1:] - 1] == kv_lens).all()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(DEV)
    max_items = len(item_req) + 3
    plan = ops.DecodePlan(t(pages), t(indptr), t(item_req), t(st), t(en), t(iptr),
                          torch.tensor([len(item_req)], dtype=torch.int32, device=DEV),
                          torch.empty(ops.decode_scratch_floats(max_items, hq, d), device=DEV),
                          max_items, r, 64, page, window_left=window)
    scale = 1 / math.sqrt(d)
    out = ops.paged_decode_attention(q, kv, plan, scale)
    qo = np.arange(r + 1, dtype=np.int32)
    want = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale, window_left=window)
    close(out, want, 2e-2)


@pytest.mark.parametrize("d,hq,hkv,rows", [(128, 32, 8, 64), (128, 8, 1, 64), (64, 4, 2, 64),
                                           (128, 32, 8, 128), (128, 8, 1, 128), (128, 4, 4, 128),
                                           (128, 32, 2, 128), (128, 8, 4, 128), (128, 32, 8, 256),
                                           (128, 8, 1, 256), (128, 4, 4, 256), (128, 32, 2, 256),
                                           (64, 4, 2, 128), (64, 16, 2, 256), (64, 64, 8, 256), (64, 8, 8, 128)])
@pytest.mark.parametrize("mode", ["causal", "custom", "window", "custom_window"])
def test_paged_prefill_attention(d, hq, hkv, rows, mode):
    """rows = 64: the mma.sync kernel; rows = 128 / 256: the tcgen05 kernel with one / two MMA
    tiles per CTA (head_dim 128, 16-token pages)."""
    page = 16
    if rows > 64:
        assert ops._lib.fn("pie_prefill_attn_tc_supported")(hq, hkv, d, page) == 1
    qlens = np.array([1, 5, 64, 130, 17, 700], dtype=np.int32)
    prev = np.array([40, 0, 0, 200, 31, 333], dtype=np.int32)
    kv_lens = qlens + prev
    r = len(qlens)
    kv, pages, indptr = make_paged(r, kv_lens, hkv, d, page, seed=21)
    qo = np.zeros(r + 1, dtype=np.int32)
    qo[1:] = np.cumsum(qlens)
    q = bf(int(qo[-1]), hq, d, seed=22)
    masks = None
    window = -1
    if mode in ("custom", "custom_window"):      # custom_window: a layer's window bounds the left side under a custom mask too
        rng = np.random.default_rng(5)
        masks = []
        for i in range(r):
            m = rng.random((qlens[i], kv_lens[i])) < 0.6
            m[:, 0] = True
            masks.append(m if i != 2 else None)
    if mode in ("window", "custom_window"):
        window = 37
    batch = ops.AttnBatch(qo, indptr, pages, kv_lens, masks, window)
    plan = ops.build_prefill_plan(batch, hq // hkv, page, DEV, tile_rows=rows)
    scale = 1 / math.sqrt(d)
    lse = torch.empty(int(qo[-1]), hq, device=DEV)
    out = ops.paged_prefill_attention(q, kv, plan, scale, lse_out=lse)
    ops.check_kernel_status(DEV)
    tmasks = None if masks is None else [None if m is None else torch.from_numpy(m) for m in masks]
    want, want_lse = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale,
                                         masks=tmasks, window_left=window, return_lse=True)
    close(out, want, 2e-2)
    close(lse, want_lse, 2e-2)


@pytest.mark.parametrize("rows", [128, 256])
def test_prefill_tc_rescales_accumulator_when_scores_grow(rows):
    """Large score magnitudes make block maxima outgrow the lazily updated reference maximum, so
    the kernel's rescale of its TMEM accumulator runs in ordinary causal blocks too."""
    d, hq, hkv, page = 128, 8, 2, 16
    qlens = np.array([300, 77], dtype=np.int32)
    prev = np.array([500, 0], dtype=np.int32)
    kv_lens = qlens + prev
    kv, pages, indptr = make_paged(2, kv_lens, hkv, d, page, seed=41)
    qo = np.zeros(3, dtype=np.int32)
    qo[1:] = np.cumsum(qlens)
    q = bf(int(qo[-1]), hq, d, seed=42, scale=8.0)
    batch = ops.AttnBatch(qo, indptr, pages, kv_lens, None, -1)
    plan = ops.build_prefill_plan(batch, hq // hkv, page, DEV, tile_rows=rows)
    scale = 1 / math.sqrt(d)
    lse = torch.empty(int(qo[-1]), hq, device=DEV)
    out = ops.paged_prefill_attention(q, kv, plan, scale, lse_out=lse)
    ops.check_kernel_status(DEV)
    want, want_lse = ref.paged_attention(q, kv, qo, indptr, torch.from_numpy(pages).to(DEV), kv_lens, scale,
                                         return_lse=True)
    close(out, want, 3e-2)
    close(lse, want_lse, 5e-2, rtol=1e-2)


def test_row_stats():
    lg = bf(7, 4096, scale=3.0, seed=30)
    close(ops.row_stats(lg), ref.row_stats(lg), 2e-3, rtol=1e-3)


def _params(rows, t, k, p, mp, seed0=1):
    return (torch.full((rows,), t, device=DEV), torch.full((rows,), k, dtype=torch.int32, device=DEV),
            torch.full((rows,), p, device=DEV), torch.full((rows,), mp, device=DEV),
            torch.arange(seed0, seed0 + rows, dtype=torch.int64, device=DEV))


def test_sample_argmax_and_topk1():
    lg = bf(16, 32000, scale=2.0, seed=31)
    want = lg.float().argmax(-1).int()
    got = ops.sample(lg, *_params(16, 0.0, 0, 1.0, 0.0))
    assert torch.equal(got, want)
    got = ops.sample(lg, *_params(16, 1.0, 1, 1.0, 0.0))
    # top-k = 1 keeps every token tied with the maximum (bf16 ties are common)
    mx = lg.float().amax(-1)
    assert bool((lg.float()[torch.arange(16), got.long()] == mx).all())


@pytest.mark.parametrize("t,k,p,mp", [(1.0, 50, 1.0, 0.0), (0.8, 0, 0.9, 0.0), (1.0, 0, 1.0, 0.05), (0.7, 40, 0.95, 0.0)])
def test_sample_stays_in_kept_set(t, k, p, mp):
    rows, vocab = 64, 8192
    lg = bf(rows, vocab, scale=3.0, seed=32)
    got = ops.sample(lg, *_params(rows, t, k, p, mp)).cpu()
    lgc = lg.cpu()
    for r in range(rows):
        keep = ref.kept_set(lgc[r], t, k, p, mp)
        assert bool(keep[got[r]]), f"row {r}: token {int(got[r])} outside the kept set"


def test_sample_distribution_matches_softmax():
    vocab, draws = 64, 20000
    row = (torch.randn(vocab, generator=torch.Generator().manual_seed(3)) * 1.5).to(torch.bfloat16)
    lg = row.to(DEV).repeat(draws, 1).contiguous()
    got = ops.sample(lg, *_params(draws, 1.0, 0, 1.0, 0.0, seed0=1000)).cpu()
    freq = torch.bincount(got.long(), minlength=vocab).float() / draws
    p = torch.softmax(row.float(), -1)
    assert float((freq - p).abs().max()) < 0.02
    # same seeds -> same tokens (counter-based stream)
    again = ops.sample(lg, *_params(draws, 1.0, 0, 1.0, 0.0, seed0=1000)).cpu()
    assert torch.equal(got, again)


def test_sample_with_vocab_mask():
    rows, vocab = 8, 4096
    lg = bf(rows, vocab, scale=2.0, seed=33)
    runs = [[100, 50, 1000, 7]]           # allowed: [100,150) and [1150,1157)
    bits = ops.brle_expand(runs, vocab, DEV)
    mrow = torch.tensor([0, -1] * 4, dtype=torch.int32, device=DEV)
    got = ops.sample(lg, *_params(rows, 1.0, 0, 1.0, 0.0), mask_bits=bits, mask_row=mrow).cpu()
    for r in range(0, rows, 2):
        t = int(got[r])
        assert 100 <= t < 150 or 1150 <= t < 1157
    # greedy under a mask = arg-max over the allowed set
    got = ops.sample(lg, *_params(rows, 0.0, 0, 1.0, 0.0), mask_bits=bits, mask_row=mrow).cpu()
    allowed = torch.zeros(vocab, dtype=torch.bool)
    allowed[100:150] = True
    allowed[1150:1157] = True
    for r in range(0, rows, 2):
        want = int(lg[r].float().cpu().masked_fill(~allowed, float("-inf")).argmax())
        assert int(got[r]) == want


def test_fp8_block_dequant_and_gemm():
    """fp8 weights with per-row x 128-column scales: the dequant kernel equals the PyTorch
    expansion, and the fp8-weight GEMM (with each epilogue) equals the bf16 GEMM over it."""
    from pie_b200 import ops
    from pie_b200.ops import reference as ref
    torch.manual_seed(5)
    n, k, m = 1536, 2048, 200
    w = (torch.randn(n, k, device="cuda") * 0.05)
    q = ops.quantize_fp8_block(w)
    assert q.w8.dtype == torch.float8_e4m3fn and q.scale.shape == (n, k // 128)
    deq = ops.dequant_fp8(q)
    want = (q.w8.float() * q.scale.repeat_interleave(128, dim=1)).to(torch.bfloat16)
    assert torch.equal(deq, want)
    assert (deq.float() - w).abs().max() / w.abs().max() < 0.07
    x = (torch.randn(m, k, device="cuda") * 0.5).to(torch.bfloat16)
    r = (torch.randn(m, n, device="cuda") * 0.5).to(torch.bfloat16)
    full = x.float() @ deq.float().t()
    y = ops.gemm_fp8w(x, q, mode="dequant")
    assert (y.float() - full).abs().max() < 0.05 * full.abs().max()
    y = ops.gemm_fp8w(x, q, residual=r, epilogue=ops.EPI_RESIDUAL, mode="dequant")
    assert (y.float() - (full + r.float())).abs().max() < 0.05 * full.abs().max()
    y = ops.gemm_fp8w(x, q, epilogue=ops.EPI_SWIGLU, mode="dequant")
    assert (y.float() - ref.swiglu_interleaved(full)).abs().max() < 0.05 * full.abs().max()
    ops.check_kernel_status()


@pytest.mark.parametrize("m,n,k", [(64, 1536, 2048), (200, 1024, 5120), (512, 6400, 5120), (1000, 640, 3200), (130, 2016, 1024)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_fp8_blockscaled_gemm_fused(m, n, k, epi):
    """fp8 x fp8 tcgen05 GEMM with 1x128 activation scales and per-row x 128 weight scales against
    the fp32 evaluation of the same quantised operands; and close to the unquantised product."""
    from pie_b200 import ops
    from pie_b200.ops import reference as ref
    torch.manual_seed(m + n)
    w = torch.randn(n, k, device="cuda") * 0.05
    x = (torch.randn(m, k, device="cuda") * 0.5).to(torch.bfloat16)
    r = (torch.randn(m, n, device="cuda") * 0.5).to(torch.bfloat16) if epi == "residual" else None
    q = ops.quantize_fp8_block(w)
    x8, sx = ops.quant_act_fp8(x)
    # the quantiser itself: dequantised activations within fp8 rounding of the input
    xd = x8.float() * sx.repeat_interleave(128, dim=1)[:, :k]
    assert (xd - x.float()).abs().max() <= 0.07 * x.float().abs().max()
    want = ops.gemm_fp8_reference(x8, sx, q)
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    y = ops.gemm_fp8w(x, q, residual=r, epilogue=e, mode="fused")
    torch.cuda.synchronize()
    ops.check_kernel_status()
    tol = 2e-2 * want.abs().max().item() + 1e-3 * k ** 0.5
    assert (y.float() - want).abs().max().item() <= tol
    if epi == "store":
        exact = x.float() @ w.t()
        rel = (y.float() - exact).norm() / exact.norm()
        assert rel < 0.06, rel


@pytest.mark.parametrize("k,p", [(0, 0.6), (5, 1.0), (8, 0.8), (0, 0.05)])
def test_sample_topk_topp_distribution_is_renormalised_kept_set(k, p):
    """Draws under top-k / top-p follow the softmax renormalised over the kept set (rejection
    rounds and the radix fallback for a small top-p must agree with the reference set)."""
    vocab, draws = 64, 20000
    row = (torch.randn(vocab, generator=torch.Generator().manual_seed(9)) * 1.5).to(torch.bfloat16)
    lg = row.to(DEV).repeat(draws, 1).contiguous()
    got = ops.sample(lg, *_params(draws, 1.0, k, p, 0.0, seed0=77)).cpu()
    keep = ref.kept_set(row, 1.0, k, p, 0.0)
    assert bool(keep[got.long()].all())
    probs = torch.softmax(row.float(), -1) * keep
    probs = probs / probs.sum()
    freq = torch.bincount(got.long(), minlength=vocab).float() / draws
    assert float((freq - probs).abs().max()) < 0.02


def test_bounded_peer_wait_times_out_and_reports_status():
    """A wait on a peer flag that nothing sets gives up after its bound, records
    PIE_ERR_WAIT_PEER (4) in the status word and returns; the context stays usable and
    `check_kernel_status` raises and clears the word."""
    import ctypes as C
    import time
    from pie_b200.ops import _lib
    wait = _lib.declare("pie_tp_wait_ag", [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p])
    flags = torch.zeros(8, dtype=torch.int32, device=DEV)          # never raised
    epoch = torch.ones(1, dtype=torch.int32, device=DEV)           # the kernel expects flags >= 1
    status = ops.kernel_status(DEV)
    status.zero_()
    t0 = time.time()
    _lib.check(wait(flags.data_ptr(), epoch.data_ptr(), 2, status.data_ptr(), _lib.stream_ptr()), "tp_wait_ag")
    torch.cuda.synchronize()
    assert time.time() - t0 < 10.0
    assert int(status[0].item()) == 4
    with pytest.raises(_lib.KernelLibraryError):
        ops.check_kernel_status(DEV)
    assert int(status[0].item()) == 0
    # the device still works
    x = torch.ones(1024, device=DEV)
    assert float(x.sum()) == 1024.0
    # and a wait whose flags are already up returns at once with a clean status
    flags.fill_(1)
    _lib.check(wait(flags.data_ptr(), epoch.data_ptr(), 2, status.data_ptr(), _lib.stream_ptr()), "tp_wait_ag")
    torch.cuda.synchronize()
    assert int(status[0].item()) == 0


def test_index_validator_records_the_first_bad_entry_and_touches_nothing():
    """The `PIE_BOUNDS=1` check: entries outside [lo, hi) set PIE_ERR_BOUNDS with table and position; the
    status check raises with them and clears the block, and a clean table leaves it alone."""
    from pie_b200.ops import _lib
    ops.kernel_status(DEV).zero_()
    good = torch.arange(0, 1000, dtype=torch.int32, device=DEV)
    ops.validate_indices(good, 0, 1000, "kv_page_indices")
    torch.cuda.synchronize()
    ops.check_kernel_status(DEV)
    bad = good.clone()
    bad[637] = 1000
    ops.validate_indices(bad, 0, 1000, "kv_page_indices")
    torch.cuda.synchronize()
    with pytest.raises(_lib.KernelLibraryError, match=r"kv_page_indices\[637\]"):
        ops.check_kernel_status(DEV)
    ops.check_kernel_status(DEV)                              # cleared
    neg = good.clone()
    neg[3] = -1
    ops.validate_indices(neg, 0, 1000, "tokens")
    torch.cuda.synchronize()
    with pytest.raises(_lib.KernelLibraryError, match=r"tokens\[3\]"):
        ops.check_kernel_status(DEV)


@pytest.mark.parametrize("dk,dv,hk,hv", [(32, 32, 2, 4), (64, 64, 2, 2), (128, 128, 2, 4)])
def test_gdn_mixer_matches_reference_over_chunks(dk, dv, hk, hv):
    """Gated DeltaNet mixer kernels (short convolution with slot tails, token-serial delta rule, gated norm)
    against the fp32 reference: a ragged batch, then a second fire that continues from the cached state."""
    from types import SimpleNamespace
    from pie_b200.driver.recurrent import RecurrentStateCache
    from pie_b200.models.config import ModelConfig
    torch.manual_seed(dk + hv)
    cfg = ModelConfig(model_type="qwen3_5", num_hidden_layers=1, layer_types=["linear_attention"], linear_num_key_heads=hk,
                      linear_num_value_heads=hv, linear_key_head_dim=dk, linear_value_head_dim=dv)
    c, f = cfg.gdn_conv_channels, cfg.gdn_in_features
    lw_f = {"gdn_conv": torch.randn(c, 4) * 0.3, "gdn_A_log": torch.randn(hv) * 0.5, "gdn_dt_bias": torch.randn(hv) * 0.5,
            "gdn_norm": 1 + torch.randn(dv) * 0.1}
    lw_f = {k: v.to(torch.bfloat16).float() if k in ("gdn_conv", "gdn_norm") else v for k, v in lw_f.items()}
    lw_d = {k: (v.to(DEV).to(torch.bfloat16) if k in ("gdn_conv", "gdn_norm") else v.to(DEV)) for k, v in lw_f.items()}
    dev_cache, cpu_cache = RecurrentStateCache(cfg, 6, DEV), RecurrentStateCache(cfg, 6, "cpu")
    for lens, reset in (([5, 1, 37, 2], [1, 1, 1, 1]), ([1, 3, 1, 40], [0, 0, 0, 0]), ([2, 1, 1, 1], [1, 0, 0, 0])):
        qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        slots = np.asarray([4, 0, 2, 5], np.int32)
        mix = (torch.randn(int(qo[-1]), f) * 1.5).to(torch.bfloat16)
        want = ref.gdn_mixer(mix.float(), lw_f["gdn_conv"], lw_f["gdn_A_log"], lw_f["gdn_dt_bias"], lw_f["gdn_norm"], 1e-5,
                             hk, hv, dk, dv, qo.tolist(), cpu_cache.conv_state[0], cpu_cache.rec_state[0],
                             slots.tolist(), reset)
        got = ops.gdn_mixer(mix.to(DEV), lw_d, cfg, dev_cache.inputs(qo, slots, np.asarray(reset, np.int32)), 0)
        torch.cuda.synchronize()
        close(got.cpu(), want, 3e-2)
        assert torch.allclose(dev_cache.rec_state.cpu(), cpu_cache.rec_state, atol=2e-2, rtol=2e-2)
        assert torch.allclose(dev_cache.conv_state.cpu(), cpu_cache.conv_state, atol=1e-6)
    dev_cache.copy_slot(4, 1)
    torch.cuda.synchronize()
    assert torch.equal(dev_cache.rec_state[:, 1], dev_cache.rec_state[:, 4])
    assert torch.equal(dev_cache.conv_state[:, 1], dev_cache.conv_state[:, 4])


@pytest.mark.parametrize("heads,head_dim,state,groups", [(8, 32, 16, 2), (4, 64, 128, 1), (8, 64, 64, 4)])
def test_mamba2_mixer_matches_reference_over_chunks(heads, head_dim, state, groups):
    """Mamba-2 mixer (convolution with bias and slot tails, state-space update, gate + norm) against the fp32
    reference: a ragged batch, a second fire continuing from the cached state, and a reset."""
    from pie_b200.driver.recurrent import RecurrentStateCache
    from pie_b200.models.config import ModelConfig
    torch.manual_seed(heads + state)
    cfg = ModelConfig(model_type="mamba2_hybrid", num_hidden_layers=1, layer_types=["mamba2"], mamba_num_heads=heads,
                      mamba_head_dim=head_dim, ssm_state_size=state, mamba_n_groups=groups)
    c, f, inner = cfg.mamba_conv_channels, cfg.mamba_in_features, cfg.mamba_inner
    rb = lambda t: t.to(torch.bfloat16).float()
    lw_f = {"mamba_conv": rb(torch.randn(c, 4) * 0.3), "mamba_conv_bias": rb(torch.randn(c) * 0.1),
            "mamba_A_log": torch.randn(heads) * 0.5, "mamba_dt_bias": torch.randn(heads) * 0.5,
            "mamba_D": 1 + torch.randn(heads) * 0.2, "mamba_norm": rb(1 + torch.randn(inner) * 0.1)}
    bf = ("mamba_conv", "mamba_conv_bias", "mamba_norm")
    lw_d = {k: (v.to(DEV).to(torch.bfloat16) if k in bf else v.to(DEV)) for k, v in lw_f.items()}
    dev_cache, cpu_cache = RecurrentStateCache(cfg, 6, DEV), RecurrentStateCache(cfg, 6, "cpu")
    for lens, reset in (([5, 1, 37, 2], [1, 1, 1, 1]), ([1, 3, 1, 40], [0, 0, 0, 0]), ([2, 1, 1, 1], [1, 0, 0, 0])):
        qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        slots = np.asarray([4, 0, 2, 5], np.int32)
        mix = (torch.randn(int(qo[-1]), f) * 1.0).to(torch.bfloat16)
        want = ref.mamba2_mixer(mix.float(), lw_f["mamba_conv"], lw_f["mamba_conv_bias"], lw_f["mamba_A_log"],
                                lw_f["mamba_dt_bias"], lw_f["mamba_D"], lw_f["mamba_norm"], 1e-5, heads, head_dim, state,
                                groups, qo.tolist(), cpu_cache.conv_state[0], cpu_cache.rec_state[0], slots.tolist(), reset)
        got = ops.mamba2_mixer(mix.to(DEV), lw_d, cfg, dev_cache.inputs(qo, slots, np.asarray(reset, np.int32)), 0)
        torch.cuda.synchronize()
        close(got.cpu(), want, 3e-2)
        assert torch.allclose(dev_cache.rec_state.cpu(), cpu_cache.rec_state, atol=2e-2, rtol=2e-2)
        assert torch.allclose(dev_cache.conv_state.cpu(), cpu_cache.conv_state, atol=1e-6)


@pytest.mark.parametrize("vocab", [8, 4096, 4104, 32768, 151936, 151944, 800008, 1600000])
def test_sample_over_cluster_sizes(vocab):
    """Rows at the edges of a CTA's share and of the cluster's size, and rows too long to be kept: the drawn token's Gumbel score
    in 64 bits is the best one's up to the error of the kernel's fast logarithms (2^-22 absolute near 1: relative to -log u),
    filters keep to their set, and greedy is the arg-max."""
    rows = 3
    lg = bf(rows, vocab, scale=2.5, seed=vocab)
    seeds = torch.arange(7, 7 + rows, dtype=torch.int64)
    u64 = (1 << 64) - 1

    def splitmix(x):
        x = (x + 0x9E3779B97F4A7C15) & u64
        x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & u64
        x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & u64
        return x ^ (x >> 31)

    idx, m32 = torch.arange(vocab, device=DEV), 0xFFFFFFFF
    for k, p, mp in ((0, 1.0, 0.0), (5, 1.0, 0.0), (0, 0.3, 0.0), (0, 1.0, 0.2)):
        got = ops.sample(lg, *_params(rows, 1.0, k, p, mp, seed0=7)).long()
        for r in range(rows):
            s = splitmix(int(seeds[r]))
            h = ((idx + (s & m32) + 7 * 0x632BE5AB) & m32) * 0x9E3779B1 & m32 ^ (s >> 32)
            h = (h ^ (h >> 16)) * 0x85EBCA6B & m32
            h = (h ^ (h >> 13)) * 0xC2B2AE35 & m32
            u = (((h ^ (h >> 16)) >> 8).float() + 0.5).mul(2.0 ** -24).double()
            x = lg[r].double()
            keep = ref.kept_set(lg[r], 1.0, k, p, mp)
            score = torch.where(keep, x - x.max() - torch.log(-torch.log(u)), -math.inf)
            assert bool(keep[got[r]])
            err = 1e-4 + 4e-7 / -math.log(min(float(u[got[r]]), 1 - 2.0 ** -25)) + 4e-7 / -math.log(min(float(u[score.argmax()]), 1 - 2.0 ** -25))
            assert float(score[got[r]]) >= float(score.max()) - err
    got = ops.sample(lg, *_params(rows, 0.0, 0, 1.0, 0.0))
    first = torch.stack([(lg[r] == lg[r].max()).nonzero()[0, 0] for r in range(rows)])
    assert torch.equal(got.long(), first)
    # nothing but -inf, and rows of the lowest finite value
    lg[0] = -math.inf
    lg[1] = torch.finfo(torch.bfloat16).min
    got = ops.sample(lg, *_params(rows, 1.0, 0, 0.9, 0.0))
    assert int(got[0]) == 0 and 0 <= int(got[1]) < vocab


@pytest.mark.parametrize("dk,dv,hk,hv,lens", [
    (128, 128, 2, 4, [1, 2, 3, 4, 5, 15, 16, 17, 33]),       # walk: groups of four, stages of sixteen
    (128, 128, 2, 4, [1, 2, 1, 3, 1, 0]),                    # step: up to four tokens per request
    (128, 128, 1, 32, [7] * 10),                             # walk with four columns per lane
    (128, 32, 1, 3, [1, 1]), (64, 96, 3, 3, [1, 6, 1]), (32, 256, 1, 2, [19]), (64, 128, 2, 2, [1, 1, 2])])
def test_gdn_mixer_routes_match_reference(dk, dv, hk, hv, lens):
    """Every route of the mixer against the reference, from a state that is not zero, with one request reset, over two fires."""
    from pie_b200.driver.recurrent import RecurrentStateCache
    from pie_b200.models.config import ModelConfig
    torch.manual_seed(dk * 7 + dv + len(lens))
    cfg = ModelConfig(model_type="qwen3_5", num_hidden_layers=1, layer_types=["linear_attention"], linear_num_key_heads=hk,
                      linear_num_value_heads=hv, linear_key_head_dim=dk, linear_value_head_dim=dv)
    c, f, n = cfg.gdn_conv_channels, cfg.gdn_in_features, len(lens)
    bf32 = lambda t: t.to(torch.bfloat16).float()
    lw = {"gdn_conv": bf32(torch.randn(c, 4) * 0.3), "gdn_A_log": torch.randn(hv) * 0.5, "gdn_dt_bias": torch.randn(hv) * 0.5,
          "gdn_norm": bf32(1 + torch.randn(dv) * 0.1)}
    lw_d = {k: v.to(DEV, torch.bfloat16 if k in ("gdn_conv", "gdn_norm") else torch.float32) for k, v in lw.items()}
    dev_cache, cpu_cache = RecurrentStateCache(cfg, n + 1, DEV), RecurrentStateCache(cfg, n + 1, "cpu")
    cpu_cache.rec_state.normal_(0, 0.3)
    cpu_cache.conv_state.normal_()
    dev_cache.rec_state.copy_(cpu_cache.rec_state)
    dev_cache.conv_state.copy_(cpu_cache.conv_state)
    qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    slots = np.random.default_rng(1).permutation(n + 1)[:n].astype(np.int32)
    for reset in ([0] * (n - 1) + [1], [0] * n):
        mix = bf32(torch.randn(int(qo[-1]), f) * 1.5)
        want = ref.gdn_mixer(mix, lw["gdn_conv"], lw["gdn_A_log"], lw["gdn_dt_bias"], lw["gdn_norm"], 1e-5, hk, hv, dk, dv,
                             qo.tolist(), cpu_cache.conv_state[0], cpu_cache.rec_state[0], slots.tolist(), reset)
        got = ops.gdn_mixer(mix.to(DEV, torch.bfloat16), lw_d, cfg, dev_cache.inputs(qo, slots, np.asarray(reset, np.int32)), 0)
        torch.cuda.synchronize()
        close(got.cpu(), want, 2e-3, rtol=1e-2)                       # bf16 results of 32-bit sums
        assert torch.allclose(dev_cache.rec_state.cpu(), cpu_cache.rec_state, atol=1e-4, rtol=1e-4)
        assert torch.equal(dev_cache.conv_state.cpu(), cpu_cache.conv_state)


@pytest.mark.parametrize("d,hq,hkv", [(64, 3, 1), (128, 32, 8), (128, 5, 1), (256, 17, 2)])
def test_rope_kvwrite_of_unaligned_rows(d, hq, hkv):
    """Rows on odd boundaries take the element-wise form of the kernel: the same numbers, and the reference's."""
    n, page, width = 9, 4, (hq + 2 * hkv) * d
    packed, kn = bf(n, width, seed=5), bf(d, seed=6) + 1
    odd = torch.zeros(n, width + 3, dtype=torch.bfloat16, device=DEV)[:, 1:width + 1]
    odd.copy_(packed)
    pos = torch.tensor([0, 1, 7, 100, 4095, 8, 9, 10, 131071], dtype=torch.int32, device=DEV)
    slots = torch.tensor([3, 0, -1, 11, 5, 6, 7, 8, 9], dtype=torch.int32, device=DEV)
    freq = 500000.0 ** (-torch.arange(0, d, 2, device=DEV).float() / d)
    kv = [torch.zeros(3, 2, hkv, page, d, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    for norm in (None, kn):
        got = [ops.qk_norm_rope_kvwrite(q, pos, slots, freq, norm, norm, k, hq, hkv, d, page, 1e-5) for q, k in ((packed, kv[0]), (odd, kv[1]))]
        want = ref.qk_norm_rope_kvwrite(packed, pos, slots, freq, norm, norm, kv[2], hq, hkv, d, page, 1e-5)
        assert torch.equal(got[0], got[1]) and torch.equal(kv[0], kv[1])
        close(got[0].view(n, -1), want.reshape(n, -1), 3e-2)
        close(kv[0], kv[2], 3e-2)


@pytest.mark.parametrize("n,k", [(1, 16), (3, 1008), (7, 1024), (5, 1040), (300, 5120), (2, 25600), (9000, 144)])
def test_fp8_dequant_row_lengths(n, k):
    w8 = (torch.randn(n, k, device=DEV) * 100).clamp(-448, 448).to(torch.float8_e4m3fn)
    q = ops.Fp8Linear(w8, torch.rand(n, (k + 127) // 128, device=DEV) + 0.1)
    assert torch.equal(ops.dequant_fp8(q), (w8.float() * q.scale.repeat_interleave(128, 1)[:, :k]).to(torch.bfloat16))


@pytest.mark.parametrize("m,n,k", [(1, 128, 512), (15, 160, 528), (16, 5120, 1024), (17, 40000, 640), (48, 22016, 1168), (64, 51200, 512),
                                   (9, 640, 25600), (65, 40000, 640)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_fp8_gemm_of_small_batches(m, n, k, epi):
    """Up to 64 rows: column counts, tile heights, several tiles per CTA, K blocks that are not whole, against the fp32 evaluation
    of the same operands: one rounding to bf16 (2^-9) of 32-bit sums in another order."""
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n)
    w8 = (torch.randn(n, k, device=DEV, generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    q = ops.Fp8Linear(w8, (torch.rand(n, (k + 127) // 128, device=DEV, generator=g) + 0.5) / 50 * k ** -0.5)
    x = torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)
    r = torch.randn(m, n, device=DEV, generator=g).to(torch.bfloat16) if epi == "residual" else None
    x8, sx = ops.quant_act_fp8(x)
    want = ops.gemm_fp8_reference(x8, sx, q)
    want = want + r.float() if epi == "residual" else ref.swiglu_interleaved(want) if epi == "swiglu" else want
    code = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    y = ops.gemm_fp8w(x, q, residual=r, epilogue=code, mode="fused")
    torch.cuda.synchronize()
    ops.check_kernel_status()
    torch.testing.assert_close(y.float(), want, rtol=2 ** -8, atol=1e-3)


@pytest.mark.parametrize("m,n,k", [(33, 28672, 2064), (8, 57344, 1552), (33, 7008, 640), (60, 28672, 528), (64, 14336, 1168), (24, 4096, 1024),
                                   (50, 4000, 528), (3, 8192, 1664), (64, 6144, 912),
                                   (1, 24576, 2064)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_fp8_gemm_of_small_batches_in_tiles_of_every_height(m, n, k, epi):
    """Tiles of 104 and 112 rows (the last quarter live in part, MMA rows that overlap the batch's), of 64 (two quarters), 96 and 128, one to four
    per CTA, a last one that is not whole, K blocks that are no multiple of a group: as above, one rounding to bf16 (2^-9) of 32-bit sums in another
    order."""
    test_fp8_gemm_of_small_batches(m, n, k, epi)


@pytest.mark.parametrize("n,k", [(2048, 2048), (2064, 2048), (128, 2064), (2048, 2032)])
def test_fp8_gemm_rows_are_the_same_on_either_side_of_the_small_batches(n, k):
    """48 / 49 and 64 / 65 rows, features and K around which products change kernels: a row's bits do not depend on the kernel."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    w8 = (torch.randn(n, k, device=DEV, generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    q = ops.Fp8Linear(w8, (torch.rand(n, (k + 127) // 128, device=DEV, generator=g) + 0.5) / 50 * k ** -0.5)
    x = torch.randn(65, k, device=DEV, generator=g).to(torch.bfloat16)
    want = ops.gemm_fp8w(x, q, mode="fused")
    for m in (1, 48, 49, 64):
        assert torch.equal(ops.gemm_fp8w(x[:m], q, mode="fused"), want[:m]), m
    ops.check_kernel_status()


@pytest.mark.parametrize("vocab", [1024, 32000, 128256, 151936])
@pytest.mark.parametrize("k,base", [(0, None), (0, 0.3), (0, 0.03), (3000, 0.02)])
def test_sample_does_not_depend_on_the_batch_or_the_run(vocab, k, base):
    """A seed's token stays the same from run to run and whatever shares the batch, also where top-p lies on the edge of a key's mass
    to the last bits: a sum in another order would move some of these rows to the other side. Edges: of the first candidate's key
    (base None: rejection rounds), else of the keys around a mass of `base` (exact search)."""
    rows, near = 300, 75
    lg = bf(1, vocab, scale=2.5, seed=vocab).repeat(rows, 1)
    levels, inverse = torch.unique(lg[0].float(), return_inverse=True)
    mass = torch.zeros(len(levels), dtype=torch.float64, device=DEV).index_add_(0, inverse, torch.softmax(lg[0].double(), 0))
    above = mass.sum() - mass.cumsum(0)                                           # of the keys over each

    def draw(a, p, seeds):
        n = len(seeds[a])
        return ops.sample(lg[:n], torch.ones(n, device=DEV), torch.full((n,), k, dtype=torch.int32, device=DEV), p[a],
                          torch.zeros(n, device=DEV), seeds[a])

    many = torch.arange(1, rows + 1, dtype=torch.int64, device=DEV)
    for turn in range(4):
        if base is None:
            first = draw(slice(0, rows), torch.full((rows,), 1 - 2.0 ** -24, device=DEV), many + turn * rows).long()
            edge = above[inverse[first]]
            at = ((edge > 0.5) & (edge < 0.99)).nonzero().flatten()[:rows // near]
            edge, seed = edge[at], (many + turn * rows)[at]
        else:
            edge = above[(above - base).abs().argsort()[turn * 4:turn * 4 + 4]]
            seed = many[turn * 4:turn * 4 + 4]
        ulp = (torch.arange(near, device=DEV) - near // 2).double() * 2.0 ** -24
        p = (edge[:, None] * (1 + ulp)).flatten().float().clamp(max=1 - 2.0 ** -24)
        seeds = seed[:, None].repeat(1, near).flatten()
        want = draw(slice(0, len(p)), p, seeds)
        for step in (len(p), len(p), 148, 40, 1):
            got = torch.cat([draw(slice(a, min(a + step, len(p))), p, seeds) for a in range(0, len(p), step)])
            assert torch.equal(got, want), (step, int((got != want).sum()))


def test_sample_top_p_of_nothing_is_the_arg_max():
    """top_p = 0 keeps no mass: the lowest index of the largest entries, however many are equal and whatever else is asked for."""
    rows, vocab = 40, 32000
    lg = bf(rows, vocab, scale=2.0, seed=77)
    for r in range(rows):
        lg[r, torch.randperm(vocab, device=DEV)[: 1 + r * 7]] = 30.0
    want = torch.stack([(lg[r] == 30.0).nonzero()[0, 0] for r in range(rows)])
    for t, k, mp in ((1.0, 0, 0.0), (0.7, 50, 0.0), (5.0, 0, 0.1)):
        assert torch.equal(ops.sample(lg, *_params(rows, t, k, 0.0, mp)).long(), want)


def test_sample_at_an_infinite_temperature():
    """All allowed entries weigh the same, entries outside the mask and past the row's end nothing: top-p keeps that share of the keys."""
    rows, vocab = 64, 1000
    lg = torch.randperm(vocab, device=DEV).float().mul(0.25).to(torch.bfloat16).repeat(rows, 1)
    allowed = torch.zeros(vocab, dtype=torch.bool, device=DEV)
    allowed[::2] = True
    words = torch.zeros(32 * 32, dtype=torch.int64, device=DEV)
    words[:vocab] = allowed
    words = (words.view(32, 32) << torch.arange(32, device=DEV)).sum(1)
    mask = torch.where(words >= 2 ** 31, words - 2 ** 32, words).int()[None]
    for p in (0.2, 0.6):
        got = ops.sample(lg, *_params(rows, math.inf, 0, p, 0.0), mask_bits=mask, mask_row=torch.zeros(rows, dtype=torch.int32, device=DEV)).long()
        x = lg[0].float()
        higher = torch.stack([(allowed & (x > x[g])).sum() for g in got])
        assert bool(allowed[got].all()) and bool((higher < p * allowed.sum()).all()) and len(got.unique()) > 20


@pytest.mark.parametrize("dk,dv,hk,hv", [(32, 32, 2, 2), (32, 64, 1, 2), (64, 64, 2, 4), (64, 96, 1, 3), (128, 64, 2, 2), (128, 96, 1, 2),
                                         (32, 160, 1, 2), (64, 256, 2, 2)])
def test_gdn_short_requests_of_all_head_sizes(dk, dv, hk, hv):
    """The step up to its last token and the walk from there on: columns that fill a group of lanes and columns that do not."""
    for lens in ([1, 2, 1, 3, 1, 0, 1], [4, 1, 4], [5, 1, 0]):
        test_gdn_mixer_routes_match_reference(dk, dv, hk, hv, lens)


@pytest.mark.parametrize("d,hq,hkv", [(64, 1, 1), (64, 3, 1), (64, 32, 8), (128, 1, 1), (128, 4, 1), (128, 6, 2), (128, 12, 2), (128, 64, 8),
                                      (256, 2, 1), (256, 16, 2)])
def test_rope_kvwrite_splits_of_blocks(d, hq, hkv):
    """Several tokens per block, heads over several blocks and heads in turn: the reference's numbers, and those of every token alone."""
    page = 16
    freq = 500000.0 ** (-torch.arange(0, d, 2, device=DEV).float() / d)
    for n in (1, 2, 7, 33, 148, 149, 300):
        packed, qn, kn = bf(n, (hq + 2 * hkv) * d, seed=n), bf(d, seed=7) + 1, bf(d, seed=8) + 1
        pos = torch.randint(0, 100000, (n,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(n)).int()
        slots = torch.randperm(n, device=DEV).int()
        if n > 2:
            slots[n // 2] = -1
        pages = -(-max(n, 16) // page)
        kv = [torch.zeros(pages, 2, hkv, page, d, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
        norm = lambda q, k, a: ops.qk_norm_rope_kvwrite(q[a], pos[a], slots[a], freq, qn, kn, k, hq, hkv, d, page, 1e-5)
        got = norm(packed, kv[0], slice(None))
        want = ref.qk_norm_rope_kvwrite(packed, pos, slots, freq, qn, kn, kv[1], hq, hkv, d, page, 1e-5)
        close(got.view(n, -1), want.reshape(n, -1), 3e-2)
        close(kv[0], kv[1], 3e-2)
        one = torch.cat([norm(packed, kv[2], slice(t, t + 1)) for t in range(n)])
        assert torch.equal(one, got) and torch.equal(kv[2], kv[0])


@pytest.mark.parametrize("parts", [1, 2, 7, 8, 9, 31, 32, 33, 40, 64, 65, 129])
@pytest.mark.parametrize("d,group", [(64, 1), (128, 4), (256, 2)])
def test_merge_of_decode_parts(parts, d, group):
    """Parts of split requests, added up eight and weighed 32 at a time: counts around both, requests of one part (left alone) and of none
    beside them, parts without a visible key, a plan that ends before the last part, sinks. Against 64 bits: one rounding to bf16 (2^-9)."""
    import ctypes as C
    from pie_b200.ops import _lib
    hkv, max_items = 2, 2 * parts + 2
    hq = hkv * group
    g = torch.Generator(device=DEV).manual_seed(parts * 7 + d)
    counts = [parts, 1, 0, parts, 3]                              # the last one's parts lie beyond max_items in part
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    o = torch.randn(int(indptr[-1]), hq, d, generator=g, device=DEV)
    lse = torch.randn(int(indptr[-1]), hq, generator=g, device=DEV) * 4
    lse[torch.rand(lse.shape, generator=g, device=DEV) < 0.2] = -float("inf")
    sinks = torch.randn(hq, generator=g, device=DEV)
    out = torch.full((len(counts), hq, d), 7.0, dtype=torch.bfloat16, device=DEV)
    ip = torch.from_numpy(indptr).to(DEV)
    merge = _lib.declare("pie_decode_merge", [C.c_void_p] * 4 + [C.c_int] * 4 + [C.c_void_p, C.c_int, C.c_void_p])
    assert merge(o.data_ptr(), lse.data_ptr(), ip.data_ptr(), out.data_ptr(), len(counts), hq, hkv, d, sinks.data_ptr(), max_items,
                 torch.cuda.current_stream().cuda_stream) == 0
    for r in range(len(counts)):
        a, b = int(indptr[r]), min(int(indptr[r + 1]), max_items)
        if b - a <= 1:
            assert bool((out[r] == 7.0).all())
            continue
        w = torch.exp2(lse[a:b].double())
        total = w.sum(0) + torch.exp2(sinks.double())
        want = (w[..., None] * o[a:b].double()).sum(0) / total[:, None]
        want[w.sum(0) == 0] = 0.0
        torch.testing.assert_close(out[r].double(), want, rtol=2 ** -8, atol=1e-5)


@pytest.mark.parametrize("parts,cut", [(2, 1), (7, 3), (9, 1), (31, 3), (32, 1), (33, 8), (40, 5), (65, 33), (129, 3)])
@pytest.mark.parametrize("sinks", [False, True])
def test_merge_of_decode_parts_of_a_plan_that_ends_inside_a_request(parts, cut, sinks):
    """A plan that holds all but the last parts of a request, also inside 8 and 32 of them: what it holds is merged, and what lies beyond
    (here numbers that would show) is neither added nor weighed. Against 64 bits: one rounding to bf16 (2^-9)."""
    import ctypes as C
    from pie_b200.ops import _lib
    hkv, group, d = 2, 4, 128
    hq = hkv * group
    counts = [parts, 1, 0, parts, parts + 5]
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    max_items = int(indptr[-1]) - cut
    g = torch.Generator(device=DEV).manual_seed(parts * 7 + cut)
    o = torch.randn(int(indptr[-1]), hq, d, generator=g, device=DEV)
    lse = torch.randn(int(indptr[-1]), hq, generator=g, device=DEV) * 4
    o[max_items:], lse[max_items:] = 1e30, 100.0
    sink = torch.randn(hq, generator=g, device=DEV) if sinks else None
    out = torch.full((len(counts), hq, d), 7.0, dtype=torch.bfloat16, device=DEV)
    ip = torch.from_numpy(indptr).to(DEV)
    merge = _lib.declare("pie_decode_merge", [C.c_void_p] * 4 + [C.c_int] * 4 + [C.c_void_p, C.c_int, C.c_void_p])
    assert merge(o.data_ptr(), lse.data_ptr(), ip.data_ptr(), out.data_ptr(), len(counts), hq, hkv, d, sink.data_ptr() if sinks else None,
                 max_items, torch.cuda.current_stream().cuda_stream) == 0
    for r in range(len(counts)):
        a, b = int(indptr[r]), min(int(indptr[r + 1]), max_items)
        if b - a <= 1:
            assert bool((out[r] == 7.0).all())
            continue
        w = torch.exp2(lse[a:b].double())
        total = w.sum(0) + (torch.exp2(sink.double()) if sinks else 0.0)
        want = (w[..., None] * o[a:b].double()).sum(0) / total[:, None]
        torch.testing.assert_close(out[r].double(), want, rtol=2 ** -8, atol=1e-5)
