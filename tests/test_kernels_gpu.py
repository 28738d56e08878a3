"""Each kernel alone against its plain reference, at other sizes than the engine's tests,
with inputs made so that an addressing fault shows (a far key that dominates, a window's
edge, stale and non-finite contents in unused cache rows)."""
import math

import numpy as np
import pytest
import torch

import plain_llama as pl
from helpers import TOL, rel_err

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def _i32(x, dev):
    return torch.tensor(x, dtype=torch.int32, device=dev)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,hidden,vocab", [(7, 72, 101), (3, 2048, 50)])
def test_embed_gather(cuda, dtype, rows, hidden, vocab):
    from camelid_b200.csrc import ops
    table = torch.randn(vocab, hidden).to(DT[dtype]).to(cuda)
    toks = torch.randint(0, vocab, (rows,), dtype=torch.int32, device=cuda)
    out = torch.empty(rows, hidden, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    ops.embed_gather(table, toks, out, err)
    assert torch.equal(out, table.float()[toks.long()]) and int(err) == 0
    toks[1] = vocab
    ops.embed_gather(table, toks, out, err)
    assert int(err) == 1 and float(out[1].abs().max()) == 0.0


@pytest.mark.parametrize("out_dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("w_dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,hidden,eps", [(5, 72, 1e-5), (2, 3000, 1e-6), (1, 16, 1e-2)])
def test_rmsnorm(cuda, out_dtype, w_dtype, rows, hidden, eps):
    from camelid_b200.csrc import ops
    x = (torch.randn(rows + 3, hidden) * 3).to(cuda)
    w = (1 + 0.1 * torch.randn(hidden)).to(DT[w_dtype]).to(cuda)
    idx = _i32([(r * 2) % (rows + 3) for r in range(rows)], cuda)
    out = torch.empty(rows, hidden, dtype=DT[out_dtype], device=cuda)
    ops.rmsnorm(x, w, eps, out, idx)
    ref = pl.rms_norm(x.cpu().double()[idx.cpu().long()], w.cpu().double(), eps)
    tol = 1e-5 if out_dtype == "float32" else 2 ** -8
    assert rel_err(out.cpu(), ref) <= tol
    ops.rmsnorm(x, w, eps, out[:1], None)
    assert rel_err(out[:1].cpu(), pl.rms_norm(x[:1].cpu().double(), w.cpu().double(), eps)) <= tol


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [(1, 40, 24), (70, 130, 200), (129, 64, 1030), (5, 517, 96), (300, 520, 136),
                                   (2048, 384, 2048), (64, 129, 4), (257, 128, 20)])
def test_gemm_simt_epilogues(cuda, dtype, M, N, K):
    from camelid_b200.csrc import ops
    a = torch.randn(M, K).to(DT[dtype]).to(cuda)
    w = (torch.randn(N, K) / math.sqrt(K)).to(DT[dtype]).to(cuda)
    ref = a.cpu().double() @ w.cpu().double().T
    tol = 1e-5 if dtype == "float32" else 2 ** -8
    c = torch.empty(M, N, dtype=DT[dtype], device=cuda)
    ops.gemm_tn_simt(a, w, c, ops.EPI_STORE)
    assert rel_err(c.cpu(), ref) <= tol
    c32 = torch.empty(M, N, device=cuda)
    ops.gemm_tn_simt(a, w, c32, ops.EPI_STORE_F32)
    assert rel_err(c32.cpu(), ref) <= 1e-5
    res = torch.randn(M, N, device=cuda)
    want = res.cpu().double() + ref
    ops.gemm_tn_simt(a, w, res, ops.EPI_ADD_F32)
    assert rel_err(res.cpu(), want) <= 1e-5
    # rows of a wider matrix (strided views), as the attention mixer uses
    wide = torch.randn(M, K + 8).to(DT[dtype]).to(cuda)
    ops.gemm_tn_simt(wide[:, 8:], w, c32, ops.EPI_STORE_F32)
    assert rel_err(c32.cpu(), wide[:, 8:].cpu().double() @ w.cpu().double().T) <= 1e-5


@pytest.mark.parametrize("M,N,K", [(1, 3072, 2048), (8, 2048, 2048), (8, 2048, 8192), (5, 517, 132), (32, 100, 640),
                                   (17, 33, 4100), (2, 128256, 256), (8, 40, 128), (64, 96, 640), (41, 2048, 2048)])
def test_gemv_float_streaming_form(cuda, M, N, K):
    """Float products of at most 64 rows whose sizes allow 16-byte loads: tiles of 32 weight rows,
    K split over blocks where there are few tiles, the splits summed in index order by the
    block that comes last. Every epilogue; tickets are left zero, so a second call is as good; a row's
    value does not depend on the other rows of the step."""
    from camelid_b200.csrc import ops
    g = torch.Generator().manual_seed(M * 1000 + N + K)
    a = torch.randn(M, K, generator=g).to(cuda)
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).to(cuda)
    ref = a.cpu().double() @ w.cpu().double().T
    for rep in range(2):
        c = torch.full((M, N), float("nan"), device=cuda)
        ops.gemm_tn_simt(a, w, c, ops.EPI_STORE_F32)
        assert rel_err(c.cpu(), ref) <= 2e-6, rep
    res = torch.randn(M, N, generator=g).to(cuda)
    want = res.cpu().double() + ref
    ops.gemm_tn_simt(a, w, res, ops.EPI_ADD_F32)
    assert rel_err(res.cpu(), want) <= 2e-6
    one = torch.empty(1, N, device=cuda)
    ops.gemm_tn_simt(a[M - 1:], w, one, ops.EPI_STORE_F32)
    assert torch.equal(one[0], c[M - 1]), "a row alone differs from the same row in a step of several"
    # products of other shapes share the scratch: their sums must not land on this one's tickets
    other = torch.randn(8, 4096, generator=g).to(cuda)
    ops.gemm_tn_simt(other, torch.randn(64, 4096, generator=g).to(cuda), torch.empty(8, 64, device=cuda), ops.EPI_STORE_F32)
    ops.gemm_tn_simt(a, w, c, ops.EPI_STORE_F32)
    assert rel_err(c.cpu(), ref) <= 2e-6
    if N % 32 == 0:
        inter = N // 2
        act = torch.full((M, inter), float("nan"), device=cuda)
        from camelid_b200.parts.linear import pack_gate_up
        packed = pack_gate_up(w[:inter].contiguous(), w[inter:].contiguous(), 16)
        ops.gemm_tn_simt(a, packed, act, ops.EPI_SWIGLU, 16)
        gate, up = ref[:, :inter], ref[:, inter:]
        assert rel_err(act.cpu(), (gate / (1 + torch.exp(-gate))) * up) <= 2e-6
    # rows of a wider matrix (a strided view whose rows still start on 16-byte boundaries)
    wide = torch.randn(M, K + 8, generator=g).to(cuda)
    ops.gemm_tn_simt(wide[:, 8:], w, c, ops.EPI_STORE_F32)
    assert rel_err(c.cpu(), wide[:, 8:].cpu().double() @ w.cpu().double().T) <= 2e-6
    assert int(ops.simt_error_word(cuda).item()) == 0


@pytest.mark.parametrize("M,N,K", [(1, 3072, 2048), (8, 2048, 2048), (8, 2048, 8192), (5, 517, 260), (3, 33, 4100),
                                   (8, 40, 256), (7, 100, 648), (64, 2048, 2048), (19, 96, 1024)])
def test_gemv_float_partial_sums(cuda, M, N, K):
    """The streaming float product with its K ranges left as partial sums: their sum in range order is the
    product; ranges do not overlap or leave a gap (a row of ones against weights that name their column)."""
    from camelid_b200.csrc import ops
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g).to(cuda)
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).to(cuda)
    splits = ops.gemv_f32_partial_splits(a, w)
    assert splits >= 1
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    part = torch.full((splits, M, N), float("nan"), device=cuda)
    ops.gemv_f32_partial(a, w, part, err)
    assert int(err.item()) == 0
    assert rel_err(part.sum(0).cpu(), a.cpu().double() @ w.cpu().double().T) <= 2e-6
    ones = torch.ones(M, K, device=cuda)
    cols = torch.arange(K, dtype=torch.float32, device=cuda).repeat(N, 1).contiguous()
    ops.gemv_f32_partial(ones, cols, part, err)
    per = part[:, 0, 0].cpu().double()
    assert (per > 0).all() or K < 256, per                   # no empty range
    assert float(per.sum()) == K * (K - 1) / 2               # exact in float up to 2^24 per range
    assert ops.gemv_f32_partial_splits(torch.randn(65, K, device=cuda), w) == 0      # more than 64 rows: not taken


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,inter,K,group", [(3, 48, 40, 16), (66, 136, 72, 136), (9, 160, 64, 16), (200, 160, 64, 16),
                                             (129, 8192, 256, 16), (64, 16, 12, 16)])
def test_gemm_swiglu_and_packing(cuda, dtype, M, inter, K, group):
    from camelid_b200.csrc import ops
    from camelid_b200.parts.linear import pack_gate_up
    x = torch.randn(M, K).to(DT[dtype]).to(cuda)
    wg = (torch.randn(inter, K) / math.sqrt(K)).to(DT[dtype]).to(cuda)
    wu = (torch.randn(inter, K) / math.sqrt(K)).to(DT[dtype]).to(cuda)
    packed = pack_gate_up(wg, wu, group)
    g = x.cpu().double() @ wg.cpu().double().T
    u = x.cpu().double() @ wu.cpu().double().T
    ref = (g / (1 + torch.exp(-g))) * u
    act = torch.empty(M, inter, dtype=DT[dtype], device=cuda)
    ops.gemm_tn_simt(x, packed, act, ops.EPI_SWIGLU, group)
    tol = 1e-5 if dtype == "float32" else 2 ** -7
    assert rel_err(act.cpu(), ref) <= tol
    gu = torch.empty(M, 2 * inter, dtype=DT[dtype], device=cuda)
    ops.gemm_tn_simt(x, packed, gu, ops.EPI_STORE)
    act2 = torch.empty_like(act)
    ops.swiglu_packed(gu, act2, group)
    assert rel_err(act2.cpu(), ref) <= (1e-5 if dtype == "float32" else 2 ** -6)


def _paged(seq_lens, n_kv, hd, dtype, dev, n_pages=64, seed=0):
    """Random keys and values for sequences of the given lengths, scattered over shuffled
    pages; unused rows hold NaN."""
    g = torch.Generator().manual_seed(seed)
    k_pages = torch.full((n_pages, n_kv, 64, hd), float("nan")).to(dtype)
    v_pages = torch.full((n_pages, n_kv, 64, hd), float("nan")).to(dtype)
    perm = torch.randperm(n_pages, generator=g).tolist()
    tables, ks, vs = [], [], []
    for n in seq_lens:
        k = torch.randn(n, n_kv, hd, generator=g).to(dtype)
        v = torch.randn(n, n_kv, hd, generator=g).to(dtype)
        blocks = [perm.pop() for _ in range((n + 63) // 64)]
        for p in range(n):
            k_pages[blocks[p // 64], :, p % 64] = k[p]
            v_pages[blocks[p // 64], :, p % 64] = v[p]
        tables.append(blocks)
        ks.append(k)
        vs.append(v)
    width = max(len(t) for t in tables)
    table = torch.tensor([t + [-1] * (width - len(t)) for t in tables], dtype=torch.int32)
    return k_pages.to(dev), v_pages.to(dev), table.to(dev), ks, vs


def _attn_case(cuda, dtype, n_heads, n_kv, hd, starts, news, window, decode, n_splits=1, spike=None):
    from camelid_b200.csrc import ops
    dt = DT[dtype]
    totals = [s + n for s, n in zip(starts, news)]
    k_pages, v_pages, table, ks, vs = _paged(totals, n_kv, hd, dt, cuda)
    g = torch.Generator().manual_seed(1)
    n_rows = sum(news)
    q = torch.randn(n_rows, n_heads, hd, generator=g).to(dt)
    row0 = [sum(news[:i]) for i in range(len(news))]
    if spike is not None:            # one far key gets a score that stands out for one query
        seq, key = spike
        r = row0[seq] + news[seq] - 1
        ks[seq][key] *= 0
        ks[seq][key, :, 0] = 8.0
        q[r, :, 0] = 8.0 * math.sqrt(hd) / 4
        k_pages[int(table[seq, key // 64]), :, key % 64] = ks[seq][key].to(cuda)
    rows, hpc, chunks = ops.attn_tiling(n_heads, n_kv, decode)
    tile_seq, tile_q0 = [], []
    for i, n in enumerate(news):
        for q0 in range(0, n, rows):
            tile_seq.append(i)
            tile_q0.append(q0)
    out = torch.empty(n_rows, n_heads * hd, dtype=dt, device=cuda)
    partial = torch.empty(max(1, ops.attn_partial_floats(n_rows, n_heads, hd, n_splits)), device=cuda)
    ops.attn_paged_simt(q.view(n_rows, -1).to(cuda), out, k_pages, v_pages, table, _i32(tile_seq, cuda),
                        _i32(tile_q0, cuda), len(tile_seq), _i32(row0, cuda), _i32(starts, cuda), _i32(news, cuda),
                        n_rows, n_heads, n_kv, hd, rows, hpc, chunks, n_splits, window or 0, 1 / math.sqrt(hd), partial)
    out = out.cpu().view(n_rows, n_heads, hd)
    for i, (s, n) in enumerate(zip(starts, news)):
        qfull = torch.zeros(s + n, n_heads, hd, dtype=torch.float64)
        qfull[s:] = q[row0[i]:row0[i] + n].double()
        ref = pl.attention(qfull, ks[i].double(), vs[i].double(), window)[s:]
        e = rel_err(out[row0[i]:row0[i] + n], ref)
        assert e <= (1e-5 if dtype == "float32" else 2 ** -7), f"sequence {i}: {e}"
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n_heads,n_kv,hd", [(4, 2, 16), (6, 1, 32), (5, 5, 48), (8, 2, 128), (34, 1, 64), (2, 1, 256)])
def test_attention_prefill_shapes(cuda, dtype, n_heads, n_kv, hd):
    _attn_case(cuda, dtype, n_heads, n_kv, hd, starts=[0, 0, 0], news=[1, 70, 129], window=None, decode=False)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_continues_from_cache_and_far_key(cuda, dtype):
    """New rows on top of cached positions; one key hundreds of positions back dominates the
    last query of the second sequence: if a page were addressed wrongly it would show."""
    out = _attn_case(cuda, dtype, 4, 2, 32, starts=[64, 300, 5], news=[3, 20, 64], window=None, decode=False,
                     spike=(1, 7))
    assert out is not None


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n_splits", [1, 2, 5, 16])
def test_attention_decode_splits(cuda, dtype, n_splits):
    """One new row per sequence, keys split over several blocks (also more splits than pages)."""
    _attn_case(cuda, dtype, 8, 2, 64, starts=[0, 63, 64, 700], news=[1, 1, 1, 1], window=None, decode=True,
               n_splits=n_splits, spike=(3, 130))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n_heads,n_kv,hd", [(3, 1, 16), (6, 1, 48), (5, 5, 32), (12, 2, 128), (2, 1, 256), (34, 1, 64)])
def test_attention_decode_shapes(cuda, dtype, n_heads, n_kv, hd):
    """Decode tiling of the float kernel at other groupings and head sizes: groups that do not fill a block's 2 or
    4 heads (3, 6, 34 heads on one kv head), single heads (their own warp each), the largest head size (one
    page deep)."""
    _attn_case(cuda, dtype, n_heads, n_kv, hd, starts=[0, 5, 64, 130], news=[1, 1, 1, 1], window=None, decode=True,
               n_splits=2, spike=(3, 70))
    _attn_case(cuda, dtype, n_heads, n_kv, hd, starts=[17, 200], news=[1, 1], window=40, decode=True, n_splits=1)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("edge", [0, 1], ids=["first key outside", "first key inside"])
@pytest.mark.parametrize("window", [1, 64, 70, 199])
def test_attention_window_edges(cuda, dtype, window, edge):
    """The query at position 199 sees keys 200 - window .. 199. A key just outside the window must
    not count and the first one inside must: the outstanding key sits on each in turn."""
    _attn_case(cuda, dtype, 4, 2, 32, starts=[0, 190], news=[150, 10], window=window, decode=False,
               spike=(1, 199 - window + edge))
    _attn_case(cuda, dtype, 4, 2, 32, starts=[199, 80], news=[1, 1], window=window, decode=True, n_splits=3,
               spike=(0, 199 - window + edge))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n_heads,n_kv,hd,rot", [(4, 2, 16, 16), (3, 1, 48, 32), (2, 2, 64, 0), (32, 8, 64, 64), (5, 1, 128, 64),
                                                 (3, 3, 48, 24), (2, 1, 32, 6)])
def test_rope_kv_write(cuda, dtype, n_heads, n_kv, hd, rot):
    from camelid_b200.csrc import ops
    from camelid_b200.parts.position import rotary_frequencies
    dt = DT[dtype]
    cfg = {"hidden_size": rot, "num_attention_heads": 1, "head_dim": rot, "rope_theta": 10000.0}
    freqs = rotary_frequencies(rot, 10000.0, None) if rot else np.zeros(0, dtype=np.float32)
    if rot:
        assert np.array_equal(freqs, pl.rope_frequencies(cfg))
    positions = [0, 1, 63, 64, 130, 5]
    seqs = [0, 0, 0, 0, 0, 1]
    table = _i32([[9, 2, 4], [7, -1, -1]], cuda)
    width = (n_heads + 2 * n_kv) * hd
    qkv = torch.randn(len(positions), width + 5).to(dt)
    k_pages = torch.zeros(12, n_kv, 64, hd, dtype=dt, device=cuda)
    v_pages = torch.zeros_like(k_pages)
    dev = qkv.to(cuda)[:, :width]
    ops.rope_kv_write(dev, _i32(positions, cuda), _i32(seqs, cuda), table, k_pages, v_pages,
                      torch.from_numpy(freqs).to(cuda), rot, n_heads, n_kv, hd, True)
    q = qkv[:, :n_heads * hd].double().view(-1, n_heads, hd)
    k = qkv[:, n_heads * hd:(n_heads + n_kv) * hd].double().view(-1, n_kv, hd)
    v = qkv[:, (n_heads + n_kv) * hd:width].view(-1, n_kv, hd)
    pos = torch.tensor(positions)
    q_ref = pl.rope(q, pos, freqs) if rot else q
    k_ref = pl.rope(k, pos, freqs) if rot else k
    tol = 1e-6 if dtype == "float32" else 2 ** -8
    assert rel_err(dev.cpu()[:, :n_heads * hd].view(-1, n_heads, hd), q_ref) <= tol
    tab = table.cpu()
    for r, (p, s) in enumerate(zip(positions, seqs)):
        page = int(tab[s, p // 64])
        assert rel_err(k_pages[page, :, p % 64].cpu(), k_ref[r]) <= tol
        assert torch.equal(v_pages[page, :, p % 64].cpu(), v[r])
    assert int((k_pages != 0).any(dim=-1).sum()) <= len(positions) * n_kv     # nothing else was written
    before = k_pages.clone()
    ops.rope_kv_write(dev, _i32(positions, cuda), _i32(seqs, cuda), table, k_pages, v_pages,
                      torch.from_numpy(freqs).to(cuda), rot, n_heads, n_kv, hd, False)
    assert torch.equal(before, k_pages)


def test_kernels_refuse_what_they_cannot_do(cuda):
    from camelid_b200 import KernelError
    from camelid_b200.csrc import ops
    with pytest.raises(KernelError):
        ops.rmsnorm(torch.zeros(2, 8), torch.ones(8), 1e-5, torch.zeros(2, 8))          # CPU tensors
    with pytest.raises(KernelError):
        ops.dtype_code(torch.float16)
    a = torch.zeros(4, 8, device=cuda)
    with pytest.raises(KernelError):
        ops.gemm_tn_simt(a, torch.zeros(6, 8, device=cuda), torch.zeros(4, 3, device=cuda), ops.EPI_SWIGLU, 2)


# ---- the tensor-core attention kernel (bfloat16, head sizes 64 and 128) ----

def _attn_mma_case(cuda, n_heads, n_kv, hd, starts, news, window, decode, n_splits=1, spike=None):
    from camelid_b200.csrc import ops
    dt = torch.bfloat16
    totals = [s + n for s, n in zip(starts, news)]
    k_pages, v_pages, table, ks, vs = _paged(totals, n_kv, hd, dt, cuda)
    g = torch.Generator().manual_seed(1)
    n_rows = sum(news)
    q = torch.randn(n_rows, n_heads, hd, generator=g).to(dt)
    row0 = [sum(news[:i]) for i in range(len(news))]
    if spike is not None:
        seq, key = spike
        r = row0[seq] + news[seq] - 1
        ks[seq][key] *= 0
        ks[seq][key, :, 0] = 8.0
        q[r, :, 0] = 8.0 * math.sqrt(hd) / 4
        k_pages[int(table[seq, key // 64]), :, key % 64] = ks[seq][key].to(cuda)
    rows, hpc, chunks = ops.attn_mma_tiling(n_heads, n_kv, decode)
    tile_seq, tile_q0 = [], []
    for i, n in enumerate(news):
        for q0 in range(0, n, rows):
            tile_seq.append(i)
            tile_q0.append(q0)
    out = torch.full((n_rows, n_heads * hd), float("nan"), dtype=dt, device=cuda)
    partial = torch.empty(max(1, ops.attn_partial_floats(n_rows, n_heads, hd, n_splits)), device=cuda)
    ops.attn_paged_mma(q.view(n_rows, -1).to(cuda), out, k_pages, v_pages, table, _i32(tile_seq, cuda),
                       _i32(tile_q0, cuda), len(tile_seq), _i32(row0, cuda), _i32(starts, cuda), _i32(news, cuda),
                       n_rows, n_heads, n_kv, hd, rows, hpc, chunks, n_splits, window or 0, 1 / math.sqrt(hd), partial)
    out = out.cpu().view(n_rows, n_heads, hd)
    for i, (s, n) in enumerate(zip(starts, news)):
        qfull = torch.zeros(s + n, n_heads, hd, dtype=torch.float64)
        qfull[s:] = q[row0[i]:row0[i] + n].double()
        ref = pl.attention(qfull, ks[i].double(), vs[i].double(), window)[s:]
        e = rel_err(out[row0[i]:row0[i] + n], ref)
        assert e <= 2 ** -6, f"sequence {i}: {e}"


@pytest.mark.parametrize("n_heads,n_kv,hd", [(4, 1, 64), (32, 8, 64), (6, 2, 128), (5, 5, 64), (34, 1, 128), (12, 2, 64)])
def test_attention_mma_rows_of_several_tokens(cuda, n_heads, n_kv, hd):
    _attn_mma_case(cuda, n_heads, n_kv, hd, starts=[0, 0, 0, 64], news=[1, 70, 129, 33], window=None, decode=False,
                   spike=(2, 3))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n_splits", [1, 2, 5, 16])
def test_attention_mma_decode_splits(cuda, hd, n_splits):
    _attn_mma_case(cuda, 8, 2, hd, starts=[0, 31, 32, 63, 64, 700], news=[1] * 6, window=None, decode=True,
                   n_splits=n_splits, spike=(5, 130))


@pytest.mark.parametrize("edge", [0, 1], ids=["first key outside", "first key inside"])
@pytest.mark.parametrize("window", [1, 32, 70, 199])
def test_attention_mma_window_edges(cuda, window, edge):
    _attn_mma_case(cuda, 4, 2, 64, starts=[0, 190], news=[150, 10], window=window, decode=False,
                   spike=(1, 199 - window + edge))
    _attn_mma_case(cuda, 4, 2, 64, starts=[199, 80], news=[1, 1], window=window, decode=True, n_splits=3,
                   spike=(0, 199 - window + edge))


# ---- the tcgen05 prefill attention kernel ----

def _attn_tc_case(cuda, n_heads, n_kv, hd, starts, news, window, spike=None):
    from camelid_b200.csrc import ops
    dt = torch.bfloat16
    totals = [s + n for s, n in zip(starts, news)]
    k_pages, v_pages, table, ks, vs = _paged(totals, n_kv, hd, dt, cuda)
    g = torch.Generator().manual_seed(1)
    n_rows = sum(news)
    q = torch.randn(n_rows, n_heads, hd, generator=g).to(dt)
    row0 = [sum(news[:i]) for i in range(len(news))]
    if spike is not None:
        seq, key = spike
        r = row0[seq] + news[seq] - 1
        ks[seq][key] *= 0
        ks[seq][key, :, 0] = 8.0
        q[r, :, 0] = 8.0 * math.sqrt(hd) / 4
        k_pages[int(table[seq, key // 64]), :, key % 64] = ks[seq][key].to(cuda)
    rows, hpc, chunks = ops.attn_tc_tiling(n_heads, n_kv)
    tile_seq, tile_q0 = [], []
    for i, n in enumerate(news):
        for q0 in range(0, n, rows):
            tile_seq.append(i)
            tile_q0.append(q0)
    out = torch.full((n_rows, n_heads * hd), float("nan"), dtype=dt, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    ops.attn_prefill_tc(q.view(n_rows, -1).to(cuda), out, k_pages, v_pages, table, _i32(tile_seq, cuda),
                        _i32(tile_q0, cuda), len(tile_seq), _i32(row0, cuda), _i32(starts, cuda), _i32(news, cuda),
                        n_heads, n_kv, hd, rows, hpc, chunks, window or 0, 1 / math.sqrt(hd), err)
    assert int(err) == 0
    out = out.cpu().view(n_rows, n_heads, hd)
    for i, (s, n) in enumerate(zip(starts, news)):
        qfull = torch.zeros(s + n, n_heads, hd, dtype=torch.float64)
        qfull[s:] = q[row0[i]:row0[i] + n].double()
        ref = pl.attention(qfull, ks[i].double(), vs[i].double(), window)[s:]
        e = rel_err(out[row0[i]:row0[i] + n], ref)
        assert e <= 2 ** -6, f"sequence {i}: {e}"


@pytest.mark.parametrize("n_heads,n_kv,hd", [(4, 1, 64), (32, 8, 64), (6, 2, 128), (5, 5, 64), (34, 1, 128), (12, 2, 64)])
def test_attention_tc_prefill_shapes(cuda, n_heads, n_kv, hd):
    _attn_tc_case(cuda, n_heads, n_kv, hd, starts=[0, 0, 0, 64], news=[1, 70, 300, 33], spike=(2, 3), window=None)


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_tc_continues_from_cache(cuda, hd):
    _attn_tc_case(cuda, 8, 2, hd, starts=[64, 300, 5, 0], news=[3, 200, 64, 129], spike=(1, 7), window=None)


@pytest.mark.parametrize("edge", [0, 1], ids=["first key outside", "first key inside"])
@pytest.mark.parametrize("window", [1, 32, 70, 199])
def test_attention_tc_window_edges(cuda, window, edge):
    _attn_tc_case(cuda, 4, 2, 64, starts=[0, 190], news=[150, 10], window=window, spike=(1, 199 - window + edge))


def _attn_fused_case(cuda, n_heads, n_kv, hd, rot, starts, window, n_splits, gsplits, write_kv=True, spike=None,
                     n_pages=64):
    """Decode attention in one launch from the partial sums of the q/k/v product: against the
    plain rotary encoding and attention of the whole sequences, and the cache rows it writes."""
    from camelid_b200.csrc import ops
    from camelid_b200.parts.position import rotary_frequencies
    dt = torch.bfloat16
    n = len(starts)
    totals = [s + 1 for s in starts]
    k_pages, v_pages, table, ks, vs = _paged(totals, n_kv, hd, dt, cuda, n_pages=n_pages, seed=4)
    freqs = rotary_frequencies(rot, 10000.0, None) if rot else np.zeros(0, dtype=np.float32)
    g = torch.Generator().manual_seed(7)
    width = (n_heads + 2 * n_kv) * hd
    part = torch.randn(gsplits, n, width, generator=g) / math.sqrt(gsplits)
    pos = torch.tensor(starts)
    if spike is not None:
        # One cached key gets a score that stands out for every head of its sequence: the key is
        # 8 in its last dimension and nothing else, and the query is made so that, after the
        # kernel's rotation at its position, it is large in that dimension (the query before
        # the rotation is the wanted one turned back). A kernel that drops that key, or counts
        # it when the window excludes it, is off by far more than the tolerance.
        seq, key = spike
        ks[seq][key] *= 0
        ks[seq][key, :, hd - 1] = 8.0
        k_pages[int(table[seq, key // 64]), :, key % 64] = ks[seq][key].to(cuda)
        want_q = torch.randn(1, n_heads, hd, generator=g, dtype=torch.float64)
        want_q[..., hd - 1] = 8.0 * math.sqrt(hd) / 4
        before = pl.rope(want_q, -pos[seq:seq + 1], freqs) if rot else want_q
        rest = part[1:, seq, :n_heads * hd].sum(0) if gsplits > 1 else 0.0
        part[0, seq, :n_heads * hd] = before.reshape(-1).float() - rest
    total = torch.zeros(n, width)
    for s in range(gsplits):
        total = total + part[s]                       # the kernel's order of adding
    qkv = total.to(dt)
    q = qkv[:, :n_heads * hd].double().view(n, n_heads, hd)
    k = qkv[:, n_heads * hd:(n_heads + n_kv) * hd].double().view(n, n_kv, hd)
    v = qkv[:, (n_heads + n_kv) * hd:].view(n, n_kv, hd)
    q_rot = (pl.rope(q, pos, freqs) if rot else q).to(dt)
    k_rot = (pl.rope(k, pos, freqs) if rot else k).to(dt)
    tab = table.cpu()
    slots = [(int(tab[i, s // 64]), s % 64) for i, s in enumerate(starts)]
    if write_kv:                                      # the row's own place holds something else until the kernel writes it
        for page, off in slots:
            k_pages[page, :, off] = float("nan")
            v_pages[page, :, off] = float("nan")
    else:                                             # a borrowed cache already holds the row's key and value
        for i, (page, off) in enumerate(slots):
            k_pages[page, :, off] = k_rot[i].to(cuda)
            v_pages[page, :, off] = v[i].to(cuda)
    before_k = k_pages.clone()
    out = torch.full((n, n_heads * hd), float("nan"), dtype=dt, device=cuda)
    ops.attn_decode_fused(part.to(cuda), out, _i32(starts, cuda), _i32(list(range(n)), cuda), table, k_pages, v_pages,
                          torch.from_numpy(freqs).to(cuda), rot, n_heads, n_kv, hd, write_kv, window or 0,
                          1 / math.sqrt(hd), n_splits)
    out = out.cpu().view(n, n_heads, hd)
    for i, s in enumerate(starts):
        page, off = slots[i]
        if write_kv:
            assert rel_err(k_pages[page, :, off].cpu(), k_rot[i].double()) <= 2 ** -8
            assert torch.equal(v_pages[page, :, off].cpu(), v[i])
        kfull = torch.cat([ks[i][:s].double(), k_rot[i].double()[None]], dim=0)
        vfull = torch.cat([vs[i][:s].double(), v[i].double()[None]], dim=0)
        qfull = torch.zeros(s + 1, n_heads, hd, dtype=torch.float64)
        qfull[s] = q_rot[i].double()
        ref = pl.attention(qfull, kfull, vfull, window)[s:]
        e = rel_err(out[i:i + 1], ref)
        assert e <= 2 ** -6, f"sequence {i} at position {s}: {e}"
    changed = (before_k != k_pages) & ~(torch.isnan(before_k) & torch.isnan(k_pages))
    assert int(changed.any(dim=-1).sum()) <= (n * n_kv if write_kv else 0)     # nothing else was written


@pytest.mark.parametrize("n_splits", [1, 2, 5, 8])
@pytest.mark.parametrize("n_heads,n_kv,hd,rot", [(8, 2, 64, 64), (6, 2, 128, 64), (5, 5, 64, 32), (16, 1, 64, 0)])
def test_attention_decode_fused(cuda, n_heads, n_kv, hd, rot, n_splits):
    _attn_fused_case(cuda, n_heads, n_kv, hd, rot, starts=[0, 31, 32, 63, 64, 700], window=None, n_splits=n_splits,
                     gsplits=3, spike=(5, 130))


@pytest.mark.parametrize("edge", ["first key inside", "first key outside"])
@pytest.mark.parametrize("window", [1, 32, 70, 199])
def test_attention_decode_fused_window_and_borrowed_cache(cuda, window, edge):
    """The query at position 199 with a window of w sees keys 200 - w .. 199: the outstanding key
    sits once on the first key inside the window (it must count) and once on the first key
    outside (it must not)."""
    key = 200 - window if edge == "first key inside" else 199 - window
    if key == 199:              # a window of 1 sees only the new key, which the kernel makes itself
        key = None
    _attn_fused_case(cuda, 4, 2, 64, 64, starts=[199, 80, 0], window=window, n_splits=3, gsplits=9,
                     spike=None if key is None else (0, key))
    _attn_fused_case(cuda, 4, 2, 64, 64, starts=[199, 80, 0], window=window, n_splits=4, gsplits=1, write_kv=False,
                     spike=None if key is None else (0, key))
    _attn_fused_case(cuda, 8, 2, 128, 128, starts=[300, 5], window=None, n_splits=2, gsplits=2, write_kv=False)


@pytest.mark.parametrize("n_splits,key", [(1, 2100), (1, 8999), (3, 130), (3, 5003), (8, 2100), (8, 8999)])
def test_attention_decode_fused_long_context(cuda, n_splits, key):
    """Thousands of cached keys: a warp walks more tiles than the 32 page numbers it keeps in
    registers, and one outstanding key, near the start, past a warp's first 32 pages, in the
    middle or at the very end of the range, must be found."""
    _attn_fused_case(cuda, 8, 2, 64, 64, starts=[9000, 4100, 64], window=None, n_splits=n_splits, gsplits=2,
                     spike=(0, key), n_pages=256)


# The split of the keys over a cluster: positions at the edges of rounds (32), blocks (128), pages (64) and windows; one, two, three (a
# masked head) and six (two heads' chunks) query heads a key head; every term of the score; a window of fewer rounds than warps.
@pytest.mark.parametrize("D,Dv,H,G,window,chunk,keep,extras", [
    (128, 128, 16, 4, 0, 0, 0, "rel"), (128, 128, 4, 1, 1024, 0, 64, "sink gate"), (64, 128, 3, 1, 70, 0, 5, "cap"),
    (128, 64, 2, 1, 0, 200, 0, "penalty head_gate"), (64, 64, 12, 2, 300, 0, 0, "penalty gate"), (128, 128, 2, 2, 33, 0, 0, "sink"),
    (64, 64, 8, 4, 20, 0, 0, "rel sink")])
def test_window_attention_split_over_a_cluster(cuda, D, Dv, H, G, window, chunk, keep, extras):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(D + Dv + H + window)
    positions = [0, 1, 31, 32, 63, 64, 127, 128, 199, 200, 299, 300, 1055, 1088, 1301]
    n, width = len(positions), max(positions) // 64 + 1
    pages = torch.randperm(n * width + 1, generator=gen)[1:].view(n, width).to(torch.int32)
    k, v = (torch.randn(n * width + 1, G, 64, d, generator=gen).bfloat16() for d in (D, Dv))
    q = torch.randn(n, H * D, generator=gen).bfloat16()
    scale, cap = 2.0 * D ** -0.5, 3.0 if "cap" in extras else 0.0
    r1, r2 = (torch.rand(H, generator=gen) * 2, torch.rand(H, generator=gen)) if "penalty" in extras else (None, None)
    sink = torch.randn(H, generator=gen) if "sink" in extras else None
    rel = torch.randn(H, 90, generator=gen) if "rel" in extras else None
    per_head = "head_gate" in extras
    gate = torch.randn(n, 3 + (H if per_head else H * Dv), generator=gen) if "gate" in extras else None
    ref = torch.empty(n, H, Dv, dtype=torch.float64)
    for s, i in enumerate(positions):
        j = torch.arange(i + 1)
        see = (j // chunk == i // chunk) if chunk else ((i - j < window) | (j < keep)) if window else (j >= 0)
        j = j[see]
        at = pages[s, j // 64].long(), j % 64
        for h in range(H):
            sc = k[at[0], h // (H // G), at[1]].double() @ q[s, h * D:(h + 1) * D].double() * scale
            sc = cap * torch.tanh(sc / cap) if cap else sc
            if r1 is not None:
                sc = sc - r1[h].double() * torch.log1p(r2[h].double() * (i - j))
            if rel is not None:
                sc = sc + rel[h, (i - j).clamp(max=89)].double()
            z = torch.logsumexp(torch.cat([sc, sink[h:h + 1].double()]) if sink is not None else sc, 0)
            ref[s, h] = 0.5 * torch.exp(sc - z) @ v[at[0], h // (H // G), at[1]].double()
    if gate is not None:
        ref = ref * torch.sigmoid(gate[:, 3:].double()).view(n, H, -1)
    d = lambda t: None if t is None else t.to(cuda)                         # noqa: E731
    out = torch.full((n, H * Dv + 8), 7.0, dtype=torch.bfloat16, device=cuda)
    row = torch.arange(n, dtype=torch.int32, device=cuda)
    args = (d(q), d(k), d(v), d(pages), row, torch.tensor(positions, dtype=torch.int32, device=cuda), d(r1), d(r2), d(gate), 3)
    more = (H, G, D, Dv, window, scale, chunk, d(sink), per_head, cap, None, keep, False, d(rel), 0.5)
    ops.window_attention(*args, out[:, :H * Dv], *more, single=True)
    for s in (0, 9, 14):                             # a row alone (fewer heads a block), and with its keys awaited: the same bits
        one = torch.empty(1, H * Dv, dtype=torch.bfloat16, device=cuda)
        ops.window_attention(d(q)[s:s + 1], *args[1:4], *(a[s:s + 1] for a in args[4:6]), *args[6:8], None if gate is None else args[8][s:s + 1], 3,
                             one, *more)
        assert torch.equal(one[0], out[s, :H * Dv])
    got = out[:, :H * Dv].cpu().double().view(n, H, Dv)
    # half a unit of the last of the output's 8 bits; and the scores' float error (D products of a size of up to 30, 128 * 30 * 2^-24)
    # as a relative error of the weights, for values of up to 5
    assert bool(((got - ref).abs() <= ref.abs() * 2.0 ** -8 + 5 * 128 * 30 * 2.0 ** -24).all())
    assert bool((out[:, H * Dv:] == 7.0).all())


# Chunks of 64 tokens: whole, ragged and single-token ones, several sequences, states that continue and states that start (over stale
# contents); tiles of 64 values and 32 channels, whole and not (the memory's extra value in a tile of its own and inside one).
@pytest.mark.parametrize("H,D,Dv", [(3, 128, 128), (2, 24, 40), (1, 4, 4), (2, 64, 68), (1, 256, 60)])
def test_retention_and_matrix_memory_by_chunks(cuda, H, D, Dv):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(H + D + Dv)
    news, starts, slots = [64, 1, 200, 33, 128], [0, 7, 0, 50, 64], [3, 0, 5, 1, 2]
    n, B = sum(news), 6
    row0 = [sum(news[:i]) for i in range(len(news))]
    tiles = [(s, q) for s, m in enumerate(news) for q in range(0, m, 64)]
    t = [_i32([x[i] for x in tiles], cuda) for i in (0, 1)]
    seq = [_i32(x, cuda) for x in (row0, news, starts, slots)]
    q, k = (torch.randn(n, H * D, generator=gen) for _ in range(2))
    v = torch.randn(n, H * Dv, generator=gen)
    gates = torch.randn(n, 2 * H, generator=gen) * 4.0
    pad = -(2 * H * D + H * Dv + 2 * H) % 4
    proj = torch.cat([q, k, v, gates, torch.zeros(n, pad)], 1).to(cuda)
    cols = (0, H * D, 2 * H * D, 2 * H * D + H * Dv, 2 * H * D + H * Dv + H)
    scratch = lambda values: [torch.full(s, float("nan"), device=cuda) for s in                    # noqa: E731
                              ((len(tiles), H, 64, 64), (len(tiles), H, 4, 64), (len(tiles), H, values, D))]
    q64, k64, v64 = (x.double().view(n, H, -1) for x in (q, k, v))
    # ---- retention: decays near one, ordinary, and so small that a chunk's product is zero in 32 bits
    decay = torch.tensor([0.999, 0.6, 1e-4][:H])
    S0 = torch.randn(B, H, Dv, D, generator=gen)
    state, out = S0.to(cuda), torch.full((n, H * Dv), float("nan"), device=cuda)
    ops.retention_chunks(proj, cols[:3], decay.to(cuda), *t, len(tiles), *seq, state, *scratch(Dv), out, len(news), H, D, Dv)
    ref, after = torch.empty(n, H, Dv, dtype=torch.float64), S0.double()
    for s, m in enumerate(news):
        S = S0[slots[s]].double() if starts[s] else torch.zeros(H, Dv, D, dtype=torch.float64)
        for i in range(row0[s], row0[s] + m):
            S = decay.double().view(H, 1, 1) * S + v64[i].unsqueeze(2) * k64[i].unsqueeze(1)
            ref[i] = (S @ q64[i].unsqueeze(2)).squeeze(2)
        after[slots[s]] = S
    # sums of 64 products of D terms: each term's share of the largest output is rounded a few times, 2^-24 of it each, so that
    # sqrt(64 D) 2^-24 = 8e-6 (D = 256) of the largest is far out
    assert rel_err(out.cpu().double().view(n, H, Dv), ref) < 1e-5 and rel_err(state.cpu().double(), after) < 1e-5
    # ---- matrix memory: forget gates that stay open and shut, input gates that overtake the maximum
    bi, bf, cap, scale = torch.randn(H, generator=gen), torch.randn(H, generator=gen) + 3.0, 15.0, D ** -0.5
    M0, m0 = torch.randn(B, H, Dv + 1, D, generator=gen), torch.randn(B, H, 1, generator=gen).expand(B, H, Dv + 1).contiguous()
    state, state_m, out = M0.to(cuda), m0.to(cuda), torch.full((n, H, Dv + 2), float("nan"), device=cuda)
    ops.memory_chunks(proj, cols, bi.to(cuda), bf.to(cuda), cap, scale, *t, len(tiles), *seq, state, state_m, *scratch(Dv + 1), out, len(news), H,
                      D, Dv)
    gi = cap * torch.tanh((gates[:, :H].double() + bi.double()) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((gates[:, H:].double() + bf.double()) / cap))
    ref, after, after_m = torch.empty(n, H, Dv + 2, dtype=torch.float64), M0.double(), m0.double()
    one = torch.ones(H, 1, dtype=torch.float64)
    for s, m in enumerate(news):
        S = M0[slots[s]].double() if starts[s] else torch.zeros(H, Dv + 1, D, dtype=torch.float64)
        top = m0[slots[s], :, 0].double() if starts[s] else torch.zeros(H, dtype=torch.float64)
        for i in range(row0[s], row0[s] + m):
            new = torch.maximum(gf[i] + top, gi[i])
            a, b, top = torch.exp(gf[i] + top - new), torch.exp(gi[i] - new), new
            S = a.view(H, 1, 1) * S + b.view(H, 1, 1) * torch.cat([v64[i], one], 1).unsqueeze(2) * k64[i].unsqueeze(1)
            ref[i, :, :Dv + 1] = (S @ q64[i].unsqueeze(2)).squeeze(2) * scale
            ref[i, :, Dv + 1] = top
        after[slots[s]], after_m[slots[s]] = S, top.unsqueeze(1).expand(H, Dv + 1)
    got = out.cpu().double()
    assert rel_err(got[..., :Dv + 1], ref[..., :Dv + 1]) < 1e-5 and float((got[..., Dv + 1] - ref[..., Dv + 1]).abs().max()) < 1e-5
    assert rel_err(state.cpu().double(), after) < 1e-5 and float((state_m.cpu().double() - after_m).abs().max()) < 1e-5


# Float products of many rows on exact bfloat16 pieces: edges of tiles (128) and steps (64 k's), the last step's k's and columns missing; numbers whose
# pieces differ much in size; operands that have no pieces (infinite, not a number, rounding to infinity).
@pytest.mark.parametrize("M,N,K", [(65, 1, 4), (128, 127, 60), (129, 129, 64), (66, 130, 68), (257, 64, 192), (70, 256, 1028)])
def test_float_products_of_many_rows(cuda, M, N, K):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=gen) * torch.exp(3 * torch.randn(M, K, generator=gen))
    w = torch.randn(N, K, generator=gen) * torch.exp2(torch.randint(-12, 12, (N, K), generator=gen).float())
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    c = torch.full((M, N + 3), 7.0, device=cuda)
    ops.gemm_tn_simt(a.to(cuda), w.to(cuda), c[:, :N], ops.EPI_STORE_F32)
    # each of a step's four cuts is at most 2^-23 of what the step sums, each step's addition 2^-24 of the sum
    bound = (8 + K / 64) * 2.0 ** -24 * size
    assert bool(((c[:, :N].cpu().double() - ref).abs() <= bound).all()) and bool((c[:, N:] == 7.0).all())
    a[0, 1], a[1, 0], a[2, 2], a[3, 3] = float("inf"), float("nan"), 3.4e38, -float("inf")
    a[3, 0] = float("inf")
    w[0, :] = 1e-3
    w[N // 2, 1] = 0.0
    ref = a.double() @ w.double().T
    ops.gemm_tn_simt(a.to(cuda), w.to(cuda), c[:, :N], ops.EPI_STORE_F32)
    got = c[:, :N].cpu().double()
    assert torch.equal(torch.isnan(got[[0, 1, 3]]), torch.isnan(ref[[0, 1, 3]])) and torch.equal(torch.isposinf(got[0]), torch.isposinf(ref[0]))
    assert bool(torch.isfinite(got[4:]).all())
    held = ref[2].abs() < 3e38
    assert bool(((got[2] - ref[2]).abs() <= 1e-5 * (a[2].double().abs() @ w.double().abs().T))[held].all()) and not bool(torch.isfinite(got[2][ref[2].abs() > 3.5e38]).any())


# Chunks of 32 tokens: whole, ragged and of one token, several sequences, states that continue and that start over stale contents; q and k heads
# shared; a decay per channel (some that vanish at once, some near one) and per head; columns and channels that are not there.
@pytest.mark.parametrize("H,G,D,Dv,per_head", [(4, 2, 128, 128, False), (2, 2, 68, 4, False), (3, 1, 100, 20, True), (1, 1, 128, 36, True)])
def test_gated_delta_rule_by_chunks(cuda, H, G, D, Dv, per_head):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(H + D + Dv)
    news, starts, slots = [32, 1, 200, 33, 95], [0, 7, 0, 50, 64], [3, 0, 5, 1, 2]
    n, B = sum(news), 6
    row0 = [sum(news[:i]) for i in range(len(news))]
    tiles = [(s, q) for s, m in enumerate(news) for q in range(0, m, 32)]
    t = [_i32([x[i] for x in tiles], cuda) for i in (0, 1)]
    seq = [_i32(x, cuda) for x in (row0, news, starts, slots)]
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)                       # noqa: E731
    q, k = unit(torch.randn(n, G, D, generator=gen)), unit(torch.randn(n, G, D, generator=gen) + 0.5)     # (keys of one direction: large A)
    v, beta_in = torch.randn(n, H, Dv, generator=gen), torch.randn(n, 3 + H, generator=gen) * 2
    decay = torch.exp(-torch.exp(2.0 * torch.randn(n, H, 1 if per_head else D, generator=gen) - 3.0))
    decay[5, :, 0], decay[60:, 0, -1] = 0.0, 1e-30
    S0 = torch.randn(B, H, Dv, D, generator=gen)
    qkv = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)], 1).to(cuda)
    state, out = S0.to(cuda), torch.full((n, H * Dv), float("nan"), device=cuda)
    scratch = torch.full((len(tiles), H, ops.gated_chunk_floats(D, Dv)), float("nan"), device=cuda)
    ops.gated_chunks(qkv, beta_in.to(cuda), 3, decay.reshape(n, -1).to(cuda), *t, len(tiles), *seq, scratch, state, out, len(news), H, G, D, Dv)
    q64, k64 = (x.double().repeat_interleave(H // G, 1) for x in (q, k))
    beta, g64, v64 = torch.sigmoid(beta_in[:, 3:].double()), decay.double(), v.double()
    ref, after = torch.empty(n, H, Dv, dtype=torch.float64), S0.double()
    for s, m in enumerate(news):
        S = S0[slots[s]].double() if starts[s] else torch.zeros(H, Dv, D, dtype=torch.float64)
        for i in range(row0[s], row0[s] + m):
            S = S * g64[i].unsqueeze(1)
            z = beta[i].unsqueeze(1) * (v64[i] - (S @ k64[i].unsqueeze(2)).squeeze(2))
            S = S + z.unsqueeze(2) * k64[i].unsqueeze(1)
            ref[i] = (S @ q64[i].unsqueeze(2)).squeeze(2)
        after[slots[s]] = S
    # unit keys: sums of D products of 2^-24 each, gone through up to 32 tokens' corrections: sqrt(32 D) 2^-24 = 4e-6 of the largest
    assert rel_err(out.cpu().double().view(n, H, Dv), ref) < 1e-5 and rel_err(state.cpu().double(), after) < 1e-5


# Shares of 1, 64 (as many as have their weights made at once), 65 and 130 key ranges, some of them empty; channels beyond a block's 128 and short of it.
@pytest.mark.parametrize("splits,C", [(1, 32), (64, 160), (65, 128), (130, 512)])
def test_latent_shares_merged(cuda, splits, C):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(splits + C)
    H, R, n, per = 3, 16, 2, 1
    lens = [64 * splits - 5, max(1, 64 * splits // 3)]
    D, width = C + R, splits
    k = torch.randn(n * width + 1, 1, 64, D, generator=gen).bfloat16()
    q = torch.randn(n, H * D, generator=gen).bfloat16()
    sink, gate, scale = torch.randn(H, generator=gen), torch.randn(n, H, generator=gen), 2.0 * D ** -0.5
    table = torch.randperm(n * width, generator=gen).view(n, width).to(torch.int32)
    ref = torch.empty(n, H, C, dtype=torch.float64)
    for s, m in enumerate(lens):
        j = torch.arange(m)
        rows = k[table[s, j // 64].long(), 0, j % 64].double()
        for h in range(H):
            sc = rows @ q[s, h * D:(h + 1) * D].double() * scale
            z = torch.logsumexp(torch.cat([sc, sink[h:h + 1].double()]), 0)
            ref[s, h] = torch.sigmoid(gate[s, h].double()) * (torch.exp(sc - z) @ rows[:, :C])
    i32 = lambda x: _i32(x, cuda)                                           # noqa: E731
    partial = torch.full((splits, n, H, C + 2), float("nan"), device=cuda)
    out = torch.empty(n, H * C, dtype=torch.bfloat16, device=cuda)
    ops.latent_prompt(q.to(cuda), k.to(cuda), out, table.to(cuda), i32([0, 1]), i32([0, 0]), n, i32([0, 1]), i32([m - 1 for m in lens]), i32([1, 1]),
                      H, C, R, scale, sink.to(cuda), gate.to(cuda), 0, partial, per)
    # weights and output rounded to 8 bits: 2^-8 of the weighted sum of the values' sizes (up to 4) and of the output
    assert float((out.cpu().double().view(n, H, C) - ref).abs().max()) < 2.0 ** -8 * (4.0 + float(ref.abs().max()))


# The rows from which the preparing kernel gives a row fewer threads.
def test_latent_rows_prepared_at_the_line(cuda):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(9)
    n, H, D, R, C = 129, 3, 24, 16, 96
    proj = torch.randn(n, H * (D + R) + C + R, generator=gen).to(cuda)
    w, freq = torch.rand(C, generator=gen).to(cuda), torch.rand(R // 2, generator=gen).to(cuda)
    seq, pos, table = _i32([0] * n, cuda), _i32(range(n), cuda), _i32([[0, 1, 2]], cuda)
    got = []
    for rows in (128, 129):
        q, full, pages = (torch.zeros(s, device=cuda) for s in ((rows, H * D), (rows, H * (C + R)), (3, 1, 64, C + R)))
        ops.latent_prepare(proj[:rows], w, 1e-6, freq, True, 1.0, seq[:rows], pos[:rows], table, q, full, pages, H, D, R, C, None, None, None)
        got.append((q[:128], full[:128], pages.view(192, -1)[:128]))
    for few, many in zip(*got):
        assert float((few - many).abs().max()) <= 4e-6 * float(many.abs().max())      # (the sums of squares are added in another order)
    assert torch.equal(got[0][0], got[1][0])


# The convolution of many rows, a warp's eight rows at a time: sequences that end inside a warp's rows, that begin a prompt, continue one or are
# shorter than the taps; heads of one piece, of a lane short of 128 and of 128 channels.
@pytest.mark.parametrize("G,H,D,Dv", [(1, 2, 4, 128), (2, 4, 128, 20), (3, 3, 124, 8)])
def test_convolution_of_many_rows(cuda, G, H, D, Dv):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(G + D + Dv)
    news, starts, slots = [1, 30, 2, 45, 3], [0, 0, 1, 9, 2], [2, 0, 4, 1, 3]
    n, C = sum(news), 2 * G * D + H * Dv
    x, w, state = torch.randn(n, C + 4, generator=gen), torch.randn(C, 4, generator=gen), torch.randn(5, 3, C, generator=gen)
    dec, al, dt = torch.randn(n, H * D, generator=gen), torch.randn(H, generator=gen), torch.randn(H * D, generator=gen)
    row0 = [sum(news[:i]) for i in range(len(news))]
    seq = [i for i, m in enumerate(news) for _ in range(m)]
    pos = [s + j for s, m in zip(starts, news) for j in range(m)]
    out, decays = torch.full((n, C), float("nan"), device=cuda), torch.full((n, H * D), float("nan"), device=cuda)
    st = state.to(cuda)
    ops.conv_unit(x.to(cuda), w.to(cuda), st, _i32(seq, cuda), _i32(pos, cuda), _i32(row0, cuda), _i32(slots, cuda), out, G, H, D, Dv, 0.3,
                  update_state=False, decay=(dec.to(cuda), al.to(cuda), dt.to(cuda), decays))
    ref = torch.empty(n, C, dtype=torch.float64)
    for i in range(n):
        s = seq[i]
        acc = torch.zeros(C, dtype=torch.float64)
        for back in range(4):
            if back <= pos[i]:
                v = x[i - back, :C] if back <= i - row0[s] else state[slots[s], 3 + (i - row0[s]) - back]
                acc += w[:, 3 - back].double() * v.double()
        ref[i] = acc * torch.sigmoid(acc)
    qk = ref[:, :2 * G * D].view(n, 2 * G, D)
    qk /= torch.sqrt((qk * qk).sum(-1, keepdim=True) + 1e-6)
    qk[:, :G] *= 0.3
    assert float((out.cpu().double() - ref).abs().max()) < 2e-6 * max(1.0, float(ref.abs().max()))      # four terms, SiLU and the norm: 2^-24 each, a few times
    want = torch.exp(-torch.exp(al.double()).view(1, H, 1) * torch.nn.functional.softplus(dec.double() + dt.double()).view(n, H, D)).view(n, -1)
    assert float((decays.cpu().double() - want).abs().max()) < 4e-6 and torch.equal(st.cpu(), state)


def _recurrence(kind, x, gates, decays, H, D, news, starts, states, by_chunks, tiles_from=1, decay=0.9, **more):
    """Outputs [rows, .] of one of the recurrences by its scan or its chunked form (tiles of the sequences with ``tiles_from`` rows and more); ``states``
    move on. Rows: k, q, v (H x D each), then two gates a head."""
    from camelid_b200.csrc import ops
    n, cuda = x.shape[0], x.device
    row0 = [sum(news[:i]) for i in range(len(news))]
    size = 32 if kind == "gated" else 64
    tiles = [(s, q) for s, m in enumerate(news) for q in range(0, m if m >= tiles_from else 0, size)]
    tiles = (_i32([t[0] for t in tiles], cuda), _i32([t[1] for t in tiles], cuda), len(tiles))
    seq = [_i32(t, cuda) for t in (row0, news, starts, range(len(news)))]
    cols, vec, scratch = (0, H * D, 2 * H * D, 3 * H * D, 3 * H * D + H), torch.full((H,), decay, device=cuda), []
    if by_chunks and kind != "gated":
        scratch = [torch.full(s, float("nan"), device=cuda) for s in ((tiles[2], H, 64, 64), (tiles[2], H, 3 if kind == "state space" else 4, 64),
                                                                      (tiles[2], *states[0].shape[1:]))]
    out = torch.full((n, H, D + 2 if kind == "matrix memory" else D), float("nan"), device=cuda)
    flat = out.view(n, -1)
    dims, B = (H, D, D), len(news)
    if kind == "retention":
        args = (x, cols[:3], vec)
        if by_chunks:
            ops.retention_chunks(*args, *tiles, *seq, states[0], *scratch, flat, B, *dims, **more)
        else:
            ops.retention_scan(*args, states[0], *seq, flat, B, *dims, **more)
    elif kind == "matrix memory":
        args = (x, cols, vec, vec, 15.0, 0.1)
        if by_chunks:
            ops.memory_chunks(*args, *tiles, *seq, *states, *scratch, out, B, *dims, **more)
        else:
            ops.memory_scan(*args, *states, *seq, out, B, *dims, **more)
    elif kind == "state space":
        g, order = torch.cat([gates, torch.exp(-torch.exp(vec) * gates)], 1), (cols[2], cols[1], cols[0])
        if by_chunks:
            ops.ssm_chunks(x, order, g, vec, vec, *tiles, *seq, states[0], *scratch, flat, B, H, *dims, **more)
        else:
            ops.ssm_scan(x, order, g, vec, states[0], *seq, flat, B, H, *dims, **more)
    elif by_chunks:
        chunks = torch.full((tiles[2], H, ops.gated_chunk_floats(D, D)), float("nan"), device=cuda)
        ops.gated_chunks(x, gates, 0, decays, *tiles, *seq, chunks, states[0], flat, B, H, *dims, **more)
    else:
        zero = torch.zeros(H * D, device=cuda)
        ops.delta_scan(x, gates, 0, decays, zero[:H], zero, states[0], *seq, flat, B, H, *dims, decay_ready=True, **more)
    return flat


def _recurrence_inputs(cuda, kind, n, H, D, B, gen):
    """Rows (unit q and k), gates, decays, and states of B sequences."""
    x = torch.randn(n, 3 * H * D + 2 * H, generator=gen)
    x[:, :2 * H * D] = torch.nn.functional.normalize(x[:, :2 * H * D].reshape(n, 2 * H, D), dim=-1).reshape(n, -1)
    gates, decays = torch.rand(n, H, generator=gen), 0.5 + 0.5 * torch.rand(n, H * D, generator=gen)
    extra = 1 if kind == "matrix memory" else 0
    states = [torch.randn(B, H, D + extra, D, generator=gen), torch.randn(B, H, 1, generator=gen).expand(B, H, D + 1).contiguous()]
    return x.to(cuda), gates.to(cuda), decays.to(cuda), [s.to(cuda) for s in states[:1 + extra]]


RECURRENCES = ["retention", "matrix memory", "state space", "gated"]


# A value that is not finite: by chunks as in the scan, the tokens before it are untouched, itself and the later ones are not finite.
# Places inside a chunk of 64 (32), of a group of eight (four) of its tokens, and at their edges.
@pytest.mark.parametrize("at", [21, 24, 70, 95])
@pytest.mark.parametrize("kind", RECURRENCES)
def test_chunks_keep_what_is_not_finite_from_earlier_tokens(cuda, kind, at):
    n, H, D = 100, 2, 72
    x, gates, decays, states = _recurrence_inputs(cuda, kind, n, H, D, 1, torch.Generator().manual_seed(at))
    run = lambda rows, by_chunks: _recurrence(kind, rows, gates, decays, H, D, [n], [0], [s.clone() for s in states], by_chunks).cpu()      # noqa: E731
    clean = run(x, True)
    assert bool(torch.isfinite(clean).all())
    for col, value in ((2 * H * D + 3, float("inf")), (H * D + 5, float("nan"))):           # a value, a key (of the gated rule: also)
        bad = x.clone()
        bad[at, col] = value
        got, ref = run(bad, True), run(bad, False)
        assert torch.equal(got[:at], clean[:at])
        assert torch.equal(torch.isfinite(got), torch.isfinite(ref)) and not bool(torch.isfinite(got[at:]).all(1).any())


# Operands of every size that a float has, down to its smallest: the split into pieces loses nothing of them.
@pytest.mark.parametrize("low,high", [(-110, -100), (-126, -110), (-149, -126)])
def test_float_products_of_small_operands(cuda, low, high):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(-low)
    M, N, K = 66, 130, 132
    sign = lambda *s: torch.randint(0, 2, s, generator=gen) * 2.0 - 1.0       # noqa: E731
    a = (torch.exp2(low + (high - low) * torch.rand(M, K, generator=gen, dtype=torch.float64)) * sign(M, K)).float()
    w = (torch.exp2(60 + 30 * torch.rand(N, K, generator=gen, dtype=torch.float64)) * sign(N, K)).float()
    assert bool((a != 0).any())
    for x, y in ((a, w), (w, a)):                                           # either operand may be the small one
        ref, size = x.double() @ y.double().T, x.double().abs() @ y.double().abs().T
        c = torch.empty(x.shape[0], y.shape[0], device=cuda)
        ops.gemm_tn_simt(x.to(cuda), y.to(cuda), c, ops.EPI_STORE_F32)
        assert bool(((c.cpu().double() - ref).abs() <= (8 + K / 64) * 2.0 ** -24 * size).all())       # the bound of operands of ordinary size


# What the kernel just before writes: the second operand of a float product, and the positions of attention rows (unless the caller says that
# they stood before). That kernel lets its successor start early and writes for some microseconds more.
def test_operands_made_by_the_kernel_before(cuda):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(3)
    made, a = torch.randn(4096, 4096, generator=gen).to(cuda), torch.randn(128, 4096, generator=gen).to(cuda)
    w, want, got = torch.zeros_like(made), torch.empty(128, 4096, device=cuda), torch.empty(128, 4096, device=cuda)
    ops.gemm_tn_simt(a, made, want, ops.EPI_STORE_F32)
    n, V, H, D = 64, 150_000, 4, 64
    positions = torch.randint(0, 64, (n,), generator=gen)
    logits = torch.zeros(n, V)
    logits[torch.arange(n), positions] = 1.0
    logits, k, v = logits.to(cuda), *(torch.randn(n, 1, 64, D, generator=gen).bfloat16().to(cuda) for _ in range(2))
    q, table, seq = torch.randn(n, H * D, generator=gen).bfloat16().to(cuda), _i32([[i] for i in range(n)], cuda), _i32(range(n), cuda)
    pos, err = torch.zeros(n, dtype=torch.int32, device=cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    attend = lambda at, out: ops.window_attention(q, k, v, table, seq, at, None, None, None, 0, out, H, 1, D, D, 0, 0.1)     # noqa: E731
    heads, after = (torch.empty(n, H * D, dtype=torch.bfloat16, device=cuda) for _ in range(2))
    attend(_i32(positions.tolist(), cuda), heads)
    for _ in range(5):
        w.zero_()
        ops.cast_rows(made, w)
        ops.gemm_tn_simt(a, w, got, ops.EPI_STORE_F32)
        assert torch.equal(got, want)
        pos.zero_()
        ops.argmax_rows(logits, pos, err)
        attend(pos, after)
        assert torch.equal(after, heads)


# A step's portions, some by chunks and the others by the scan: each as if it were alone (the same bits), with scratch for the chunked ones only.
@pytest.mark.parametrize("kind", RECURRENCES)
def test_portions_by_chunks_beside_portions_by_the_scan(cuda, kind):
    H, D, least = 2, 72, 20
    news, starts = [1, 70, 19, 20, 1, 130, 3], [5, 0, 9, 2, 0, 64, 0]
    n, B = sum(news), len(news)
    x, gates, decays, states = _recurrence_inputs(cuda, kind, n, H, D, B, torch.Generator().manual_seed(1))
    mixed = [s.clone() for s in states]
    by_chunks = _recurrence(kind, x, gates, decays, H, D, news, starts, mixed, True, least, least=least)
    by_scan = _recurrence(kind, x, gates, decays, H, D, news, starts, mixed, False, below=least)
    r = 0
    for i, m in enumerate(news):
        own, part = [s[i:i + 1].clone() for s in states], slice(r, r + m)
        alone = _recurrence(kind, x[part].contiguous(), gates[part].contiguous(), decays[part].contiguous(), H, D, [m], starts[i:i + 1], own, m >= least)
        took, other = (by_chunks, by_scan) if m >= least else (by_scan, by_chunks)
        assert torch.equal(took[part], alone) and bool(torch.isnan(other[part]).all())
        assert all(torch.equal(a[i], b[0]) for a, b in zip(mixed, own))
        r += m


# A row's value does not depend on how many rows the step has: the convolution's kernels for few rows and for many (from 592 warps of eight rows
# of a head on; the sequences one by one stay below), a decay per channel and per head, heads that leave lanes of 128 channels idle; the threads
# that prepare a latent's row up to and beyond 128 rows.
@pytest.mark.parametrize("G,H,D,Dv,per_head", [(2, 4, 128, 20, False), (1, 3, 52, 36, True), (1, 6, 4, 128, True)])
def test_convolution_of_few_and_many_rows(cuda, G, H, D, Dv, per_head):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(D)
    C, dd = 2 * G * D + H * Dv, 1 if per_head else D
    news, starts, slots = [1, 33, 2, 300, 3, 264], [0, 0, 1, 9, 2, 0], [2, 0, 4, 1, 5, 3]
    n, row0 = sum(news), [sum(news[:i]) for i in range(6)]
    assert -(-n // 8) * (2 * G + 2 * H) >= 592 > -(-max(news) // 8) * (2 * G + 2 * H)
    seq, pos = [i for i, m in enumerate(news) for _ in range(m)], [s + j for s, m in zip(starts, news) for j in range(m)]
    x, w, st = torch.randn(n, C + 4, generator=gen).to(cuda), torch.randn(C, 4, generator=gen).to(cuda), torch.randn(6, 3, C, generator=gen).to(cuda)
    dec, al, dt = torch.randn(n, H * dd, generator=gen).to(cuda), torch.randn(H, generator=gen).to(cuda), torch.randn(H * dd, generator=gen).to(cuda)
    out = [torch.full((n, C), float("nan"), device=cuda) for _ in range(2)]
    decays = [torch.full((n, H * dd), float("nan"), device=cuda) for _ in range(2)]
    for i, cuts in enumerate(([0, n], row0 + [n])):
        for a, b in zip(cuts, cuts[1:]):                     # (cuts between sequences: nothing reaches across them)
            ops.conv_unit(x[a:b], w, st, _i32(seq[a:b], cuda), _i32(pos[a:b], cuda), _i32([r - a for r in row0], cuda), _i32(slots, cuda), out[i][a:b],
                          G, H, D, Dv, 0.3, update_state=False, decay=(dec[a:b], al, dt, decays[i][a:b]))
    assert torch.equal(out[0], out[1]) and torch.equal(decays[0], decays[1]) and bool(torch.isfinite(out[0]).all())


@pytest.mark.parametrize("H,D,R,C,Q,splits", [(3, 24, 16, 96, 0, 1), (2, 8, 10, 300, 70, 3), (0, 8, 0, 512, 513, 9)])
def test_latent_rows_of_few_and_many_rows(cuda, H, D, R, C, Q, splits):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(C)
    n = 129
    proj = torch.randn(splits, n, H * (D + R) + Q + C + R, generator=gen).to(cuda)
    w, wq, freq = torch.rand(C, generator=gen).to(cuda), torch.rand(max(Q, 1), generator=gen).to(cuda), torch.rand(max(R // 2, 1), generator=gen).to(cuda)
    seq, pos, table, got = _i32([0] * n, cuda), _i32(range(n), cuda), _i32([[0, 1, 2]], cuda), []
    for rows in (128, 129):
        q, full, pages, cq = (torch.zeros(s, device=cuda) for s in ((rows, H * D), (rows, H * (C + R)), (3, 1, 64, C + R), (rows, Q)))
        ops.latent_prepare(proj[:, :rows], w, 1e-6, freq, True, 1.0, seq[:rows], pos[:rows], table, q if H else None, full if H else None, pages, H, D, R, C,
                           None, cq if Q else None, wq if Q else None)
        got.append((q[:128], full[:128], pages.view(192, -1)[:128], cq[:128]))
    assert all(torch.equal(few, many) for few, many in zip(*got)) and bool(got[0][2].any())


# The shares of a row's keys: a share whose weight vanishes in 32 bits still hands on what is not a number, as one product over all keys would;
# a share without keys counts for nothing whatever stands in it.
def test_latent_shares_of_vanishing_weight(cuda):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(4)
    H, C, R, splits = 2, 32, 16, 4
    k = torch.zeros(splits + 1, 1, 64, C + R)
    k[..., :C] = torch.randn(splits + 1, 1, 64, C, generator=gen)
    q = torch.zeros(1, H, C + R)
    q[..., C:] = 1.0
    k[:3, :, :, C:] = torch.tensor([0.0, 40.0, 0.0]).view(3, 1, 1, 1)       # the middle page's scores are 640 above the others'
    k[0, 0, 5:7, 3] = 3e38                                                  # their sum is infinite
    out, partial = torch.empty(1, H * C, dtype=torch.bfloat16, device=cuda), torch.full((splits, 1, H, C + 2), float("nan"), device=cuda)
    i = lambda *v: _i32(v, cuda)                                            # noqa: E731
    ops.latent_prompt(q.view(1, -1).bfloat16().to(cuda), k.bfloat16().to(cuda), out, _i32([[0, 1, 2, 3]], cuda), i(0), i(0), 1, i(0), i(64 * 3 - 1), i(1),
                      H, C, R, 1.0, None, None, 0, partial, 1)
    got, want = out.float().cpu().view(H, C), k[1, 0, :, :C].bfloat16().float().mean(0)
    assert bool(torch.isnan(got[:, 3]).all())                                # 0 * inf
    keep = [c for c in range(C) if c != 3]
    assert float((got[:, keep] - want[keep]).abs().max()) < 2.0 ** -8 * 8     # 64 equal weights, 8 bits of them and of the output


# A step of many rows, whose blocks take several deals of the keys each: the bits of the same rows a few at a time (a block per deal). 8, 3 and 1
# deals; contexts with fewer rounds of keys than warps, so that deals stay empty; one, two and three query heads a key head.
@pytest.mark.parametrize("D,Dv,H,G,window,rows", [(64, 64, 8, 8, 0, 150), (128, 128, 6, 3, 300, 200), (128, 64, 3, 1, 100, 700), (64, 128, 16, 16, 0, 40)])
def test_window_attention_of_many_rows(cuda, D, Dv, H, G, window, rows):
    from camelid_b200.csrc import ops
    gen = torch.Generator().manual_seed(D + rows)
    width = 13
    pos = torch.randint(0, 64 * width, (rows,), generator=gen)
    pos[:4] = torch.tensor([0, 31, 32, 64 * width - 1])
    pages = torch.randint(0, 40, (rows, width), generator=gen).to(torch.int32).to(cuda)
    k, v = (torch.randn(40, G, 64, d, generator=gen).bfloat16().to(cuda) for d in (D, Dv))
    q, sink = torch.randn(rows, H * D, generator=gen).bfloat16().to(cuda), torch.randn(H, generator=gen).to(cuda)
    rel = torch.randn(H, 50, generator=gen).to(cuda)
    seq, pos = _i32(range(rows), cuda), _i32(pos.tolist(), cuda)
    out = [torch.empty(rows, H * Dv, dtype=torch.bfloat16, device=cuda) for _ in range(2)]
    for o, step in zip(out, (rows, 2)):
        for a in range(0, rows, step):
            part = slice(a, min(a + step, rows))
            ops.window_attention(q[part], k, v, pages, seq[part], pos[part], None, None, None, 0, o[part], H, G, D, Dv, window, D ** -0.5, 0, sink,
                                 distance_bias=rel, single=True)
    assert torch.equal(out[0], out[1]) and bool(torch.isfinite(out[0]).all())


# How far the chunked forms lie from 64 bits, beside the scans they replace: no further where the state fades slowly (the scan rounds it at every
# token), little further where it fades at once and a sum of few terms is all there is (their products are rounded once more there).
@pytest.mark.parametrize("kind,decay,most", [("retention", 0.999, 1.0), ("retention", 0.98, 1.1), ("retention", 0.5, 1.35), ("matrix memory", 0.9, 1.25),
                                             ("gated", 0.9, 1.25)])
def test_chunks_are_as_close_as_the_scan(cuda, kind, decay, most):
    n, H, D = 700, 2, 128
    x, gates, decays, states = _recurrence_inputs(cuda, kind, n, H, D, 1, torch.Generator().manual_seed(2))
    off = []
    for by_chunks in (True, False):
        out = _recurrence(kind, x, gates, decays, H, D, [n], [0], [s.clone() for s in states], by_chunks, decay=decay).double().view(n, H, -1)[..., :D]
        off.append(out)
    q, k, v = (x[:, i * H * D:(i + 1) * H * D].double().view(n, H, D, 1) for i in range(3))
    fade = torch.full((n, H, 1, 1), float(torch.tensor(decay)), dtype=torch.float64, device=cuda)
    step, beta = torch.ones_like(fade), torch.zeros_like(fade)             # S <- S fade + (step v - beta S fade k) k^T
    if kind == "matrix memory":
        b = float(torch.tensor(decay))
        gi, gf = (15.0 * torch.tanh((x[:, 3 * H * D + i * H:3 * H * D + (i + 1) * H].double() + b) / 15.0) for i in (0, 1))
        gf, top = torch.nn.functional.logsigmoid(gf), torch.zeros(H, dtype=torch.float64, device=cuda)
        for i in range(n):
            new = torch.maximum(gf[i] + top, gi[i])
            fade[i, :, 0, 0], step[i, :, 0, 0], top = torch.exp(gf[i] + top - new), torch.exp(gi[i] - new), new
        q = q * 0.1
    elif kind == "gated":
        fade, step = decays.double().view(n, H, 1, D), torch.sigmoid(gates.double()).view(n, H, 1, 1)
        beta = step
    S, ref = torch.zeros(H, D, D, dtype=torch.float64, device=cuda), []
    for i in range(n):
        S = S * fade[i]
        S = S + (step[i] * v[i] - beta[i] * (S @ k[i])) * k[i].transpose(1, 2)
        ref.append((S @ q[i]).squeeze(2))
    ref = torch.stack(ref)
    off = [float((o - ref).norm() / ref.norm()) for o in off]
    assert off[0] <= most * off[1] and off[0] < 1e-6
