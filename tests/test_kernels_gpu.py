"""Each kernel alone against a plain fp32 reference of the same op, at sizes other than the
engine tests': widths and vocabularies that are no power of two, odd head counts, head sizes in
steps of 16, pages of several sizes."""
import math

import pytest
import torch

import plain_llama

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_steadyinfer_b200.csrc import ops as o
    return o


def graph_time_us(fn, n=20):
    """Device time of one call of ``fn(i)`` in microseconds: calls i = 0 .. n-1 recorded into a CUDA graph and
    replayed, so that the host's part of a call (tens of microseconds from Python) is not in the figure."""
    fn(0)
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        fn(0)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            for i in range(n):
                fn(i)
    for _ in range(2):
        graph.replay()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    graph.replay()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) * 1000 / n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V,d,T", [(1000, 96, 7), (4099, 1336, 33)])
def test_embedding(dtype, V, d, T):
    g = torch.Generator().manual_seed(0)
    table = torch.randn(V, d, generator=g).to(dtype).to(DEV)
    tok = torch.randint(0, V, (T,), generator=g, dtype=torch.int32).to(DEV)
    out = torch.empty(T, d, dtype=torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().embedding_gather(tok, table, out, status)
    assert torch.equal(out, table[tok.long()].float())
    assert status.item() == 0
    tok[T // 2] = V                                  # outside the vocabulary: flagged, row zeroed
    ops().embedding_gather(tok, table, out, status)
    assert status.item() == 1 and out[T // 2].abs().max().item() == 0


@pytest.mark.parametrize("xdtype,wdtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                           (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("d,T,eps", [(96, 5, 1e-6), (1336, 19, 1e-5), (5120, 3, 1e-5)])
def test_add_rmsnorm(xdtype, wdtype, d, T, eps):
    g = torch.Generator().manual_seed(1)
    resid = torch.randn(T, d, generator=g).to(DEV)
    delta = torch.randn(T, d, generator=g).to(xdtype).to(DEV)
    w = (1 + 0.1 * torch.randn(d, generator=g)).to(wdtype).to(DEV)
    h = resid.double() + delta.double()
    want = plain_llama.rmsnorm(h.cpu(), w.double().cpu(), eps)
    r2 = resid.clone()
    out = torch.empty(T, d, dtype=xdtype, device=DEV)
    ops().add_rmsnorm(r2, delta, w, eps, out)
    assert torch.allclose(r2.double(), h, atol=1e-6)
    tol = 1e-5 if xdtype == torch.float32 else 2 ** -8 * want.abs().max().item()
    assert (out.double().cpu() - want).abs().max().item() <= tol
    # rows: only the listed rows, stream untouched
    rows = torch.tensor([T - 1, 0, T - 1], dtype=torch.int32, device=DEV)
    r3 = resid.clone()
    out2 = torch.empty(3, d, dtype=xdtype, device=DEV)
    ops().add_rmsnorm(r3, delta, w, eps, out2, rows=rows)
    assert torch.equal(r3, resid)
    assert torch.equal(out2, out[rows.long()])
    # without delta
    out3 = torch.empty(T, d, dtype=xdtype, device=DEV)
    ops().add_rmsnorm(r3, None, w, eps, out3)
    want3 = plain_llama.rmsnorm(resid.double().cpu(), w.double().cpu(), eps)
    assert (out3.double().cpu() - want3).abs().max().item() <= tol
    # with something to fetch ahead into L2 (a hint for the launch after this one): the same numbers,
    # for tensors below one chunk, of an odd size, and larger than the most that is fetched
    for n in (100, 4096 * 3 + 72, 20 << 20):
        nxt = torch.zeros(n, dtype=torch.uint8, device=DEV)
        r4 = resid.clone()
        out4 = torch.empty(T, d, dtype=xdtype, device=DEV)
        ops().add_rmsnorm(r4, delta, w, eps, out4, ahead=nxt)
        assert torch.equal(out4, out) and torch.equal(r4, r2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,F", [(3, 320), (17, 1336)])
def test_swiglu(dtype, T, F):
    g = torch.Generator().manual_seed(2)
    gu = (3 * torch.randn(T, 2 * F, generator=g)).to(dtype).to(DEV)
    out = torch.empty(T, F, dtype=dtype, device=DEV)
    ops().swiglu(gu, out)
    want = plain_llama.swiglu(gu[:, :F].double().cpu(), gu[:, F:].double().cpu())
    tol = 1e-5 if dtype == torch.float32 else 2 ** -8 * want.abs().max().item()
    assert (out.double().cpu() - want).abs().max().item() <= tol


def _interleave(gate, up, group):
    """Columns of gate and up interleaved in groups of `group`, as the stacked projection lays them out."""
    T, F = gate.shape
    return torch.stack([gate.view(T, F // group, group), up.view(T, F // group, group)], 2).reshape(T, 2 * F)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,F,group", [(3, 320, 8), (5, 1336, 8), (4, 36, 4), (2, 30, 3)])
def test_swiglu_interleaved(dtype, T, F, group):
    g = torch.Generator().manual_seed(22)
    gate = (3 * torch.randn(T, F, generator=g)).to(dtype)
    up = (3 * torch.randn(T, F, generator=g)).to(dtype)
    gu = _interleave(gate, up, group).contiguous().to(DEV)
    out = torch.empty(T, F, dtype=dtype, device=DEV)
    ops().swiglu(gu, out, group)
    want = plain_llama.swiglu(gate.double(), up.double())
    tol = 1e-5 if dtype == torch.float32 else 2 ** -8 * want.abs().max().item()
    assert (out.double().cpu() - want).abs().max().item() <= tol


@pytest.mark.parametrize("M,F,K", [(1, 64, 96), (8, 1336, 320), (11, 40, 1000), (16, 256, 72), (3, 4760, 2048), (8, 9600, 40), (12, 4760, 328),   # tiles in turn
                                   (5, 1184, 2088), (13, 1176, 4104), (2, 8, 2056)])                                                             # sixteen warps a tile
def test_gemm_skinny_swiglu(M, F, K):
    """The few-row gate/up product with the activation in its epilogue equals the product stored in bf16
    followed by the activation kernel."""
    g = torch.Generator().manual_seed(23)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    wg = (torch.randn(F, K, generator=g) / math.sqrt(K)).to(torch.bfloat16)
    wu = (torch.randn(F, K, generator=g) / math.sqrt(K)).to(torch.bfloat16)
    w = _interleave(wg.t().contiguous(), wu.t().contiguous(), 8).t().contiguous().to(DEV)     # rows interleaved
    out = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops().gemm_skinny_swiglu(a, w, out)
    gu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device=DEV)
    ops().gemm_skinny(a, w, gu)
    two = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    ops().swiglu(gu, two, 8)
    assert torch.equal(out, two)
    want = plain_llama.swiglu(a.double().cpu() @ wg.double().T, a.double().cpu() @ wu.double().T)
    assert (out.double().cpu() - want).abs().max().item() <= 2 ** -7 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("M,N,K", [(1, 1000, 96), (7, 513, 320), (130, 200, 1336), (64, 64, 16), (3, 5, 7)])
def test_gemm_f32(M, N, K):
    g = torch.Generator().manual_seed(3)
    a = torch.randn(M, K, generator=g).to(DEV)
    w = torch.randn(N, K, generator=g).to(DEV)
    out = torch.empty(M, N, device=DEV)
    ops().gemm_f32(a, w, out)
    want = a.double() @ w.double().T
    assert (out.double() - want).abs().max().item() <= 1e-6 * K * 4
    # a row's result does not depend on the other rows of the call
    one = torch.empty(1, N, device=DEV)
    ops().gemm_f32(a[M - 1:M], w, one)
    assert torch.equal(one[0], out[M - 1])


def build_cache(dtype, lengths, H, KV, hs, page_size, seed, shuffle=True):
    """Random q/k/v of several whole sequences laid into a paged cache with shuffled pages."""
    g = torch.Generator().manual_seed(seed)
    S = len(lengths)
    blocks = [-(-n // page_size) for n in lengths]
    num_pages = sum(blocks) + 3
    perm = torch.randperm(num_pages, generator=g).tolist() if shuffle else list(range(num_pages))
    W = max(blocks)
    table = torch.full((S, W), -1, dtype=torch.int32)
    kc = torch.zeros(num_pages, KV, page_size, hs)
    vc = torch.zeros(num_pages, KV, page_size, hs)
    seqs = []
    p = 0
    for s, n in enumerate(lengths):
        q = torch.randn(n, H, hs, generator=g).to(dtype).float()
        k = torch.randn(n, KV, hs, generator=g).to(dtype).float()
        v = torch.randn(n, KV, hs, generator=g).to(dtype).float()
        for b in range(blocks[s]):
            page = perm[p]; p += 1
            table[s, b] = page
            m = min(page_size, n - b * page_size)
            kc[page, :, :m] = k[b * page_size:b * page_size + m].transpose(0, 1)
            vc[page, :, :m] = v[b * page_size:b * page_size + m].transpose(0, 1)
        seqs.append((q, k, v))
    return seqs, table, kc.to(dtype), vc.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,KV,hs,page_size,window", [(4, 2, 16, 16, None), (3, 1, 32, 8, None), (6, 3, 48, 4, None),
                                                     (8, 2, 128, 16, None), (5, 5, 80, 32, 7), (2, 1, 256, 16, 40)])
def test_paged_attention_ref(dtype, H, KV, hs, page_size, window):
    lengths = [1, 37, 130]
    seqs, table, kc, vc = build_cache(dtype, lengths, H, KV, hs, page_size, seed=4)
    scale = 1.0 / math.sqrt(hs)
    # rows: the last 5 positions of each sequence (a portion that continues from the cache)
    qrows, pos, rseq, want = [], [], [], []
    for s, (q, k, v) in enumerate(seqs):
        full = plain_llama.attention(q.double(), k.double(), v.double(), scale, window)
        for t in range(max(0, lengths[s] - 5), lengths[s]):
            qrows.append(q[t].reshape(-1)); pos.append(t); rseq.append(s); want.append(full[t].reshape(-1))
    q = torch.stack(qrows).to(dtype).to(DEV)
    out = torch.empty_like(q)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().paged_attention_ref(q, kc.to(DEV), vc.to(DEV), table.to(DEV), torch.tensor(rseq, dtype=torch.int32, device=DEV),
                              torch.tensor(pos, dtype=torch.int32, device=DEV), out, page_size, len(lengths),
                              H, KV, hs, scale, window or 0, status)
    assert status.item() == 0
    tol = 2e-6 if dtype == torch.float32 else 2 ** -8
    assert (out.double().cpu() - torch.stack(want)).abs().max().item() <= tol * 4


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,KV,hs,rot,page_size", [(4, 2, 16, 16, 16), (3, 1, 32, 32, 8), (5, 5, 80, 40, 4), (8, 2, 128, 128, 16)])
def test_rope_kv_write(dtype, H, KV, hs, rot, page_size):
    g = torch.Generator().manual_seed(5)
    lengths = [9, 40]
    T = sum(lengths)
    qkv = torch.randn(T, (H + 2 * KV) * hs, generator=g).to(dtype)
    pos = torch.cat([torch.arange(100, 100 + n) for n in lengths]).to(torch.int32)     # far positions
    rseq = torch.cat([torch.full((n,), s) for s, n in enumerate(lengths)]).to(torch.int32)
    W = (100 + max(lengths)) // page_size + 1
    num_pages = 2 * W
    table = torch.randperm(num_pages, generator=g).to(torch.int32).view(2, W)
    freqs = plain_llama.rope_frequencies(rot, 500000.0, {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0,
                                                         "high_freq_factor": 4.0, "original_max_position_embeddings": 64})
    kc = torch.zeros(num_pages, KV, page_size, hs, dtype=dtype, device=DEV)
    vc = torch.zeros_like(kc)
    dq = qkv.clone().to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().rope_kv_write(dq, pos.to(DEV), rseq.to(DEV), freqs.to(DEV), rot, table.to(DEV), kc, vc, page_size, 2,
                        H, KV, hs, status)
    assert status.item() == 0
    x = qkv.double()
    q3 = x[:, :H * hs].view(T, H, hs); k3 = x[:, H * hs:(H + KV) * hs].view(T, KV, hs); v3 = x[:, (H + KV) * hs:].view(T, KV, hs)
    def rot_part(t3):
        r = plain_llama.rope(t3[..., :rot], pos, freqs)
        return torch.cat([r, t3[..., rot:]], -1)
    tol = 1e-5 if dtype == torch.float32 else 2 ** -8 * 5
    wq, wk = rot_part(q3), rot_part(k3)
    assert (dq[:, :H * hs].double().cpu().view(T, H, hs) - wq).abs().max().item() <= tol
    kc, vc = kc.double().cpu(), vc.double().cpu()
    for t in range(T):
        page = table[rseq[t], pos[t] // page_size].item()
        off = pos[t].item() % page_size
        assert (kc[page, :, off] - wk[t]).abs().max().item() <= tol
        assert torch.equal(vc[page, :, off], v3[t])


@pytest.mark.parametrize("R,V", [(1, 31), (5, 1000), (24, 50257), (3, 128256)])
def test_argmax_split(R, V):
    """The greedy pick with a row split over many blocks: ties to the lowest index, also across blocks;
    repeated calls with different numbers of rows share one scratch buffer."""
    g = torch.Generator().manual_seed(60 + R)
    o = ops()
    scratch = torch.zeros(o.argmax_scratch_words(32), dtype=torch.int32, device=DEV)
    for rows in (R, max(1, R // 2), R):
        logits = (2.5 * torch.randn(rows, V, generator=g)).float()
        top = logits.max().item() + 1
        logits[0, V // 3] = logits[0, V - 1] = top                 # a tie in different blocks
        dl = logits.to(DEV)
        out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
        o.argmax(dl, out, scratch)
        assert out.tolist() == [plain_llama.sample(logits[r]) for r in range(rows)]
        assert out[0].item() == V // 3
        one = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
        o.sample(dl, one)
        assert torch.equal(one, out)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm_rows_off_the_residual_stream(dtype):
    """The norm alone over rows, and over the heads of a token inside a stacked projection (a 3-D view with two
    strides), in place and into another buffer, against torch; what lies beside the rows is not touched."""
    g = torch.Generator().manual_seed(29)
    T, H, KV, hs, eps = 37, 5, 2, 48, 3e-6
    w = (1 + 0.1 * torch.randn(hs, generator=g)).to(dtype).to(DEV)
    qkv = torch.randn(T, (H + 2 * KV) * hs, generator=g).to(dtype).to(DEV)
    before = qkv.clone()
    q = qkv[:, :H * hs].view(T, H, hs)
    want = plain_llama.rmsnorm(before[:, :H * hs].double().cpu().view(T, H, hs), w.double().cpu(), eps)
    ops().rmsnorm_rows(q, w, eps)
    tol = 1e-5 if dtype == torch.float32 else 2 ** -7 * want.abs().max().item()
    assert (qkv[:, :H * hs].double().cpu().view(T, H, hs) - want).abs().max().item() <= tol
    assert torch.equal(qkv[:, H * hs:], before[:, H * hs:]), "keys and values beside the queries are as they were"
    x = torch.randn(9, 1336, generator=g).to(dtype).to(DEV)
    w2 = (1 + 0.1 * torch.randn(1336, generator=g)).to(DEV)                      # a weight kept in 32-bit
    out = torch.full_like(x, float("nan"))
    ops().rmsnorm_rows(x, w2, 1e-5, out)
    want = plain_llama.rmsnorm(x.double().cpu(), w2.double().cpu(), 1e-5)
    assert (out.double().cpu() - want).abs().max().item() <= (1e-5 if dtype == torch.float32 else 2 ** -7 * want.abs().max().item())
    with pytest.raises(ops().KernelError):
        ops().rmsnorm_rows(x.t(), w2, 1e-5)


def test_sampling_kernel_matches_plain():
    g = torch.Generator().manual_seed(6)
    V, R = 1000, 24
    logits = (2.5 * torch.randn(R, V, generator=g)).float()
    logits[3, 17] = logits[3, 400] = logits[3].max() + 1          # a tie: the lowest index wins
    dl = logits.to(DEV)
    out = torch.empty(R, dtype=torch.int32, device=DEV)
    ops().sample(dl, out)
    assert out.tolist() == [plain_llama.sample(logits[r]) for r in range(R)]
    assert out[3].item() == 17
    cases = [(0.7, 0, 0.9), (1.0, 5, 1.0), (1.3, 50, 0.5), (0.5, 0, 1.0), (1.0, 1, 1.0), (2.0, 0, 0.1)]
    for temp, k, p in cases:
        t = torch.full((R,), temp, device=DEV)
        tk = torch.full((R,), k, dtype=torch.int32, device=DEV)
        tp = torch.full((R,), p, device=DEV)
        seed = torch.arange(R, dtype=torch.int64, device=DEV) * 7919 + 1
        ctr = torch.arange(R, dtype=torch.int64, device=DEV) % 5
        ops().sample(dl, out, temperature=t, top_k=tk, top_p=tp, seed=seed, counter=ctr)
        want = [plain_llama.sample(logits[r], temp, k, p, seed=int(seed[r]), counter=int(ctr[r])) for r in range(R)]
        assert out.tolist() == want, (temp, k, p)


def test_sampling_treats_both_zeros_as_equal():
    """-0.0 and +0.0 are equal logits: top-k keeps all ties of the k-th, whichever zero they are, and the draw
    goes over all of them in index order, as the plain sampler's (a random search with rounded logits found the
    kernel's integer image of the logits telling the two zeros apart)."""
    V, R = 40, 16
    logits = torch.full((R, V), -3.0)
    zeros = [3, 7, 8, 21, 39]
    for r in range(R):
        for j, i in enumerate(zeros):
            logits[r, i] = -0.0 if (r + j) % 2 else 0.0
    dl = logits.to(DEV)
    out = torch.empty(R, dtype=torch.int32, device=DEV)
    seed = torch.arange(R, dtype=torch.int64, device=DEV) * 31 + 5
    ctr = torch.arange(R, dtype=torch.int64, device=DEV)
    for temp, k, p in [(1.0, 1, 1.0), (0.7, 2, 0.5), (1.5, 0, 0.0001)]:
        ops().sample(dl, out, temperature=torch.full((R,), temp, device=DEV),
                     top_k=torch.full((R,), k, dtype=torch.int32, device=DEV), top_p=torch.full((R,), p, device=DEV),
                     seed=seed, counter=ctr)
        want = [plain_llama.sample(logits[r], temp, k, p, seed=int(seed[r]), counter=int(ctr[r])) for r in range(R)]
        assert out.tolist() == want, (temp, k, p)
        assert len(set(want)) > 1 and set(want) <= set(zeros), "the draws spread over all five zeros"


def test_sampling_distribution():
    """Draws over many counters follow softmax(x / T) restricted by top-p."""
    V = 37
    g = torch.Generator().manual_seed(7)
    x = torch.randn(V, generator=g).float()
    R = 4096
    dl = x.to(DEV).repeat(R, 1)
    out = torch.empty(R, dtype=torch.int32, device=DEV)
    t = torch.full((R,), 0.8, device=DEV)
    tp = torch.full((R,), 0.9, device=DEV)
    seed = torch.full((R,), 1234, dtype=torch.int64, device=DEV)
    ctr = torch.arange(R, dtype=torch.int64, device=DEV)
    ops().sample(dl, out, temperature=t, top_p=tp, seed=seed, counter=ctr)
    p = torch.softmax(x.double() / 0.8, 0)
    order = torch.argsort(p, descending=True)
    csum = torch.cumsum(p[order], 0)
    kept = order[: int((csum < 0.9).sum()) + 1]
    pk = torch.zeros(V, dtype=torch.double); pk[kept] = p[kept] / p[kept].sum()
    freq = torch.bincount(out.cpu().long(), minlength=V).double() / R
    assert freq[pk == 0].sum().item() == 0
    assert (freq - pk).abs().max().item() < 4 * math.sqrt(0.25 / R)


# ---- tensor-core attention -----------------------------------------------------------------

def _torch_attention(q_row, kc, vc, table_row, pos, H, KV, hs, scale, window=0):
    """One query row [H * hs] at position ``pos`` against the pages of its sequence, in float32 with torch
    alone (no kernel of the package): softmax(scale q K^T) V over keys first..pos."""
    G = H // KV
    n_blocks = pos // kc.shape[2] + 1
    k = kc[table_row[:n_blocks].long()].float().permute(1, 0, 2, 3).reshape(KV, -1, hs)[:, :pos + 1]
    v = vc[table_row[:n_blocks].long()].float().permute(1, 0, 2, 3).reshape(KV, -1, hs)[:, :pos + 1]
    first = max(0, pos - window + 1) if window else 0
    sc = torch.einsum("kgd,kjd->kgj", q_row.float().view(KV, G, hs), k[:, first:]) * scale
    return torch.einsum("kgj,kjd->kgd", torch.softmax(sc, -1), v[:, first:]).reshape(-1)


def _items_for(lengths, tails, dec_tokens, por_tokens):
    """Rows = the last ``tails[s]`` tokens of each sequence, cut into kernel items."""
    dec, por, rows = [], [], []
    row = 0
    for s, (n, tl) in enumerate(zip(lengths, tails)):
        tl = min(tl, n)
        pos0 = n - tl
        if tl <= dec_tokens:
            dec.append((s, row, tl, pos0))
        else:
            for b in range(0, tl, por_tokens):
                por.append((s, row + b, min(por_tokens, tl - b), pos0 + b))
        rows += [(s, pos0 + i) for i in range(tl)]
        row += tl
    return dec, por, rows


def _run_tc_attention(seqs, table, kc, vc, lengths, tails, H, KV, hs, page_size, window, nsplit, tma=False, tc05=False):
    o = ops()
    G = H // KV
    if tc05 and not o.attn_portion_tc05_ok(H, KV, hs, page_size):
        pytest.skip("the tcgen05 portion kernel does not take this layout")
    if tma and not o.attn_decode_tma_ok(H, KV, hs, page_size):
        pytest.skip("the TMA decode kernel does not take this layout")
    dec_tokens = (o.attn_decode_tma_rows(H, KV) if tma else o.attn_decode_rows(H, KV, hs)) // G
    por_tokens = o.attn_portion_tc05_tokens(H, KV) if tc05 else o.attn_portion_tokens(H, KV, hs)
    dec, por, rows = _items_for(lengths, tails, dec_tokens, por_tokens)
    q = torch.stack([seqs[s][0][p].reshape(-1) for s, p in rows]).to(torch.bfloat16).to(DEV)
    out = torch.full_like(q, float("nan"))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    kcd, vcd, tb = kc.to(DEV), vc.to(DEV), table.to(DEV)
    if dec:
        items = torch.tensor(dec, dtype=torch.int32, device=DEV)
        scratch = None
        floats = o.attn_decode_tma_scratch_floats if tma else o.attn_decode_scratch_floats
        if nsplit > 1:
            scratch = torch.zeros(floats(len(dec), H, KV, hs, nsplit), device=DEV)
        more = {"max_rows": max(d[2] for d in dec) * G} if tma else {}      # few rows: the swapped products
        (o.attn_decode_tma if tma else o.attn_decode)(
            q, kcd, vcd, tb, items, out, page_size, len(lengths), H, KV, hs, scale, window or 0,
            nsplit=nsplit, scratch=scratch, status=status, **more)
    if por:
        items = torch.tensor(por, dtype=torch.int32, device=DEV)
        (o.attn_portion_tc05 if tc05 else o.attn_portion)(
            q, kcd, vcd, tb, items, out, page_size, len(lengths), H, KV, hs, scale, window or 0, status=status)
    assert status.item() == 0
    return out.double().cpu(), rows, bool(dec), bool(por)


@pytest.mark.parametrize("H,KV,hs,page_size,window", [
    (4, 2, 16, 16, None), (3, 1, 32, 8, None), (6, 3, 48, 4, None), (8, 2, 128, 16, None), (32, 8, 128, 16, None),
    (5, 5, 80, 32, 7), (2, 1, 256, 16, 40), (32, 1, 64, 16, None), (40, 1, 128, 16, None), (24, 8, 128, 16, 100),
    (14, 2, 64, 64, None), (9, 3, 96, 16, 65), (8, 8, 64, 8, None), (20, 1, 128, 32, 200), (16, 2, 64, 16, 70)])
@pytest.mark.parametrize("nsplit", [1, 3])
@pytest.mark.parametrize("tma", [False, True, "tc05"], ids=["cp_async", "tma", "tcgen05"])
def test_attention_tensor_cores(H, KV, hs, page_size, window, nsplit, tma):
    tc05 = tma == "tc05"
    tma = bool(tma)
    if tc05 and nsplit != 1:
        pytest.skip("splits concern the decode kernel only")
    lengths = [1, 37, 130, 700, 64, 129]
    tails = [1, 1, 3, 700, 64, 2]           # decode rows, short runs, a whole long prompt, an exact tile
    seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, page_size, seed=8)
    out, rows, used_dec, used_por = _run_tc_attention(seqs, table, kc, vc, lengths, tails, H, KV, hs, page_size, window,
                                                      nsplit, tma, tc05)
    assert used_por
    scale = 1.0 / math.sqrt(hs)
    full = [plain_llama.attention(q.double(), k.double(), v.double(), scale, window) for q, k, v in seqs]
    want = torch.stack([full[s][p].reshape(-1) for s, p in rows])
    assert not torch.isnan(out).any(), "every row was written"
    # probabilities and outputs are rounded to bf16 (2^-9 relative each): 2^-8 of the largest value
    vmax = max(v.abs().max().item() for _, _, v in seqs)
    assert (out - want).abs().max().item() <= 2 ** -8 * vmax


@pytest.mark.parametrize("hs,page_size", [(128, 16), (64, 8), (32, 4)])
def test_attention_finds_one_far_key(hs, page_size):
    """One key among hundreds matches the query strongly: the output is that key's value row,
    wherever the key lies (first and last slot of a page, edges of the 64-key tiles, the row's
    own position), for a decode row, with and without splits, and for a row inside a portion."""
    H, KV = 4, 2
    n = 333
    g = torch.Generator().manual_seed(9)
    for target in [0, page_size - 1, page_size, 63, 64, 65, 127, 128, 200, n - 2, n - 1]:
        q = 0.1 * torch.randn(n, H, hs, generator=g)
        k = 0.1 * torch.randn(n, KV, hs, generator=g)
        v = torch.randn(n, KV, hs, generator=g)
        direction = torch.randn(hs, generator=g)
        direction /= direction.norm()
        k[target, :, :] = 6.0 * direction
        q[n - 1, :, :] = 6.0 * math.sqrt(hs) * direction        # score 36 against ~0 elsewhere
        q[n - 5, :, :] = 6.0 * math.sqrt(hs) * direction
        seqs = [(q.to(torch.bfloat16).float(), k.to(torch.bfloat16).float(), v.to(torch.bfloat16).float())]
        blocks = -(-n // page_size)
        perm = torch.randperm(blocks + 2, generator=g)
        table = perm[:blocks].to(torch.int32).view(1, -1)
        kc = torch.zeros(blocks + 2, KV, page_size, hs); vc = torch.zeros_like(kc)
        for b in range(blocks):
            m = min(page_size, n - b * page_size)
            kc[table[0, b], :, :m] = seqs[0][1][b * page_size:b * page_size + m].transpose(0, 1)
            vc[table[0, b], :, :m] = seqs[0][2][b * page_size:b * page_size + m].transpose(0, 1)
        kc, vc = kc.to(torch.bfloat16), vc.to(torch.bfloat16)
        for tails, nsplit, tma, tc05 in (([1], 1, False, False), ([1], 4, False, False), ([n], 1, False, False),
                                         ([1], 1, True, False), ([1], 4, True, False), ([n], 1, True, True)):
            if tma and not ops().attn_decode_tma_ok(H, KV, hs, page_size):
                continue
            if tc05 and not ops().attn_portion_tc05_ok(H, KV, hs, page_size):
                continue
            out, rows, _, _ = _run_tc_attention(seqs, table, kc, vc, [n], tails, H, KV, hs, page_size, None, nsplit, tma, tc05)
            for r, (s, p) in enumerate(rows):
                if p not in (n - 1, n - 5) or target > p:
                    continue
                got = out[r].view(H, hs)
                want = seqs[0][2][target].double().repeat_interleave(H // KV, 0)
                assert (got - want).abs().max().item() < 0.02, (target, tails, nsplit, p)


def test_attention_window_edge():
    """The key just inside the window counts, the one just outside does not."""
    H, KV, hs, page_size, window, n = 2, 1, 64, 16, 50, 180
    g = torch.Generator().manual_seed(10)
    direction = torch.randn(hs, generator=g); direction /= direction.norm()
    for target, visible in ((n - 1 - window, False), (n - window, True)):
        q = 0.1 * torch.randn(n, H, hs, generator=g)
        k = 0.1 * torch.randn(n, KV, hs, generator=g)
        v = torch.randn(n, KV, hs, generator=g)
        k[target] = 6.0 * direction
        q[n - 1] = 6.0 * math.sqrt(hs) * direction
        seqs = [(q.to(torch.bfloat16).float(), k.to(torch.bfloat16).float(), v.to(torch.bfloat16).float())]
        blocks = -(-n // page_size)
        table = torch.arange(blocks, dtype=torch.int32).view(1, -1)
        kc = torch.zeros(blocks, KV, page_size, hs); vc = torch.zeros_like(kc)
        for b in range(blocks):
            m = min(page_size, n - b * page_size)
            kc[b, :, :m] = seqs[0][1][b * page_size:b * page_size + m].transpose(0, 1)
            vc[b, :, :m] = seqs[0][2][b * page_size:b * page_size + m].transpose(0, 1)
        for tails, tma, tc05 in (([1], False, False), ([n], False, False), ([1], True, False), ([n], True, True)):
            out, rows, _, _ = _run_tc_attention(seqs, table, kc.to(torch.bfloat16), vc.to(torch.bfloat16), [n], tails,
                                                H, KV, hs, page_size, window, 1, tma, tc05)
            got = out[-1].view(H, hs)
            hit = (got - seqs[0][2][target].double()).abs().max().item() < 0.02
            assert hit == visible, (target, tails)


@pytest.mark.parametrize("H,KV,hs,page_size,window", [
    (4, 2, 64, 16, 40), (8, 2, 128, 16, 100), (2, 1, 64, 8, 11), (6, 3, 64, 16, 70), (5, 5, 80, 32, 7),
    (16, 2, 128, 32, 200), (3, 1, 32, 4, 5), (2, 1, 256, 16, 129)])
@pytest.mark.parametrize("nsplit", [1, 3])
@pytest.mark.parametrize("tma", [False, True, "tc05"], ids=["cp_async", "tma", "tcgen05"])
def test_attention_window_with_pages_given_back(H, KV, hs, page_size, window, nsplit, tma):
    """Pages that lie wholly before the window of a step's first token have been given back: their table
    entries are -1 and the pages hold someone else's data (NaN here). The kernels round the first key
    down to a tile of 64, so such pages fall inside their first tile; they are neither looked up
    nor read, and no status is raised."""
    tc05 = tma == "tc05"
    tma = bool(tma)
    if tc05 and nsplit != 1:
        pytest.skip("splits concern the decode kernel only")
    lengths = [1, 37, 130, 700, 64, 129, 650, 333]
    tails = [1, 1, 3, 45, 64, 2, 300, 1]
    seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, page_size, seed=12)
    gone = 0
    for s, (n, tl) in enumerate(zip(lengths, tails)):
        first_needed = (n - min(tl, n)) - window + 1          # what the step's first token reads from
        for b in range(max(0, first_needed) // page_size):
            kc[table[s, b]] = float("nan"); vc[table[s, b]] = float("nan")
            table[s, b] = -1
            gone += 1
    assert gone > 20
    out, rows, used_dec, used_por = _run_tc_attention(seqs, table, kc, vc, lengths, tails, H, KV, hs, page_size, window,
                                                      nsplit, tma, tc05)
    assert used_dec and used_por
    scale = 1.0 / math.sqrt(hs)
    full = [plain_llama.attention(q.double(), k.double(), v.double(), scale, window) for q, k, v in seqs]
    want = torch.stack([full[s][p].reshape(-1) for s, p in rows])
    assert not torch.isnan(out).any(), "every row was written, and nothing of a page given back was read"
    vmax = max(v.abs().max().item() for _, _, v in seqs)
    assert (out - want).abs().max().item() <= 2 ** -8 * vmax


@pytest.mark.parametrize("H,KV,hs,page_size,window", [(32, 8, 128, 16, None), (4, 2, 64, 8, None), (16, 2, 128, 32, 300),
                                                     (8, 8, 64, 16, None), (40, 1, 128, 16, None)])
@pytest.mark.parametrize("budget", [1, 7, 37, 200])
def test_decode_with_shares_of_equal_length(H, KV, hs, page_size, window, budget):
    """Decode items of very different lengths, each cut into its own number of shares by ``split_work``:
    the same outputs as whole sequences give, whatever the budget of shares, with empty items and unused
    work entries in between, twice over the same scratch."""
    o = ops()
    if not o.attn_decode_tma_ok(H, KV, hs, page_size):
        pytest.skip("the TMA decode kernel does not take this layout")
    G = H // KV
    lengths = [2000, 3, 64, 700, 129, 1, 65, 1200]
    seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, page_size, seed=21)
    dec = [(s, s, 1, n - 1) for s, n in enumerate(lengths)]
    dec.insert(3, (0, 0, 0, 0))                                  # an empty item, as fixed shapes are padded with
    tiles = []
    for (_, _, n, pos0) in dec:
        first = max(0, pos0 - window + 1) // 64 * 64 if window else 0
        tiles.append(-(-(pos0 + n - first) // 64) if n else 0)
    entries = budget + len(dec)
    work_h = o.split_work(tiles, budget, entries, 32, 2)
    live = work_h[work_h[:, 0] >= 0]
    assert len(live) <= budget + len(lengths) and set(live[:, 0].tolist()) == {i for i, t in enumerate(tiles) if t}
    for i in set(live[:, 0].tolist()):
        mine = live[live[:, 0] == i]
        assert sorted(mine[:, 1].tolist()) == list(range(mine[0, 2])) and len(set(mine[:, 3].tolist())) == 1
    if budget >= 37 and not window:
        shares = {i: (live[:, 0] == i).sum() for i in range(len(dec))}
        assert shares[0] > 4 * shares[1 + 1], "the longest item is cut into the most shares"
    q = torch.stack([seqs[s][0][n - 1].reshape(-1) for s, n in enumerate(lengths)]).to(torch.bfloat16).to(DEV)
    items = torch.tensor(dec, dtype=torch.int32, device=DEV)
    work = torch.tensor(work_h, dtype=torch.int32, device=DEV)
    scratch = torch.zeros(o.attn_decode_tma_work_floats(entries, H, KV, hs), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    full = [plain_llama.attention(qq.double(), k.double(), v.double(), scale, window) for qq, k, v in seqs]
    want = torch.stack([full[s][n - 1].reshape(-1) for s, n in enumerate(lengths)])
    vmax = max(v.abs().max().item() for _, _, v in seqs)
    for turn in range(2):
        out = torch.full_like(q, float("nan"))
        o.attn_decode_tma(q, kc.to(DEV), vc.to(DEV), table.to(DEV), items, out, page_size, len(lengths), H, KV, hs, scale,
                          window or 0, work=work, scratch=scratch, status=status, max_rows=G)
        assert status.item() == 0
        assert not torch.isnan(out).any(), "every row was written"
        assert (out.double().cpu() - want).abs().max().item() <= 2 ** -8 * vmax, turn


def test_decode_with_more_work_entries_than_65535():
    """A work list of any length: the entries with work first, the others leave. Outputs to the bit those of the short list."""
    o = ops()
    H, KV, hs, ps, lengths = 8, 2, 64, 16, [700, 3, 129]
    if not o.attn_decode_tma_ok(H, KV, hs, ps):
        pytest.skip("the TMA decode kernel does not take this layout")
    seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, ps, seed=5)
    items = torch.tensor([(s, s, 1, n - 1) for s, n in enumerate(lengths)], dtype=torch.int32, device=DEV)
    q = torch.stack([seqs[s][0][n - 1].reshape(-1) for s, n in enumerate(lengths)]).to(torch.bfloat16).to(DEV)
    outs = []
    for entries in (12, 65535, 70001):
        work = torch.tensor(o.split_work([-(-n // 64) for n in lengths], 9, entries, 32, 2), dtype=torch.int32, device=DEV)
        scratch = torch.zeros(o.attn_decode_tma_work_floats(entries, H, KV, hs), device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        outs.append(torch.full_like(q, float("nan")))
        o.attn_decode_tma(q, kc.to(DEV), vc.to(DEV), table.to(DEV), items, outs[-1], ps, len(lengths), H, KV, hs, hs ** -0.5, work=work,
                          scratch=scratch, status=status, max_rows=H // KV)
        assert status.item() == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and not torch.isnan(outs[0]).any()


@pytest.mark.parametrize("tma", [False, True], ids=["cp_async", "tma"])
def test_split_decode_shares_its_scratch_between_shapes(tma):
    """One scratch buffer serves launches with different numbers of items and splits, as the engine's does
    from step to step: a launch with many items and splits fills it with partial results, a launch with few
    follows and must find its tickets at zero all the same (they have a region of their own)."""
    o = ops()
    H, KV, hs, page_size = 16, 1, 64, 16                # 16 query heads per KV head: every row of a partial tile is written
    lengths = [300, 290, 280, 270, 260, 250]
    seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, page_size, seed=31)
    kcd, vcd, tb = kc.to(DEV), vc.to(DEV), table.to(DEV)
    floats = o.attn_decode_tma_scratch_floats if tma else o.attn_decode_scratch_floats
    decode = o.attn_decode_tma if tma else o.attn_decode
    scratch = torch.zeros(floats(len(lengths), H, KV, hs, 4), device=DEV)
    scale = 1.0 / math.sqrt(hs)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    full = [plain_llama.attention(q.double(), k.double(), v.double(), scale, None) for q, k, v in seqs]
    vmax = max(v.abs().max().item() for _, _, v in seqs)
    for which, nsplit in (([0, 1, 2, 3, 4, 5], 4), ([1], 2), ([0, 2, 4], 3), ([5], 4), ([0, 1, 2, 3, 4, 5], 2)):
        items = torch.tensor([(s, i, 1, lengths[s] - 1) for i, s in enumerate(which)], dtype=torch.int32, device=DEV)
        q = torch.stack([seqs[s][0][lengths[s] - 1].reshape(-1) for s in which]).to(torch.bfloat16).to(DEV)
        out = torch.full_like(q, float("nan"))
        decode(q, kcd, vcd, tb, items, out, page_size, len(lengths), H, KV, hs, scale, 0, nsplit=nsplit,
               scratch=scratch, status=status)
        want = torch.stack([full[s][lengths[s] - 1].reshape(-1) for s in which])
        assert status.item() == 0
        assert not torch.isnan(out).any(), (which, nsplit)
        assert (out.double().cpu() - want).abs().max().item() <= 2 ** -8 * vmax, (which, nsplit)


@pytest.mark.parametrize("batch,ctx,nsplit", [(8, 8192, 4), (64, 2048, 1), (1, 8192, 32)])
@pytest.mark.parametrize("tma", [False, True], ids=["cp_async", "tma"])
def test_attention_decode_at_serving_size(batch, ctx, nsplit, tma):
    """Decode rows at the Llama-3.1-8B head layout over long contexts (a cache larger than L2):
    the tensor-core kernel against the plain kernel, and its achieved bandwidth (printed)."""
    o = ops()
    H, KV, hs, page_size = 32, 8, 128, 16
    g = torch.Generator(device=DEV).manual_seed(11)
    blocks = -(-ctx // page_size)
    num_pages = batch * blocks
    kc = torch.randn(num_pages, KV, page_size, hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    vc = torch.randn(num_pages, KV, page_size, hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    table = torch.randperm(num_pages, generator=g, device=DEV).to(torch.int32).view(batch, blocks)
    q = torch.randn(batch, H * hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    lens = [ctx - 3 * i for i in range(batch)]
    items = torch.tensor([(s, s, 1, lens[s] - 1) for s in range(batch)], dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    rseq = torch.arange(batch, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    want = torch.empty_like(q)
    o.paged_attention_ref(q, kc, vc, table, rseq, pos, want, page_size, batch, H, KV, hs, scale, 0, status)
    out = torch.empty_like(q)
    floats = o.attn_decode_tma_scratch_floats if tma else o.attn_decode_scratch_floats
    scratch = torch.zeros(max(1, floats(batch, H, KV, hs, nsplit)), device=DEV)
    decode = o.attn_decode_tma if tma else o.attn_decode
    more = {"max_rows": H // KV} if tma else {}
    run = lambda: decode(q, kc, vc, table, items, out, page_size, batch, H, KV, hs, scale, 0,
                         nsplit=nsplit, scratch=scratch if nsplit > 1 else None, status=status, **more)
    run()
    assert status.item() == 0
    assert (out.float() - want.float()).abs().max().item() <= 2 ** -8 * 4       # outputs of size up to ~4 in bf16
    # and against torch alone, so that the yardstick is not a kernel of the package: the first, a middle and the last row
    for s_ in sorted({0, batch // 2, batch - 1}):
        ref = _torch_attention(q[s_], kc, vc, table[s_], lens[s_] - 1, H, KV, hs, scale)
        assert (out[s_].float() - ref).abs().max().item() <= 2 ** -8 * 4, f"sequence {s_} against torch"
    for _ in range(3):
        run()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    a.record()
    for _ in range(10):
        run()
    b.record()
    torch.cuda.synchronize()
    us = a.elapsed_time(b) * 100
    gbs = sum(lens) * KV * hs * 2 * 2 / (us * 1e-6) / 1e9
    print(f"attn_decode {'tma' if tma else 'cp.async'} batch {batch} ctx {ctx} nsplit {nsplit}: {us:.1f} us, "
          f"{gbs:.0f} GB/s of cache read")


@pytest.mark.parametrize("lens", [[8192] * 8, [8192] + [512] * 7, [8192, 4096, 2048, 1024, 512, 256, 128, 64],
                                  [8192] + [256] * 63, [8192] * 40], ids=["even", "one_long", "halving", "one_long_of_64", "forty"])
def test_attention_decode_shares_at_serving_size(lens):
    """Sequences of unequal length at the Llama-3.1-8B head layout: shares of equal length (``split_work``)
    against the same number of splits for every sequence; the same outputs, and the time of both (printed)."""
    o = ops()
    H, KV, hs, page_size = 32, 8, 128, 16
    batch = len(lens)
    g = torch.Generator(device=DEV).manual_seed(11)
    blocks = [-(-n // page_size) for n in lens]
    num_pages = sum(blocks)
    kc = torch.randn(num_pages, KV, page_size, hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    vc = torch.randn(num_pages, KV, page_size, hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    perm = torch.randperm(num_pages, generator=g, device=DEV).to(torch.int32)
    table = torch.full((batch, max(blocks)), -1, dtype=torch.int32, device=DEV)
    at = 0
    for s_, nb in enumerate(blocks):
        table[s_, :nb] = perm[at:at + nb]
        at += nb
    q = torch.randn(batch, H * hs, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)
    items = torch.tensor([(s_, s_, 1, n - 1) for s_, n in enumerate(lens)], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    nsplit = max(1, min(32, 296 // (batch * KV)))
    scratch = torch.zeros(max(1, o.attn_decode_tma_scratch_floats(batch, H, KV, hs, nsplit)), device=DEV)
    entries = 296 // KV + 4 * batch
    work = torch.tensor(o.split_work([-(-n // 64) for n in lens], 296 // KV, entries, 32, 2), dtype=torch.int32, device=DEV)
    scratch2 = torch.zeros(o.attn_decode_tma_work_floats(entries, H, KV, hs), device=DEV)
    outs, times = [], []
    for kw in ({"nsplit": nsplit, "scratch": scratch if nsplit > 1 else None}, {"work": work, "scratch": scratch2}):
        out = torch.empty_like(q)
        run = lambda: o.attn_decode_tma(q, kc, vc, table, items, out, page_size, batch, H, KV, hs, scale, 0,
                                        status=status, max_rows=H // KV, **kw)
        for _ in range(3):
            run()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            run()
        b.record()
        torch.cuda.synchronize()
        outs.append(out)
        times.append(a.elapsed_time(b) * 100)
    assert status.item() == 0
    assert (outs[0].float() - outs[1].float()).abs().max().item() <= 2 ** -8 * 4
    mb = sum(lens) * KV * hs * 2 * 2 / 1e6
    print(f"attn_decode tma {batch} sequences, {sum(lens)} tokens ({mb:.0f} MB): {nsplit} splits each {times[0]:.1f} us, "
          f"shares of equal length {times[1]:.1f} us ({mb / times[1]:.2f} TB/s)")


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(1, 1000, 96), (3, 513, 320), (8, 200, 1336), (16, 64, 16), (9, 37, 8), (5, 4096, 4096)])
def test_gemm_skinny(M, N, K, out_dtype):
    g = torch.Generator().manual_seed(12)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, K, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    ops().gemm_skinny(a, w, out)
    want = a.double() @ w.double().T
    tol = 1e-4 * math.sqrt(K) if out_dtype == torch.float32 else 2 ** -8 * want.abs().max().item()
    assert (out.double() - want).abs().max().item() <= tol
    # a row does not depend on the rows beside it; a strided view of x works
    wide = torch.zeros(M, K + 24, dtype=torch.bfloat16, device=DEV)
    wide[:, :K] = a
    one = torch.empty(1, N, dtype=out_dtype, device=DEV)
    ops().gemm_skinny(wide[M - 1:M, :K], w, one)
    assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("M,H,KV,hs,K,page_size", [(1, 4, 2, 64, 256, 16), (8, 32, 8, 128, 4096, 16), (16, 3, 1, 32, 96, 8),
                                                   (11, 6, 3, 16, 136, 4), (5, 2, 2, 96, 320, 32),
                                                   (4, 59, 8, 128, 264, 16), (10, 64, 6, 128, 2048, 16),         # tiles in turn
                                                   (3, 10, 4, 128, 2120, 16), (14, 12, 3, 128, 4104, 8)])        # sixteen warps a tile
def test_gemm_skinny_qkv_rope(M, H, KV, hs, K, page_size):
    """The q/k/v product with the rotation and the cache store in its epilogue against the three kernels it
    stands for (product, then rotation and store): rotated q, and the pages of k and v, a padding row included."""
    g = torch.Generator(device=DEV).manual_seed(31)
    o = ops()
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((H + 2 * KV) * hs, K, generator=g, device=DEV) / K ** 0.5).to(torch.bfloat16)
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, hs, 2, dtype=torch.float64) / hs))).float().to(DEV)
    num_seqs, width = M, 6
    num_pages = num_seqs * width + 3
    table = torch.randperm(num_pages, generator=g, device=DEV)[:num_seqs * width].to(torch.int32).view(num_seqs, width)
    positions = torch.randint(0, width * page_size, (M,), generator=g, device=DEV).to(torch.int32)
    row_seq = torch.arange(M, dtype=torch.int32, device=DEV)
    if M > 2:
        row_seq[M - 2] = -1                       # a padding row of a fixed-shape step: nothing stored for it
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    caches = []
    outs = []
    for fused in (False, True):
        kc = torch.zeros(num_pages, KV, page_size, hs, dtype=torch.bfloat16, device=DEV)
        vc = torch.zeros_like(kc)
        qkv = torch.zeros(M, (H + 2 * KV) * hs, dtype=torch.bfloat16, device=DEV)
        if fused:
            o.gemm_skinny_qkv_rope(x, w, qkv, positions, row_seq, inv_freq, table, kc, vc, page_size, num_seqs, H, KV, hs, status)
        else:
            o.gemm_skinny(x, w, qkv)
            o.rope_kv_write(qkv, positions, row_seq, inv_freq, hs, table, kc, vc, page_size, num_seqs, H, KV, hs, status)
        assert status.item() == 0
        outs.append(qkv[:, :H * hs].float())
        caches.append((kc.float(), vc.float()))
    # the same roundings in the same places; a product and a sum may be contracted differently: one bf16 step
    step = 2 ** -7
    assert (outs[0] - outs[1]).abs().max().item() <= step * max(1.0, outs[0].abs().max().item())
    assert (caches[0][0] - caches[1][0]).abs().max().item() <= step * max(1.0, caches[0][0].abs().max().item())
    assert torch.equal(caches[0][1], caches[1][1]), "v is stored as the product gave it"
    assert caches[1][0].abs().sum().item() > 0 and caches[1][1].abs().sum().item() > 0
    # against torch alone: one row's rotated first q head
    m = 0
    q0 = (x[m].double() @ w[:hs].double().T).to(torch.bfloat16).double()
    ang = positions[m].item() * inv_freq.double().cpu()
    c, sn = torch.cos(ang).to(DEV), torch.sin(ang).to(DEV)
    want = torch.cat([q0[:hs // 2] * c - q0[hs // 2:] * sn, q0[hs // 2:] * c + q0[:hs // 2] * sn])
    assert (outs[1][m, :hs].double() - want).abs().max().item() <= 2 ** -7 * max(1.0, want.abs().max().item())
    # a table entry outside the pool is reported, nothing is written for that row
    bad = table.clone()
    bad[0] = num_pages + 5
    kc = torch.zeros(num_pages, KV, page_size, hs, dtype=torch.bfloat16, device=DEV)
    o.gemm_skinny_qkv_rope(x[:1], w, torch.zeros(1, (H + 2 * KV) * hs, dtype=torch.bfloat16, device=DEV), positions[:1],
                           row_seq[:1], inv_freq, bad, kc, torch.zeros_like(kc), page_size, num_seqs, H, KV, hs, status)
    assert status.item() == 2 and kc.abs().sum().item() == 0


def test_gemm_skinny_at_serving_size():
    """The four projections of the Llama-3.1-8B block at 8 rows: achieved weight bandwidth (printed)
    beside the library product."""
    g = torch.Generator(device=DEV).manual_seed(13)
    for name, N, K in (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336)):
        a = torch.randn(8, K, generator=g, device=DEV).to(torch.bfloat16)
        # several copies of the weight so that consecutive runs do not find it in L2
        ws = [(0.02 * torch.randn(N, K, generator=g, device=DEV)).to(torch.bfloat16) for _ in range(4)]
        out = torch.empty(8, N, dtype=torch.bfloat16, device=DEV)
        res = {}
        for label, fn in (("skinny", lambda w: ops().gemm_skinny(a, w, out)), ("library", lambda w: torch.mm(a, w.t(), out=out))):
            for w in ws:
                fn(w)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()           # replayed from a graph: the host's launch cost stays out
            with torch.cuda.graph(graph):
                for _ in range(5):
                    for w in ws:
                        fn(w)
            graph.replay()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            graph.replay()
            e1.record()
            torch.cuda.synchronize()
            res[label] = e0.elapsed_time(e1) * 1e3 / 20
        want = a.double() @ ws[-1].double().T
        ops().gemm_skinny(a, ws[-1], out)
        assert (out.double() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
        mb = N * K * 2 / 1e6
        print(f"{name}: skinny {res['skinny']:.1f} us ({mb / res['skinny']:.2f} TB/s), "
              f"library {res['library']:.1f} us ({mb / res['library']:.2f} TB/s)")


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 128, 256), (256, 384, 512), (200, 1000, 320), (33, 96, 1336),
                                   (1, 128, 64), (2048, 512, 4096)])
def test_gemm_tc05(M, N, K, out_dtype):
    g = torch.Generator().manual_seed(14)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(N, K, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().gemm_tc05(a, w, out, status)
    torch.cuda.synchronize()
    assert status.item() == 0
    want = a.double() @ w.double().T
    tol = 1e-4 * math.sqrt(K) if out_dtype == torch.float32 else 2 ** -8 * want.abs().max().item()
    assert not torch.isnan(out).any()
    assert (out.double() - want).abs().max().item() <= tol


@pytest.mark.parametrize("M,F,K", [(128, 128, 64), (200, 1336, 320), (2048, 512, 4096), (77, 40, 72)])
def test_gemm_tc05_swiglu(M, F, K):
    """The many-row gate/up product with the activation in its epilogue equals the product stored in bf16
    followed by the activation kernel."""
    g = torch.Generator().manual_seed(24)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * F, K, generator=g) / math.sqrt(K)).to(torch.bfloat16).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops().gemm_tc05_swiglu(a, w, out, status)
    gu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device=DEV)
    ops().gemm_tc05(a, w, gu, status)
    two = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    ops().swiglu(gu, two, 8)
    assert status.item() == 0
    assert torch.equal(out, two)
    ref = (a.double() @ w.double().T).view(M, F // 8, 2, 8)
    want = plain_llama.swiglu(ref[:, :, 0].reshape(M, F).cpu(), ref[:, :, 1].reshape(M, F).cpu())
    assert (out.double().cpu() - want).abs().max().item() <= 2 ** -7 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(17, 128, 64), (1, 1000, 96), (33, 513, 320), (64, 200, 1336), (128, 384, 4096), (100, 6144, 512),
                                   (16, 64, 16), (127, 37, 8), (48, 4096, 4096), (5, 128256, 256)])
def test_gemm_rows(M, N, K, out_dtype):
    """The product for up to 128 rows: tiles shared between blocks (their partial sums added by the tile's
    owner), tails in every dimension, and the same call twice (the flags are back at zero)."""
    g = torch.Generator(device=DEV).manual_seed(21)
    a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device=DEV).to(torch.bfloat16)
    want = a.double() @ w.double().T
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    tol = (2 ** -8 if out_dtype == torch.bfloat16 else 2e-6) * max(1.0, want.abs().max().item()) + 1e-5 * K ** 0.5
    for _ in range(2):
        out = torch.full((M, N), float("nan"), dtype=out_dtype, device=DEV)
        ops().gemm_rows(a, w, out, status)
        assert status.item() == 0
        assert not torch.isnan(out).any()
        assert (out.double() - want).abs().max().item() <= tol
    # a row's result does not depend on the other rows of the call
    if M > 1:
        alone = torch.empty(1, N, dtype=out_dtype, device=DEV)
        ops().gemm_rows(a[M // 2:M // 2 + 1], w, alone, status)
        assert torch.equal(alone[0], out[M // 2])


@pytest.mark.parametrize("M,F,K", [(17, 64, 96), (64, 1336, 320), (128, 520, 4096), (30, 40, 72), (100, 14336, 256)])
def test_gemm_rows_swiglu(M, F, K):
    g = torch.Generator(device=DEV).manual_seed(22)
    a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    gate = (0.3 * torch.randn(F, K, generator=g, device=DEV)).to(torch.bfloat16)
    up = (0.3 * torch.randn(F, K, generator=g, device=DEV)).to(torch.bfloat16)
    w = torch.stack([gate.view(F // 8, 8, K), up.view(F // 8, 8, K)], 1).reshape(2 * F, K).contiguous()
    gd = (a.double() @ gate.double().T).to(torch.bfloat16).double()
    ud = (a.double() @ up.double().T).to(torch.bfloat16).double()
    want = gd / (1 + torch.exp(-gd)) * ud
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops().gemm_rows_swiglu(a, w, out, status)
    assert status.item() == 0 and not torch.isnan(out).any()
    # gate and up are rounded to bf16 before the activation: a rounding that falls the other way moves the result by
    # one bf16 step of gate or up
    scale = max(1.0, want.abs().max().item())
    assert (out.double() - want).abs().max().item() <= 2 ** -6 * scale


def test_gemm_rows_at_serving_size():
    """The projections of the Llama-3.1-8B block and the output head at 8 to 128 rows: time from a CUDA graph and
    bandwidth of the weight stream (printed) beside the few-row kernel (up to 16 rows) and the library; the calls
    of a graph go round several copies of the weight, so that none finds its weight in L2."""
    g = torch.Generator(device=DEV).manual_seed(23)
    shapes = (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336), ("head", 128256, 4096))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for M in (8, 16, 32, 64, 128):
        for name, N, K in shapes:
            a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
            # copies of the weight, 300 MB of them: a call does not find its weight in L2 (126 MB) from the call before
            ws = [(0.02 * torch.randn(N, K, generator=g, device=DEV)).to(torch.bfloat16)
                  for _ in range(max(1, -(-300_000_000 // (N * K * 2))))]
            w = ws[-1]
            out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
            runs = {"rows": lambda i: ops().gemm_rows(a, ws[i % len(ws)], out, status),
                    "library": lambda i: torch.mm(a, ws[i % len(ws)].t(), out=out)}
            if M <= 16:
                runs["few-row"] = lambda i: ops().gemm_skinny(a, ws[i % len(ws)], out)
            res = {label: graph_time_us(fn) for label, fn in runs.items()}
            assert status.item() == 0
            out.fill_(float("nan"))
            ops().gemm_rows(a, w, out, status)
            want = a.double() @ w[:4096].double().T
            assert (out[:, :4096].double() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
            assert not torch.isnan(out).any()
            gb = N * K * 2 / 1e3
            print(f"{M:4d} rows {name:8s}: " + ", ".join(f"{k} {v:.1f} us ({gb / v:.0f} GB/s)" for k, v in res.items()))


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (200, 1000, 320), (300, 4096, 512), (129, 96, 1336), (2048, 520, 256)])
def test_gemm_tc05_add_into_the_residual_stream(M, N, K):
    """The product that adds itself into an fp32 tensor: equal, bit for bit, to storing the product in bf16 and
    adding that (what the norm kernel after it would do), with one CTA a tile and with pairs."""
    g = torch.Generator(device=DEV).manual_seed(41)
    a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=DEV) / K ** 0.5).to(torch.bfloat16)
    resid0 = torch.randn(M, N, generator=g, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    stored = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops().gemm_tc05(a, w, stored, status)
    want = resid0 + stored.float()
    got = resid0.clone()
    ops().gemm_tc05_add(a, w, got, status)
    assert status.item() == 0
    assert torch.equal(got, want)
    ref = resid0.double() + (a.double() @ w.double().T)
    assert (got.double() - ref).abs().max().item() <= 2 ** -8 * max(1.0, (a.double() @ w.double().T).abs().max().item())


def test_gemm_tc05_at_prefill_size():
    """The projections of the Llama-3.1-8B block at 2,048 rows: achieved TFLOP/s (printed) beside the library."""
    g = torch.Generator(device=DEV).manual_seed(15)
    M = 2048
    for name, N, K in (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336)):
        a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
        w = (0.02 * torch.randn(N, K, generator=g, device=DEV)).to(torch.bfloat16)
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        res = {}
        for label, fn in (("tcgen05", lambda: ops().gemm_tc05(a, w, out, status)), ("library", lambda: torch.mm(a, w.t(), out=out))):
            for _ in range(3):
                fn()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(10):
                fn()
            e1.record()
            torch.cuda.synchronize()
            res[label] = e0.elapsed_time(e1) * 100
        assert status.item() == 0
        out.fill_(float("nan"))
        ops().gemm_tc05(a, w, out, status)
        want = a.double() @ w.double().T                     # every element of every tile
        assert not torch.isnan(out).any()
        assert (out.double() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
        del want
        tf = 2.0 * M * N * K / 1e6
        print(f"{name}: tcgen05 {res['tcgen05']:.1f} us ({tf / res['tcgen05']:.0f} TFLOP/s), "
              f"library {res['library']:.1f} us ({tf / res['library']:.0f} TFLOP/s)")


def test_attention_portion_at_prefill_size():
    """A 2,048-token prompt at the Llama-3.1-8B head layout: both portion kernels against the plain
    kernel on sampled rows, and their times (printed)."""
    o = ops()
    H, KV, hs, page_size, T = 32, 8, 128, 16, 2048
    g = torch.Generator(device=DEV).manual_seed(16)
    blocks = T // page_size
    kc = torch.randn(blocks + 5, KV, page_size, hs, generator=g, device=DEV).to(torch.bfloat16)
    vc = torch.randn(blocks + 5, KV, page_size, hs, generator=g, device=DEV).to(torch.bfloat16)
    table = torch.randperm(blocks + 5, generator=g, device=DEV)[:blocks].to(torch.int32).view(1, blocks)
    q = torch.randn(T, H * hs, generator=g, device=DEV).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    rows = torch.tensor([0, 1, 15, 16, 127, 128, 129, 1000, 2046, 2047], device=DEV)
    want = torch.empty(len(rows), H * hs, dtype=torch.bfloat16, device=DEV)
    o.paged_attention_ref(q[rows], kc, vc, table, torch.zeros(len(rows), dtype=torch.int32, device=DEV),
                          rows.to(torch.int32), want, page_size, 1, H, KV, hs, scale, 0, status)
    for label, fn, tok in (("mma.sync", o.attn_portion, o.attn_portion_tokens(H, KV, hs)),
                           ("tcgen05", o.attn_portion_tc05, o.attn_portion_tc05_tokens(H, KV))):
        items = torch.tensor([(0, b, min(tok, T - b), b) for b in range(0, T, tok)], dtype=torch.int32, device=DEV)
        out = torch.full_like(q, float("nan"))
        run = lambda: fn(q, kc, vc, table, items, out, page_size, 1, H, KV, hs, scale, 0, status=status)
        run()
        assert status.item() == 0 and not torch.isnan(out).any()
        assert (out[rows].float() - want.float()).abs().max().item() <= 2 ** -8 * 4
        for r in rows.tolist():                            # and against torch alone
            ref = _torch_attention(q[r], kc, vc, table[0], r, H, KV, hs, scale)
            assert (out[r].float() - ref).abs().max().item() <= 2 ** -8 * 4, f"{label}: row {r} against torch"
        for _ in range(2):
            run()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(10):
            run()
        e1.record()
        torch.cuda.synchronize()
        us = e0.elapsed_time(e1) * 100
        flops = 4.0 * H * hs * T * (T + 1) / 2
        print(f"attn_portion {label}: {us:.1f} us, {flops / us / 1e6:.0f} TFLOP/s (causal)")


def test_attention_portion_at_the_end_of_a_long_context():
    """The last 2,048 tokens of a 16,384-token prompt at the Llama-3.1-8B head layout (what a prompt cut into
    portions asks of the kernel): sampled rows against torch, and the time (printed). Nearly every key tile lies
    before the diagonal here, so the figure is the kernel's steady rate, without the causal edge."""
    o = ops()
    H, KV, hs, page_size, T, C = 32, 8, 128, 16, 2048, 16384
    if not o.attn_portion_tc05_ok(H, KV, hs, page_size):
        pytest.skip("the tcgen05 kernel does not take this layout")
    g = torch.Generator(device=DEV).manual_seed(61)
    blocks = C // page_size
    kc = torch.randn(blocks + 7, KV, page_size, hs, generator=g, device=DEV).to(torch.bfloat16)
    vc = torch.randn(blocks + 7, KV, page_size, hs, generator=g, device=DEV).to(torch.bfloat16)
    table = torch.randperm(blocks + 7, generator=g, device=DEV)[:blocks].to(torch.int32).view(1, blocks)
    q = torch.randn(T, H * hs, generator=g, device=DEV).to(torch.bfloat16)
    q[777] *= 6.0                                           # one row whose softmax is sharp: a far key must be found
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1.0 / math.sqrt(hs)
    tok = o.attn_portion_tc05_tokens(H, KV)
    items = torch.tensor([(0, b, min(tok, T - b), C - T + b) for b in range(0, T, tok)], dtype=torch.int32, device=DEV)
    out = torch.full_like(q, float("nan"))
    run = lambda: o.attn_portion_tc05(q, kc, vc, table, items, out, page_size, 1, H, KV, hs, scale, 0, status=status)
    run()
    assert status.item() == 0 and not torch.isnan(out).any()
    for r in (0, 1, 63, 64, 777, 1024, 2046, 2047):
        ref = _torch_attention(q[r], kc, vc, table[0], C - T + r, H, KV, hs, scale)
        assert (out[r].float() - ref).abs().max().item() <= 2 ** -8 * 4, f"row {r} against torch"
    us = graph_time_us(lambda i: run(), n=5)
    flops = 4.0 * H * hs * sum(C - T + r + 1 for r in range(T))
    print(f"attn_portion tcgen05, 2,048 tokens ending at {C}: {us:.1f} us, {flops / us / 1e6:.0f} TFLOP/s")


# ---- random searches over sizes ---------------------------------------------------------------------------------

def _swiglu_of_interleaved(y, F):
    """silu(gate) * up of a product whose columns hold 8 gates, their 8 ups, 8 gates, ... (both rounded to bf16)."""
    y = y.to(torch.bfloat16).double().view(y.shape[0], F // 8, 2, 8)
    gate, up = y[:, :, 0], y[:, :, 1]
    return (gate / (1 + torch.exp(-gate)) * up).reshape(y.shape[0], F)


def test_matrix_products_at_random_sizes():
    """Every matrix-product kernel of the package (few rows, up to 128 rows, many rows; plain, with the gated
    activation, into the residual stream) at 400 random sizes and row strides against a float64 product."""
    import random
    o = ops()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for seed in range(400):
        rng = random.Random(seed)
        g = torch.Generator(device=DEV).manual_seed(seed)
        kind = rng.choice(["skinny", "skinny_swiglu", "tc05", "tc05", "tc05_swiglu", "tc05_add", "rows", "rows_swiglu"])
        K = 8 * rng.choice([1, 2, 5, 8, 12, 33, 64, 100, 167, 512, 1792])
        M = (rng.randint(1, 16) if kind.startswith("skinny") else rng.randint(1, 128) if kind.startswith("rows")
             else rng.choice([1, 17, 100, 127, 128, 129, 200, 255, 256, 257, 300, 511, 513, 700, 1025]))
        N = rng.choice([8, 16, 40, 96, 128, 136, 256, 264, 520, 1000, 1024, 2056, 4096 + 8 * rng.randint(0, 40)])
        if "swiglu" in kind:
            N = 2 * (N // 2 // 8 * 8 or 8)
        ldx, ldw = K + 8 * rng.choice([0, 0, 1, 3]), K + 8 * rng.choice([0, 0, 2])
        x = torch.randn(M, ldx, generator=g, device=DEV).to(torch.bfloat16)[:, :K]
        w = (torch.randn(N, ldw, generator=g, device=DEV) / K ** 0.5).to(torch.bfloat16)[:, :K]
        want = x.double() @ w.double().T
        what = f"seed {seed}: {kind}, {M} x {N} x {K}, row strides {ldx} and {ldw}"
        if kind in ("skinny", "tc05", "rows"):
            odt = rng.choice([torch.bfloat16, torch.float32])
            out = torch.full((M, N), float("nan"), dtype=odt, device=DEV)
            {"skinny": lambda: o.gemm_skinny(x, w, out), "tc05": lambda: o.gemm_tc05(x, w, out, status),
             "rows": lambda: o.gemm_rows(x, w, out, status)}[kind]()
            tol = 2 ** -8 * max(1.0, want.abs().max().item()) if odt == torch.bfloat16 else 1e-3
            err = (out.double() - want).abs().max().item()
        elif kind == "tc05_add":
            resid = torch.randn(M, N, generator=g, device=DEV)
            before = resid.clone()
            o.gemm_tc05_add(x, w, resid, status)
            err = (resid.double() - (before.double() + want.to(torch.bfloat16).double())).abs().max().item()
            tol = 2 ** -7 * max(1.0, want.abs().max().item())
        else:
            F = N // 2
            out = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=DEV)
            {"skinny_swiglu": lambda: o.gemm_skinny_swiglu(x, w, out), "tc05_swiglu": lambda: o.gemm_tc05_swiglu(x, w, out, status),
             "rows_swiglu": lambda: o.gemm_rows_swiglu(x, w, out, status)}[kind]()
            ref = _swiglu_of_interleaved(want, F)
            err = (out.double() - ref).abs().max().item()
            tol = 2 ** -6 * max(1.0, ref.abs().max().item())
        assert err <= tol and status.item() == 0, f"{what}: off by {err:.3e} (allowed {tol:.3e}), status {status.item()}"


def test_attention_kernels_at_random_layouts():
    """The tensor-core attention kernels at 250 random layouts (head sizes, heads, groups, page sizes, windows),
    lengths around the edges of pages and tiles, tails from one decode row to whole prompts, and numbers of
    splits, against the plain attention. Layouts that a kernel declines by contract are passed over."""
    import random
    ran = 0
    for seed in range(250):
        rng = random.Random(seed)
        hs = rng.choice([16, 32, 48, 64, 64, 64, 80, 96, 128, 128, 128, 256])
        KV, G = rng.choice([1, 2, 3, 8]), rng.choice([1, 2, 3, 4, 5, 8, 16, 32])
        if KV * G > 40:
            G = rng.choice([1, 2, 4])
        H, page = KV * G, rng.choice([4, 8, 16, 32, 64])
        window = rng.choice([None, None, 5, 64, 65, 130])
        S = rng.randint(1, 6)
        lengths = [rng.choice([1, 2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 200, 333, 512, 640]) for _ in range(S)]
        tails = [rng.choice([1, 1, 1, 2, 3, 8, 40, 64, 128, 10 ** 6]) for _ in range(S)]
        mode = rng.choice(["cp_async", "tma", "tcgen05"])
        nsplit = 1 if mode == "tcgen05" else rng.choice([1, 1, 2, 3, 5, 8])
        what = (f"seed {seed}: {mode}, {H} heads, {KV} groups, head size {hs}, page {page}, window {window}, "
                f"lengths {lengths}, tails {tails}, {nsplit} splits")
        seqs, table, kc, vc = build_cache(torch.bfloat16, lengths, H, KV, hs, page, seed=seed)
        try:
            out, rows, _, _ = _run_tc_attention(seqs, table, kc, vc, lengths, tails, H, KV, hs, page, window, nsplit,
                                                mode != "cp_async", mode == "tcgen05")
        except pytest.skip.Exception:
            continue
        except ops().KernelError as e:
            assert "do not fit" in str(e) or "outside what the kernel supports" in str(e), f"{what}: {e}"
            continue
        ran += 1
        scale = 1.0 / math.sqrt(hs)
        full = [plain_llama.attention(q.double(), k.double(), v.double(), scale, window) for q, k, v in seqs]
        want = torch.stack([full[s][p].reshape(-1) for s, p in rows])
        vmax = max(v.abs().max().item() for _, _, v in seqs)
        assert not torch.isnan(out).any(), f"{what}: a row was not written"
        err = (out - want).abs().max().item()
        assert err <= 2 ** -8 * vmax, f"{what}: off by {err:.3e}"
    assert ran >= 100


def test_sampling_at_random_rows():
    """The sampling kernel against the plain sampler over 300 random batches: vocabularies from 2 to 4,099,
    temperatures, top-k from 1 to beyond the vocabulary, top-p down to 0.0001, ties, many equal logits (both
    zeros among them), rows half masked with -inf, flat rows."""
    import random
    for seed in range(300):
        rng = random.Random(seed)
        g = torch.Generator().manual_seed(seed)
        V, R = rng.choice([2, 3, 31, 32, 33, 130, 1000, 1024, 4099]), rng.randint(1, 9)
        scale = rng.choice([0.01, 1.0, 2.5, 30.0])
        logits = (scale * torch.randn(R, V, generator=g)).float()
        kind = rng.choice(["plain", "ties", "rounded", "masked", "flat"])
        if kind == "ties":
            for r in range(R):
                logits[r, torch.randint(0, V, (min(V, 5),), generator=g)] = logits[r].max() + rng.choice([0.0, 1.0])
        elif kind == "rounded":
            logits = (logits * 2).round() / 2
        elif kind == "masked":
            mask = torch.rand(R, V, generator=g) < 0.5
            mask[:, 0] = False
            logits[mask] = float("-inf")
        elif kind == "flat":
            logits[:] = 1.25
        temps = [rng.choice([0.0, 0.3, 0.7, 1.0, 1.5]) for _ in range(R)]
        ks = [rng.choice([0, 1, 2, 5, 50, V, V + 5]) for _ in range(R)]
        ps = [rng.choice([1.0, 0.99, 0.9, 0.5, 0.1, 0.0001]) for _ in range(R)]
        seeds, ctrs = [rng.randrange(2 ** 31) for _ in range(R)], [rng.randrange(1000) for _ in range(R)]
        out = torch.empty(R, dtype=torch.int32, device=DEV)
        ops().sample(logits.to(DEV), out, temperature=torch.tensor(temps, device=DEV),
                     top_k=torch.tensor(ks, dtype=torch.int32, device=DEV), top_p=torch.tensor(ps, device=DEV),
                     seed=torch.tensor(seeds, dtype=torch.int64, device=DEV), counter=torch.tensor(ctrs, dtype=torch.int64, device=DEV))
        want = [plain_llama.sample(logits[r], temps[r], ks[r], ps[r], seed=seeds[r], counter=ctrs[r]) for r in range(R)]
        got = out.tolist()
        for r in range(R):
            if got[r] == want[r]:
                continue
            # a draw that lands within rounding of a boundary between two kept tokens may fall either way (the
            # kernel sums in float32, the plain sampler in float64): both must then be kept tokens of equal
            # or neighbouring cumulative mass; anything else is a fault
            assert temps[r] > 0 and logits[r, got[r]] > float("-inf"), (
                f"seed {seed}, {kind}, row {r}: kernel {got[r]}, plain {want[r]} (T {temps[r]}, k {ks[r]}, p {ps[r]})")
            p = torch.softmax(logits[r].double() / temps[r], 0)
            lo, hi = sorted((got[r], want[r]))
            between = p[lo:hi + 1].sum().item() - max(p[lo].item(), p[hi].item())
            assert between <= 1e-5, (
                f"seed {seed}, {kind}, row {r}: kernel {got[r]}, plain {want[r]} with mass {between:.2e} between them")


@pytest.mark.parametrize("V", [1, 3, 4095, 4097, 16388, 32769, 65537, 131075, 262144, 262180])
def test_sampling_over_cluster_sizes(V):
    """Vocabularies around every border of the sampling kernel's layout (one block, a cluster, the groups a thread holds, rows
    read again beyond what a cluster holds), rows at odd strides, top-k and top-p on and off, masked (-inf) logits, greedy rows
    among the others. The kernel sums in float32 (relative error below 1e-5 for these sizes), the plain sampler in float64: where
    they differ, the plain draw's mass position must lie within 1e-5 of the border of the kernel's token."""
    g = torch.Generator().manual_seed(V)
    R = 5
    wide = (3.0 * torch.randn(R, V + 3, generator=g)).float()
    for off in (0, 3):                              # 3: the rows begin off a 16-byte border
        logits = wide[:, off:off + V]
        if V > 8:
            logits[1, ::3] = -math.inf
            logits[2, V // 2] = 60.0
        dl = wide.to(DEV)[:, off:off + V]
        seed = torch.arange(R, dtype=torch.int64, device=DEV) * 977 + 13
        ctr = torch.arange(R, dtype=torch.int64, device=DEV)
        for temps, k, p in (([0.7, 1.0, 0.6, 0.0, 1.5], 0, 0.9), ([1.0] * 5, 40, 0.95), ([0.8] * 5, 0, 1.0)):
            out = torch.full((R,), -1, dtype=torch.int32, device=DEV)
            ops().sample(dl, out, temperature=torch.tensor(temps, device=DEV), top_k=torch.full((R,), k, dtype=torch.int32, device=DEV),
                         top_p=torch.full((R,), p, device=DEV), seed=seed, counter=ctr)
            for r in range(R):
                x, T, got = logits[r], temps[r], int(out[r])
                if not T > 0:
                    assert got == plain_llama.sample(x)
                    continue
                w = torch.exp((x - x.max()).double() / T)
                order = torch.sort(x, descending=True).values
                keep = x >= order[k - 1] if 0 < k < V else torch.ones(V, dtype=torch.bool)
                if p < 1.0:
                    ordered = torch.sort(torch.where(keep, x, torch.tensor(-math.inf)), descending=True).values
                    mass = torch.cumsum(torch.exp((ordered - x.max()).double() / T), 0)
                    at = min(int((mass < p * mass[-1]).sum()), V - 1)
                    keep &= x >= ordered[at]
                assert bool(keep[got]), (V, off, r)
                c = torch.cumsum(torch.where(keep, w, torch.zeros_like(w)), 0)
                u = plain_llama.uniform01(int(seed[r]), int(ctr[r])) * float(c[-1])
                slack = 1e-5 * float(c[-1])
                assert (float(c[got - 1]) if got else 0.0) - slack <= u < float(c[got]) + slack, (V, off, r, T, k, p)


@pytest.mark.parametrize("act", ["none", "relu2", "glu_limited"])
@pytest.mark.parametrize("T,top,E,N,K", [(1, 1, 3, 16, 8), (1, 2, 5, 40, 264), (5, 4, 4, 18, 1408), (8, 4, 9, 50, 2056), (16, 2, 40, 34, 520), (16, 2, 2, 64, 4096)])
def test_experts_weights_streamed_for_few_places(T, top, E, N, K, act):
    """The streaming grouped product at the edges of its tiles (columns and chunks of k that fill none, one to sixteen places an
    expert, experts without any, ids of identity experts): pairs without a plan against float64, and with a plan to the same
    bits. Sums of K products of bf16 numbers of size one in fp32: 1e-6 sqrt(K) of the sum, before the activation."""
    g = torch.Generator().manual_seed(T * 100 + E)
    a = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E + 1, generator=g)[:top] for _ in range(T)]).int()      # id E: an identity expert
    o, P, pair = ops(), T * top, act == "glu_limited"
    kw = {"limit": 0.7, "alpha": 1.5, "shift": 1.0} if pair else {}
    out = torch.full((P, N // 2 if pair else N), 7.0, device=DEV)
    assert o.moe_pairs_ok(a.to(DEV), w.to(DEV), w.to(DEV), T, top)
    o.moe_gemm_pairs(a.to(DEV), ids.to(DEV), w.to(DEV), out, True, act, **kw)
    own = torch.full_like(out, 7.0)                                # rows by pair instead of by row
    o.moe_gemm_pairs(a.repeat_interleave(top, 0).to(DEV), ids.to(DEV), w.to(DEV), own, False, act, **kw)
    assert torch.equal(own, out)
    planned = torch.full_like(out, 7.0)
    scratch = torch.zeros(o.moe_plan_ints(P, E + 1), dtype=torch.int32, device=DEV)
    offsets, row_of = torch.zeros(E + 2, dtype=torch.int32, device=DEV), torch.zeros(P, dtype=torch.int32, device=DEV)
    place_of = torch.zeros(T, top, dtype=torch.int32, device=DEV)
    o.moe_plan(ids.to(DEV), E + 1, scratch, offsets, row_of, place_of)
    o.moe_gemm_tiles(a.to(DEV), row_of, w.to(DEV), planned, offsets, act, **kw)
    for p, e in enumerate(ids.flatten().tolist()):
        if e == E:
            assert bool((out[p] == 7.0).all())
            continue
        z = a[p // top].double() @ w[e].double().t()
        if pair:
            gv, uv = z[0::2].clamp(max=0.7), z[1::2].clamp(-0.7, 0.7)
            z = gv * torch.sigmoid(1.5 * gv) * (uv + 1.0)
        elif act == "relu2":
            z = z.clamp(min=0) ** 2
        assert (out[p].cpu().double() - z).abs().max().item() <= 2e-6 * K ** 0.5 * max(1.0, z.abs().max().item())
        assert torch.equal(planned[place_of.view(-1)[p]], out[p])


@pytest.mark.parametrize("T,ids", [(2, [[0] * 16, [0] * 16]), (8, [[0, 0, 1, 0]] * 8), (3, [[1, 0, 1, 1, 1, 1]] * 3), (1, [[2] * 32]), (16, [[1, 1]] * 16)])
def test_pairs_that_name_an_expert_more_often_than_there_are_rows(T, ids):
    """Ids that no router makes, an expert named up to 32 times, against float64: more places than one tile has sums for. Sums of K products of
    bf16 numbers of size one in fp32, the weights divided by sqrt(K): 2e-6 sqrt(K)."""
    g = torch.Generator().manual_seed(T)
    o, E, N, K = ops(), 3, 40, 264
    a, w = torch.randn(T, K, generator=g).to(torch.bfloat16), (torch.randn(E, N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    ids = torch.tensor(ids, dtype=torch.int32)
    out = torch.full((ids.numel(), N), 7.0, device=DEV)
    o.moe_gemm_pairs(a.to(DEV), ids.to(DEV), w.to(DEV), out, True)
    want = torch.einsum("pk,pnk->pn", a.double().repeat_interleave(ids.shape[1], 0), w.double()[ids.flatten().long()])
    assert (out.cpu().double() - want).abs().max().item() <= 2e-6 * K ** 0.5 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("form", ["none", "relu2", "silu_glu", "glu_limited"])
@pytest.mark.parametrize("T,top,N,K,sN,sK", [(1, 1, 16, 8, 16, 8), (3, 2, 40, 264, 304, 520), (9, 2, 64, 520, 16, 2056), (16, 2, 48, 264, 1008, 264)])
def test_shared_product_beside_the_experts(T, top, N, K, sN, sK, form):
    """The shared matrix's blocks in the experts' launch, from fewer column tiles than the experts have to many more: the experts' results to
    the bit what they are alone, the shared ones what the few-row product gives (its warps may be four: sums in another order, so a sum may
    round to the neighbouring bf16 number, 2^-8, which the square of relu doubles and the last rounding adds to), and against float64: a sum
    is off by its rounding, 2^-8 of it, which the form multiplies by its slope (a tenth more for its curve), and the result is rounded so."""
    g = torch.Generator().manual_seed(T + sN)
    o, E = ops(), 4
    rand = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)                      # noqa: E731
    a, w = rand(T, K), rand(E, N, K) / K ** 0.5
    sa, sw = rand(T, sK), rand(sN, sK) / sK ** 0.5
    ids = torch.stack([torch.randperm(E + 1, generator=g)[:top] for _ in range(T)]).int().to(DEV)
    glu = form in ("silu_glu", "glu_limited")
    alone, out = (torch.full((T * top, N), 7.0, device=DEV) for _ in range(2))
    want, got = (torch.full((T, sN // 2 if glu else sN), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    bias = torch.randn(sN, generator=g).to(DEV) if form == "glu_limited" else None
    o.moe_gemm_pairs(a, ids, w, alone, True)
    o.moe_gemm_pairs(a, ids, w, out, True, shared={"a": sa, "w": sw, "out": got, "form": form, "bias": bias, "limit": 0.9, "alpha": 1.7})
    assert torch.equal(alone, out)
    if form == "none":
        o.gemm_skinny(sa, sw, want)
    elif form == "relu2":
        o.gemm_skinny_relu2(sa, sw, want)
    elif form == "silu_glu":
        o.gemm_skinny_swiglu(sa, sw, want)
    else:
        o.gemm_skinny_glu_limited(sa, sw, bias, want, 0.9, 1.7)
    d = (got.double() - want.double()).abs()
    assert bool((d <= 2 ** -6 * want.double().abs() + 2 ** -7).all())
    s = sa.double() @ sw.double().t()
    gate, up = s.view(T, -1, 2, 8).unbind(2) if glu else (s, s)
    gate, up = gate.reshape(T, -1), up.reshape(T, -1)
    if form == "none":
        exact, slope = s, s.abs()
    elif form == "relu2":
        exact, slope = s.clamp(min=0) ** 2, 2 * s.clamp(min=0) * s.abs()
    else:
        alpha, zg, zu = 1.0, gate, up
        if form == "glu_limited":
            b = bias.double().view(-1, 2, 8)
            alpha, zg, zu = 1.7, (gate + b[:, 0].reshape(-1)).clamp(max=0.9), (up + b[:, 1].reshape(-1)).clamp(-0.9, 0.9) + 1.0
        sig = torch.sigmoid(alpha * zg)
        exact = zg * sig * zu
        slope = (gate * zu).abs() * (sig * (1 + alpha * zg * (1 - sig))).abs() + (up * zg * sig).abs()
    assert bool(((got.double() - exact).abs() <= 2 ** -8 * (1.1 * slope + exact.abs()) + 1e-4).all())


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K,columns", [(129, 8, 72, 64), (203, 2048, 2048, 64), (256, 200, 64, 64), (257, 2312, 1096, 64), (300, 2400, 8, 128),
                                           (938, 2048, 136, 128), (513, 3000, 520, 128), (2048, 2048, 72, 256), (129, 9600, 200, 256)])
def test_pairs_tiles_of_fewer_columns(M, N, K, columns, out_dtype):
    """The pair kernel's tiles of 64, 128 and 256 columns, at remainders of rows, columns and k, against float64: K / 16 instructions that each
    add to a sum of at most some 6 in 32 bits, rounding by up to 2^-23 of it, and where the result is bf16 its rounding (2^-8 of it)."""
    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV), (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    assert ops().gemm_tc05_columns(M, N) == columns
    wide = torch.full((M, N + 8), 7.0, dtype=out_dtype, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops().gemm_tc05(x, w, wide[:, :N], status)
    assert int(status) == 0 and bool((wide[:, N:] == 7.0).all())
    err = (wide[:, :N].double() - x.double() @ w.double().t()).abs().max().item()
    assert err <= -(-K // 16) * 6 * 2 ** -23 + (6 * 2 ** -8 if out_dtype == torch.bfloat16 else 0.0)


@pytest.mark.parametrize("M,N,K", [(1, 48, 8), (3, 40, 264), (8, 96, 1408), (9, 64, 1416), (16, 128, 2816), (8, 64, 5632), (2, 5000, 768),
                                   (1, 9480, 8), (5, 9490, 2040), (8, 14300, 264), (9, 9490, 2056), (16, 9490, 72),      # tiles in turn
                                   (2, 40, 2056), (8, 2368, 2088), (12, 2360, 4104), (1, 2376, 2056)])                  # sixteen warps a tile, and one tile too many
def test_few_row_product_at_ragged_k(M, N, K):
    """The few-row product where k fills no whole round of a block's loads, against float64 (fp32 sums of K products)."""
    g = torch.Generator().manual_seed(K + M)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16), (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    out = torch.full((M, N), 7.0, device=DEV)
    ops().gemm_skinny(x.to(DEV), w.to(DEV), out)
    assert (out.cpu().double() - x.double() @ w.double().t()).abs().max().item() <= 1e-5


@pytest.mark.parametrize("H,KV,dk,dv,share,page,bias,cap,window,chunk,sink,n,pos0", [
    (8, 2, 128, 128, 1, 16, 40, 0.0, 0, 0, True, 150, 0),          # a bias by distance, its table shorter than the context
    (8, 2, 128, 128, 1, 8, 300, 0.0, 0, 0, False, 64, 203),        # a whole item behind a context
    (6, 2, 72, 40, 1, 16, 7, 0.0, 50, 0, True, 131, 77),           # heads that do not fill a tile, sizes below a half
    (3, 3, 64, 128, 1, 32, 33, 0.0, 0, 64, False, 300, 1),         # one head a key head, chunks
    (16, 8, 64, 128, 2, 16, 0, 30.0, 100, 0, False, 190, 30),      # a soft limit, key heads that share values, a window
    (8, 4, 128, 64, 4, 64, 0, 2.0, 0, 0, False, 129, 0),           # a limit that cuts (the quotient form)
    (8, 2, 128, 256, 2, 16, 0, 0.0, 0, 0, True, 140, 12),          # values in two blocks
    (4, 1, 40, 520, 1, 16, 0, 0.0, 33, 0, True, 70, 100),          # values in five, the last one narrow
    (4, 4, 192, 128, 1, 0, 0, 0.0, 0, 0, True, 300, 17),           # rows of matrices, keys of three halves
    (3, 3, 136, 72, 1, 0, 0, 0.0, 90, 0, False, 257, 40),          # the same at sizes that are no halves: boxes reach into the next head
    (4, 2, 192, 128, 1, 16, 0, 0.0, 0, 0, False, 70, 129),         # wide keys in pages
])
@pytest.mark.parametrize("f32", [False, True])
def test_portions_in_the_general_form_on_tcgen05(H, KV, dk, dv, share, page, bias, cap, window, chunk, sink, n, pos0, f32):
    """The tcgen05 prompt kernel's general form against float64 on the same bf16 inputs, two sequences a launch, pages scattered over
    a pool whose other pages hold numbers that would show. Probabilities meet the values as bf16 (2^-9 relative each) and results
    are stored in bf16 or fp32: 2^-7 of the largest value is allowed, the plain kernels' bound."""
    o = ops()
    assert o.attn_portion_gen_ok(H, KV, dk, dv, share, page, bias > 0, cap > 0)
    g = torch.Generator().manual_seed(H * 1000 + dk + n)
    KVv, scale, ends = KV // share, 2.0 * dk ** -0.5, [pos0 + n, pos0 + n + 35]
    starts = [pos0, pos0 + 35]
    ks = [torch.randn(e, KV, dk, generator=g).to(torch.bfloat16) for e in ends]
    vs = [torch.randn(e, KVv, dv, generator=g).to(torch.bfloat16) for e in ends]
    q = torch.randn(2 * n + 3, H * dk, generator=g).to(torch.bfloat16)
    rel = torch.randn(bias, H, generator=g) * 2 if bias else None
    sk = torch.randn(H, generator=g) * 2 if sink else None
    if page:
        need = [-(-e // page) for e in ends]
        pool = sum(need) + 3
        order = torch.randperm(pool, generator=g).tolist()
        kc = torch.full((pool, KV, page, dk), 50.0, dtype=torch.bfloat16)
        vc = torch.full((pool, KVv, page, dv), 50.0, dtype=torch.bfloat16)
        table = torch.full((2, max(need) + 2), -1, dtype=torch.int32)
        for s in range(2):
            first = max(0, starts[s] - window + 1) if window else (starts[s] // chunk * chunk if chunk else 0)
            for b in range(need[s]):
                pg = order.pop()
                a, e = b * page, min(ends[s], (b + 1) * page)
                kc[pg, :, :e - a], vc[pg, :, :e - a] = ks[s][a:e].transpose(0, 1), vs[s][a:e].transpose(0, 1)
                table[s, b] = -1 if e <= first else pg               # pages before every row's window have been given back
        k_in, v_in = kc.to(DEV), vc.to(DEV)
    else:
        k_in, v_in = torch.cat(ks).reshape(-1, KV * dk).to(DEV), torch.cat(vs).reshape(-1, KVv * dv).to(DEV)
        table = torch.tensor([[0], [ends[0]]], dtype=torch.int32)
    per, items = o.attn_portion_tc05_tokens(H, KV), []
    for s, row0 in ((0, 1), (1, n + 2)):
        items += [(s, row0 + b, min(per, n - b), starts[s] + b) for b in range(0, n, per)]
    items.sort(key=lambda it: it[2] + it[3])
    out = torch.full((2 * n + 3, H * dv), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.attn_portion_gen(q.to(DEV), k_in, v_in, table.to(DEV), torch.tensor(items, dtype=torch.int32, device=DEV), out, page, 2, H, KV, dk, dv, scale,
                       window, dist_bias=None if rel is None else rel.to(DEV), sink=None if sk is None else sk.to(DEV), status=status, softcap=cap,
                       v_share=share, chunk=chunk)
    assert status.item() == 0
    got = out.cpu().double()
    for s, row0 in ((0, 1), (1, n + 2)):
        i, j = torch.arange(starts[s], ends[s])[:, None], torch.arange(ends[s])[None, :]
        seen = j <= i
        if window:
            seen &= i - j < window
        if chunk:
            seen &= i // chunk == j // chunk
        for h in range(H):
            kh = h * KV // H
            z = q[row0:row0 + n, h * dk:(h + 1) * dk].double() @ ks[s][:, kh].double().t() * scale
            if cap:
                z = cap * torch.tanh(z / cap)
            if rel is not None:
                z = z + rel[:, h].double()[(i - j).clamp(0, bias - 1)]
            z = z.masked_fill(~seen, -math.inf)
            m = z.amax(-1, keepdim=True)
            den = torch.exp(z - m).sum(-1, keepdim=True) + (torch.exp(sk[h].double() - m) if sk is not None else 0.0)
            want = torch.exp(z - m) / den @ vs[s][:, kh // share].double()
            diff = (got[row0:row0 + n, h * dv:(h + 1) * dv] - want).abs().max().item()
            assert diff <= 2 ** -7 * vs[s].abs().max().item(), (s, h, diff)
    for r in (0, n + 1, 2 * n + 2):
        assert bool((got[r] == 7.0).all()), "rows of no item stay as they are"


@pytest.mark.parametrize("H,KV,hs,n,pos0,window,sink,blocks", [(6, 2, 128, 200, 5000, 0, True, 9), (8, 8, 64, 300, 4444, 0, False, 24), (4, 1, 96, 70, 6000, 4300, True, 9)])
def test_portions_whose_keys_are_cut_over_blocks(H, KV, hs, n, pos0, window, sink, blocks):
    """A long prompt's portion on the tcgen05 kernel with its items' keys cut into shares, against float64 (sampled rows) and against
    whole items: probabilities and results are bf16, so 2^-7 of the largest value either way. Rows whose window lies behind a share's
    keys get nothing from it."""
    o = ops()
    g = torch.Generator().manual_seed(n)
    end, page, G = pos0 + n, 16, H // KV
    need = -(-end // page)
    table = torch.randperm(need + 2, generator=g)[:need].int().view(1, -1)
    kc, vc = (torch.randn(need + 2, KV, page, hs, generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(n, H * hs, generator=g).to(torch.bfloat16)
    sk = torch.randn(H, generator=g).to(DEV) if sink else None
    per = o.attn_portion_tc05_tokens(H, KV)
    items = [(0, b, min(per, n - b), pos0 + b) for b in range(0, n, per)]
    first = lambda p: max(0, p - window + 1) // 128 * 128 if window else 0          # noqa: E731
    tiles = [-(-(p0 + m - first(p0)) // 128) for _, _, m, p0 in items]
    entries, cut, slots = o.cut_portions(tiles, KV, blocks)
    assert len(cut) and (entries[:, 2] > 1).any() and len({(e[0], e[1]) for e in entries.tolist()}) == len(entries)
    assert sorted(e[0] for e in entries.tolist() if e[1] == 0) == list(range(len(items))), "every item once"
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = []
    for shares in (None, (torch.tensor(entries, device=DEV), torch.tensor(cut, device=DEV), slots,
                          torch.full((o.attn_portion_share_floats(slots, KV, hs, hs),), float("nan"), device=DEV))):
        out = torch.full((n, H * hs), 7.0, dtype=torch.bfloat16, device=DEV)
        o.attn_portion_tc05(q.to(DEV), kc.to(DEV), vc.to(DEV), table.to(DEV), torch.tensor(items, dtype=torch.int32, device=DEV), out, page, 1, H, KV, hs,
                            1.5 * hs ** -0.5, window, status=status, sink=sk, vs=hs, shares=shares)
        outs.append(out.cpu().double())
    assert status.item() == 0
    k, v = (c[table[0].long()].transpose(0, 1).reshape(KV, -1, hs)[:, :end].double() for c in (kc, vc))
    bound = 2 ** -7 * v.abs().max().item()
    assert (outs[1] - outs[0]).abs().max().item() <= bound
    for r in (0, 1, n // 2, n - 1):
        lo = max(0, pos0 + r - window + 1) if window else 0
        for h in range(H):
            z = k[h // G, lo:pos0 + r + 1] @ q[r, h * hs:(h + 1) * hs].double() * 1.5 * hs ** -0.5
            e = torch.exp(z - z.max())
            den = e.sum() + (torch.exp(sk[h].cpu().double() - z.max()) if sink else 0.0)
            assert (outs[1][r, h * hs:(h + 1) * hs] - e @ v[h // G, lo:pos0 + r + 1] / den).abs().max().item() <= bound


@pytest.mark.parametrize("G,H,dk,dv", [(1, 2, 128, 128), (2, 2, 64, 40), (1, 3, 100, 12)])
def test_gated_delta_portions_in_groups_of_four(G, H, dk, dv):
    """The gated delta rule (one decay a head) by groups of four tokens against the token-by-token scan, both fp32: portions of 1 to 9
    rows beside each other, from position 0 and going on from a slot. Unit keys and decays below one keep the state of the values'
    size, so the two orders of the sums differ by some 1e-6 a token: 2e-5 of the largest value is allowed."""
    o = ops()
    assert o.channel_delta_groups_ok(dk, dv)
    g = torch.Generator().manual_seed(dk)
    lens, starts = [9, 1, 4, 7, 2], [0, 5, 0, 3, 11]
    T, S, C = sum(lens), len(lens), 2 * G * dk + H * dv
    xc = torch.randn(T, C, generator=g).to(DEV)
    u = torch.randn(T, 2 * H + 3, generator=g).to(DEV)
    a_log, dt_bias = torch.rand(H, generator=g).to(DEV), (torch.rand(H, generator=g) * 4 - 5).to(DEV)
    q_start = torch.tensor([sum(lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    ctx_len = torch.tensor([n + p for n, p in zip(lens, starts)], dtype=torch.int32, device=DEV)
    slots = torch.tensor([4, 0, 2, 1, 3], dtype=torch.int32, device=DEV)
    row_seq = torch.repeat_interleave(torch.arange(S), torch.tensor(lens)).int().to(DEV)
    bg = torch.empty(T, 2 * H + G, device=DEV)
    o.delta_prepare(xc, u, 0, H, a_log, dt_bias, bg, G, H, dk, dk ** -0.5)
    one = torch.zeros(S, H * o.delta_state_floats(dk, dv) + 8, device=DEV)
    seen, was = torch.randn(sum(starts), C, generator=g).to(DEV), torch.randn(sum(starts), 2 * H + 3, generator=g).to(DEV)
    before = torch.tensor([sum(starts[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    bg0 = torch.empty(sum(starts), 2 * H + G, device=DEV)
    o.delta_prepare(seen, was, 0, H, a_log, dt_bias, bg0, G, H, dk, dk ** -0.5)
    o.delta_scan(seen, bg0, one, torch.empty(sum(starts), H * dv, device=DEV), before, torch.tensor(starts, dtype=torch.int32, device=DEV), slots, S,
                 G, H, dk, dv)                                     # what the slots hold
    four = one.clone()
    y1, y4 = torch.empty(T, H * dv, device=DEV), torch.full((T, H * dv), 7.0, device=DEV)
    o.delta_scan(xc, bg, one, y1, q_start, ctx_len, slots, S, G, H, dk, dv)
    dec, rec, sc = torch.empty(T, H * dk, device=DEV), torch.empty(T, H, 3, dk, device=DEV), torch.empty(T, H, o.GROUP_SCALARS, device=DEV)
    o.channel_delta_groups(xc, u, 0, dec, a_log, dt_bias, rec, sc, row_seq, q_start, S, G, H, dk, a_off=H)
    o.channel_delta_group_scan(rec, sc, dec, xc, four, y4, q_start, ctx_len, slots, S, G, H, dk, dv)
    for a, b in ((y1, y4), (one, four)):
        assert bool(torch.isfinite(b).all()) and (a - b).abs().max().item() <= 2e-5 * a.abs().max().item()


@pytest.mark.parametrize("H,n", [(2, 64), (9, 36), (1, 44)])
def test_decaying_state_in_groups_of_four(H, n):
    """Time mixing's recurrence by groups of four tokens against the token-by-token scan, both fp32: portions of 1 to 9 rows beside each
    other, from position 0 and going on from a slot. Sums of n products in another order: 2e-5 of the largest value is allowed."""
    o = ops()
    assert o.decay_groups_ok(n)
    g = torch.Generator().manual_seed(n)
    lens, starts = [9, 1, 4, 7, 2], [0, 5, 0, 3, 11]
    T, S, C = sum(lens), len(lens), H * n
    xs = torch.randn(T, 4 * C, generator=g)
    xs[:, 3 * C:] = 1.0 - 0.3 * torch.rand(T, C, generator=g)
    xs = xs.to(DEV)
    u = torch.randn(H, n, generator=g).to(DEV)
    q_start = torch.tensor([sum(lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    ctx_len = torch.tensor([m + p for m, p in zip(lens, starts)], dtype=torch.int32, device=DEV)
    slots = torch.tensor([4, 0, 2, 1, 3], dtype=torch.int32, device=DEV)
    row_seq = torch.repeat_interleave(torch.arange(S), torch.tensor(lens)).int().to(DEV)
    width = H * o.decay_state_floats(n) + 8
    one = torch.zeros(S, width, device=DEV)
    seen = torch.randn(sum(starts), 4 * C, generator=g)
    seen[:, 3 * C:] = 0.9
    before = torch.tensor([sum(starts[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    y0 = torch.empty(sum(starts), C, device=DEV)
    o.decay_scan(seen.to(DEV), u, one, y0, before, torch.tensor(starts, dtype=torch.int32, device=DEV), slots, S, H, n)      # what the slots hold
    four = one.clone()
    y1, y4 = torch.empty(T, C, device=DEV), torch.full((T, C), 7.0, device=DEV)
    o.decay_scan(xs, u, one, y1, q_start, ctx_len, slots, S, H, n)
    o.decay_group_scan(xs.clone(), u, torch.empty(T, H, 4, device=DEV), four, y4, row_seq, q_start, ctx_len, slots, S, H, n)
    for a, b in ((y1, y4), (one, four)):
        assert bool(torch.isfinite(b).all()) and (a - b).abs().max().item() <= 2e-5 * a.abs().max().item()


@pytest.mark.parametrize("M,N,K", [(700, 1000, 96), (641, 961, 68), (705, 1001, 33)])
def test_gemm_f32_over_both_tiles(M, N, K):
    """Enough tiles of 64 x 64 for every SM, rows of 16-byte words and not: against float64 (K fp32 sums of products of size one), and a
    row by itself, which takes the smaller tiles, to the same bits."""
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    out, one = torch.empty(M, N, device=DEV), torch.empty(1, N, device=DEV)
    ops().gemm_f32(a, w, out)
    assert (out.double() - a.double() @ w.double().T).abs().max().item() <= 1e-6 * K * 4
    for m in (0, 63, M - 1):
        ops().gemm_f32(a[m:m + 1], w, one)
        assert torch.equal(one[0], out[m])


@pytest.mark.parametrize("heads,groups,N,P", [(4, 2, 128, 64), (3, 1, 64, 64), (2, 2, 100, 60), (64, 8, 128, 64)])
def test_state_space_portions_two_columns_a_thread(heads, groups, N, P):
    """A portion in one call (two columns a thread) and in pieces of three rows (one column): the same sums in the same order, so the
    same bits, in the results and in the slots; rows that fill no whole group of eight or chunk of 32, one sequence that continues."""
    o = ops()
    g = torch.Generator().manual_seed(N)
    lens = [37, 64, 1, 5, 0, 90]
    S, T, W = len(lens), sum(lens), heads * P + 2 * groups * N
    xbc, dt = torch.randn(T, W, generator=g).to(DEV), torch.randn(T, heads, generator=g).to(torch.bfloat16).to(DEV)
    dt_bias, a_log, skip = (torch.randn(heads, generator=g).to(DEV) for _ in range(3))
    start = torch.tensor([sum(lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    before = torch.tensor([0, 0, 7, 0, 0, 12], dtype=torch.int32, device=DEV)
    slots = torch.tensor([3, 0, 5, 1, 2, 4], dtype=torch.int32, device=DEV)
    whole = torch.randn(S, heads * o.ssm_padded_state(N, P) * P + 4, generator=g).to(DEV)
    parts = whole.clone()
    y, yp = torch.full((T, heads * P), 7.0, device=DEV), torch.full((T, heads * P), 7.0, device=DEV)
    ctx = before + torch.tensor(lens, dtype=torch.int32, device=DEV)
    o.ssm_scan(xbc, dt, dt_bias, a_log, skip, whole, y, start, ctx, slots, S, heads, groups, N, P)
    for s in range(S):
        for a in range(0, lens[s], 3):
            b = min(a + 3, lens[s])
            i0 = int(start[s])
            o.ssm_scan(xbc[i0 + a:i0 + b], dt[i0 + a:i0 + b], dt_bias, a_log, skip, parts, yp[i0 + a:i0 + b],
                       torch.tensor([0, b - a], dtype=torch.int32, device=DEV), before[s:s + 1] + b, slots[s:s + 1], 1, heads, groups, N, P)
    assert torch.isfinite(y).all() and torch.equal(y, yp) and torch.equal(whole, parts)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,K", [(12, 4), (2048, 4), (516, 1), (516, 3), (10, 4), (64, 7)])
def test_causal_convolution_of_portions_and_single_rows(C, K, dtype):
    """Portions, then single rows beside a padding row, then a step of two rows of one sequence and none of another: results and
    slots against float64 over the whole sequences (K fp32 products of size one; the channels that fill no fours and the longer taps
    take the plain kernel)."""
    o = ops()
    g = torch.Generator().manual_seed(C + K)
    S, off = 4, 8
    slots = [2, 0, 3, 1]
    w, b = torch.randn(C, K, generator=g), torch.randn(C, generator=g)
    seqs = [torch.randn(80, C, generator=g).to(dtype) for _ in range(S)]
    want = [torch.nn.functional.silu(torch.nn.functional.conv1d(torch.nn.functional.pad(q.double().t()[None], (K - 1, 0)), w.double()[:, None],
                                                                b.double(), groups=C))[0].t() for q in seqs]
    state = torch.full((S, off + (K - 1) * C + 4), float("nan"), device=DEV)         # what stale slots hold must not be read
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    done = [0] * S
    for lens, pad in (([1, 2, 17, 33], 0), ([30, 1, 1, 9], 0), ([1, 1, 1, 1], 0), ([1, 1, 1, 0], 1), ([2, 0, 1, 1], 0), ([20, 1, 1, 1], 0)):
        T = sum(lens) + pad
        rows = torch.full((T, C + 4), 3.0).to(dtype)
        seq, pos, at = [-1] * T, [0] * T, 0
        for s, n in enumerate(lens):
            rows[at:at + n, 4:] = seqs[s][done[s]:done[s] + n]
            seq[at:at + n], pos[at:at + n] = [s] * n, list(range(done[s], done[s] + n))
            at += n
        out = torch.full((T, C), 7.0, device=DEV)
        o.causal_conv(rows.to(DEV)[:, 4:], w.to(DEV), b.to(DEV), state, off, out, i32(pos), i32(seq), i32([sum(lens[:s]) for s in range(S + 1)]),
                      i32([done[s] + lens[s] for s in range(S)]), i32(slots), S, status=status)
        at = 0
        for s, n in enumerate(lens):
            if n:
                assert (out[at:at + n].double().cpu() - want[s][done[s]:done[s] + n]).abs().max().item() <= 1e-6 * K * 16
            at += n
            done[s] += n
            if lens[s]:
                kept = state[slots[s], off:off + (K - 1) * C].view(K - 1, C).cpu()
                past = torch.cat([torch.zeros(K - 1, C), seqs[s][:done[s]].float()])[len(seqs[s][:done[s]]):]
                assert torch.equal(kept, past[-(K - 1):] if K > 1 else past[:0])
        if pad:
            assert (out[-pad:] == 0).all()
    assert status.item() == 0


@pytest.mark.parametrize("H,KV,dk,dv,share,page,bias,cap", [
    (2, 2, 192, 128, 1, 0, 0, 0.0),          # rows of matrices: the next sequence's rows stand behind the last
    (2, 2, 136, 72, 1, 0, 0, 0.0),           # boxes wider than a head
    (4, 2, 64, 264, 2, 16, 0, 0.0),          # pages: what an earlier owner left in them, values in three blocks
    (4, 2, 128, 128, 1, 64, 9, 0.0),
    (4, 2, 64, 64, 1, 8, 0, 20.0),
])
@pytest.mark.parametrize("end", [1, 63, 130, 255, 300])
def test_portions_in_the_general_form_beside_numbers_that_are_not_finite(H, KV, dk, dv, share, page, bias, cap, end):
    """What lies behind a sequence's last key, in its last page or in the next sequence's rows, and what other key heads hold, reaches no
    result: the same bits with zeros and with NaN and infinities there."""
    o = ops()
    assert o.attn_portion_gen_ok(H, KV, dk, dv, share, page, bias > 0, cap > 0)
    g = torch.Generator().manual_seed(dk + end)
    KVv = KV // share
    rows = end + 200 if not page else -(-end // page) * page
    q = torch.randn(end, H * dk, generator=g).to(torch.bfloat16).to(DEV)
    k, v = torch.randn(rows, KV, dk, generator=g).to(torch.bfloat16), torch.randn(rows, KVv, dv, generator=g).to(torch.bfloat16)
    rel = torch.randn(bias, H, generator=g).to(DEV) if bias else None
    per = o.attn_portion_tc05_tokens(H, KV)
    items = torch.tensor([(0, b, min(per, end - b), b) for b in range(0, end, per)], dtype=torch.int32, device=DEV)
    G, got = H // KV, []
    for behind in (0.0, math.nan, math.inf):
        k[end:], v[end:] = behind, behind
        k[:, 1:] = behind                       # (queries of the first key head only are looked at; values stay where heads share them)
        if KVv > 1:
            v[:, 1:] = behind
        if page:
            def paged(t):
                return t.view(-1, page, *t.shape[1:]).transpose(1, 2).contiguous().to(DEV)
            k_in, v_in, table = paged(k), paged(v), torch.arange(rows // page, dtype=torch.int32, device=DEV).view(1, -1)
        else:
            k_in, v_in, table = k.reshape(rows, -1).to(DEV), v.reshape(rows, -1).to(DEV), torch.zeros(1, 1, dtype=torch.int32, device=DEV)
        out = torch.zeros(end, H * dv, device=DEV)
        o.attn_portion_gen(q, k_in, v_in, table, items, out, page, 1, H, KV, dk, dv, dk ** -0.5, dist_bias=rel, softcap=cap, v_share=share)
        got.append(out[:, :G * dv].clone())
    assert bool(torch.isfinite(got[0]).all()) and bool(got[0].abs().amax() > 0)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("kind", ["delta", "decay"])
@pytest.mark.parametrize("at", [1, 2, 3, 6, 8])
def test_groups_of_four_keep_the_order_of_tokens(kind, at):
    """A token whose value is not finite leaves every earlier token's result as it is, also those of its own group of four: the same
    bits as with another number there."""
    o = ops()
    g = torch.Generator().manual_seed(at)
    H, n, T = 2, 64, 9
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q_start, ctx, slot, row_seq = i32([0, T]), i32([T]), i32([0]), i32([0] * T)
    outs = []
    if kind == "delta":
        xc, u = torch.randn(T, 2 * n + H * n, generator=g), torch.randn(T, 2 * H, generator=g).to(DEV)
        a_log, dt_bias = torch.rand(H, generator=g).to(DEV), torch.rand(H, generator=g).to(DEV)
    else:
        xs, u = torch.randn(T, 4 * H * n, generator=g), torch.randn(H, n, generator=g).to(DEV)
        xs[:, 3 * H * n:] = 0.9
    for odd in (1.0, math.nan, math.inf):
        y = torch.zeros(T, H * n, device=DEV)
        if kind == "delta":
            x = xc.clone()
            x[at, 2 * n:] = odd
            x = x.to(DEV)
            state, bg = torch.zeros(1, H * o.delta_state_floats(n, n), device=DEV), torch.empty(T, 2 * H + 1, device=DEV)
            o.delta_prepare(x, u, 0, H, a_log, dt_bias, bg, 1, H, n, n ** -0.5)
            dec, rec, sc = torch.empty(T, H * n, device=DEV), torch.empty(T, H, 3, n, device=DEV), torch.empty(T, H, o.GROUP_SCALARS, device=DEV)
            o.channel_delta_groups(x, u, 0, dec, a_log, dt_bias, rec, sc, row_seq, q_start, 1, 1, H, n, a_off=H)
            o.channel_delta_group_scan(rec, sc, dec, x, state, y, q_start, ctx, slot, 1, 1, H, n, n)
        else:
            x = xs.clone()
            x[at, 2 * H * n:3 * H * n] = odd
            state = torch.zeros(1, H * o.decay_state_floats(n), device=DEV)
            o.decay_group_scan(x.to(DEV), u, torch.empty(T, H, 4, device=DEV), state, y, row_seq, q_start, ctx, slot, 1, H, n)
        outs.append(y[:at].cpu())
    assert bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("dk,dv,ok", [(152, 8, True), (156, 8, False), (256, 4, False), (256, 12, True), (256, 16, True), (8, 4, False)])
def test_group_sizes_that_are_taken_run(dk, dv, ok):
    """Few columns have few threads, which copy the pieces of a group of wide keys no longer: such heads go token by token. What is taken
    runs."""
    o = ops()
    assert o.channel_delta_groups_ok(dk, dv) == ok
    if not ok:
        return
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    rec, sc, dec = torch.zeros(5, 1, 3, dk, device=DEV), torch.zeros(5, 1, o.GROUP_SCALARS, device=DEV), torch.ones(5, dk, device=DEV)
    state = torch.ones(1, o.delta_state_floats(dk, dv), device=DEV)
    o.channel_delta_group_scan(rec, sc, dec, torch.zeros(5, 2 * dk + dv, device=DEV), state, torch.empty(5, dv, device=DEV), i32([0, 5]), i32([7]), i32([0]),
                               1, 1, 1, dk, dv)
    assert bool((state <= 1).all()) and float(state.sum()) == dk * dv      # (entries behind dk are written as zeros)


@pytest.mark.parametrize("odd", [math.nan, math.inf])
@pytest.mark.parametrize("at", [0, 7, 8, 16])
def test_plain_attention_keeps_no_result_that_is_not_finite_from_sight(at, odd):
    """A key that is not finite (here the only one of its warp's run, or one of eight) spoils the rows that see it: they come out as zeros,
    the mark of a row without a finite sum, and never as the weighted sum of the other keys. Rows before it are what they were."""
    o = ops()
    g = torch.Generator().manual_seed(at)
    T, hs = 17, 32
    q, k, v = (torch.randn(T, hs, generator=g) for _ in range(3))
    q = q.abs() + 0.1                                 # an infinite key gives infinite scores, not NaN
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    outs = []
    for x in (0.5, odd):
        k[at] = x
        out = torch.full((T, hs), 7.0, device=DEV)
        o.paged_attention_ref(q.to(DEV), k.view(T, 1, 1, hs).to(DEV), v.view(T, 1, 1, hs).to(DEV), i32(list(range(T))).view(1, -1), i32([0] * T),
                              i32(list(range(T))), out, 1, 1, 1, 1, hs, hs ** -0.5)
        outs.append(out.cpu())
    assert torch.equal(outs[0][:at], outs[1][:at]) and bool(outs[0].abs().amax(1).min() > 0)
    assert bool((outs[1][at:] == 0).all() | torch.isnan(outs[1][at:]).all())


def test_experts_results_with_no_rows_for_identity_experts():
    """The combining sum with results of the experts that have weights only: places of identity experts have no row."""
    o = ops()
    g = torch.Generator().manual_seed(1)
    y, x, wts = torch.randn(3, 40, generator=g), torch.randn(2, 40, generator=g), torch.rand(2, 2, generator=g)
    ids = torch.tensor([[0, 5], [1, 2]], dtype=torch.int32)
    place = torch.tensor([[1, 3], [0, 2]], dtype=torch.int32)         # place 3 is the identity expert's: y has no such row
    out = torch.empty(2, 40, device=DEV)
    o.moe_combine(y.to(DEV), place.to(DEV), wts.to(DEV), out, ids=ids.to(DEV), real=4, x=x.to(DEV))
    want = torch.stack([wts[0, 0] * y[1] + wts[0, 1] * x[0], wts[1, 0] * y[0] + wts[1, 1] * y[2]])
    assert (out.cpu() - want).abs().max().item() <= 1e-6
