"""Each kernel alone against a plain float32/float64 reference of the same operation,
at sizes other than the engine's: widths and vocabularies that are no power of two,
head sizes in steps of 16, several heads-per-group ratios."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# relative to the magnitude of the outputs (order 1 here): float32 sums of a few hundred
# terms; bfloat16 results rounded once to 8 bits of mantissa
TOL = {"float32": 2e-5, "bfloat16": 1.6e-2}


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).cuda()


def close(got, want, dtype, what=""):
    got, want = got.double().cpu(), want.double().cpu()
    err = (got - want).abs().max().item()
    mag = max(want.abs().max().item(), 1.0)
    assert math.isfinite(err) and err <= TOL[dtype] * mag, f"{what}: max err {err:.3e} (magnitude {mag:.2f})"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("V,E", [(300, 72), (1003, 200)])
def test_embed_rows(dtype, V, E):
    from alpacca_b200 import ops
    table = rnd(V, E, dtype=DT[dtype])
    toks = torch.tensor([0, V - 1, 5, 5, 17], dtype=torch.int32).cuda()
    out = torch.empty(5, E, dtype=torch.float32, device="cuda")
    ops.embed_rows(table, toks, out)
    assert torch.equal(out, table[toks.long()].float())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,E,eps", [(1, 72, 1e-5), (7, 200, 1e-6), (33, 2056, 3e-6)])
def test_add_rmsnorm(dtype, T, E, eps):
    from alpacca_b200 import ops
    res = rnd(T, E, seed=1)
    delta = rnd(T, E, dtype=DT[dtype], seed=2)
    w = 1 + rnd(E, seed=3) * 0.1
    want_res = res.double() + delta.double()
    want = want_res / torch.sqrt((want_res ** 2).mean(-1, keepdim=True) + eps) * w.double()
    r = res.clone()
    out = torch.empty(T, E, dtype=DT[dtype], device="cuda")
    ops.add_rmsnorm(r, delta, w, eps, out)
    close(out, want, dtype, "normed")
    close(r, want_res, "float32", "residual after the add")
    # rows: picked rows only, residual untouched
    rows = torch.tensor([T - 1, 0], dtype=torch.int32).cuda()
    r2 = res.clone()
    out2 = torch.empty(2, E, dtype=DT[dtype], device="cuda")
    ops.add_rmsnorm(r2, delta, w, eps, out2, rows=rows)
    close(out2, want[[T - 1, 0]], dtype, "picked rows")
    assert torch.equal(r2, res)
    # without delta
    out3 = torch.empty(T, E, dtype=DT[dtype], device="cuda")
    ops.add_rmsnorm(res.clone(), None, w, eps, out3)
    want3 = res.double() / torch.sqrt((res.double() ** 2).mean(-1, keepdim=True) + eps) * w.double()
    close(out3, want3, dtype, "no delta")


def ref_rope(x, pos, n_rot, pairing, cos, sin):
    """x [T, heads, D] float64."""
    x = x.clone()
    half = n_rot // 2
    c, s = cos[pos][:, None, :].double(), sin[pos][:, None, :].double()
    if pairing == 0:
        a, b = x[..., 0:n_rot:2].clone(), x[..., 1:n_rot:2].clone()
        x[..., 0:n_rot:2], x[..., 1:n_rot:2] = a * c - b * s, a * s + b * c
    else:
        a, b = x[..., :half].clone(), x[..., half:n_rot].clone()
        x[..., :half], x[..., half:n_rot] = a * c - b * s, a * s + b * c
    return x


def make_paged(lengths, n_pages, K, D, dtype, page=64, seed=0):
    """Block table with pages handed out in a scattered order; returns table, k/v pages."""
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(n_pages, generator=g).tolist()
    width = max(-(-n // page) for n in lengths)
    table = torch.zeros(len(lengths), width, dtype=torch.int32)
    for b, n in enumerate(lengths):
        for i in range(-(-n // page)):
            table[b, i] = perm.pop()
    k = torch.zeros(n_pages, K, page, D, dtype=dtype, device="cuda")
    v = torch.zeros_like(k)
    return table.cuda(), k, v


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,K,D,n_rot,pairing", [(4, 4, 16, 16, 0), (6, 2, 32, 32, 1), (10, 5, 48, 32, 1),
                                                 (3, 1, 80, 40, 0)])
def test_rope_append(dtype, H, K, D, n_rot, pairing):
    from alpacca_b200 import ops
    lengths = [70, 3, 130]           # tokens already there + new ones; new tokens are the last q_len
    q_lens = [5, 3, 66]
    table, kp, vp = make_paged(lengths, 8, K, D, DT[dtype])
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=DT[dtype], seed=5)
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32)
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32)
    P = 160
    inv = 10000.0 ** (-torch.arange(n_rot // 2, dtype=torch.float64) * 2 / n_rot)
    ang = torch.arange(P, dtype=torch.float64)[:, None] * inv
    cos, sin = torch.cos(ang).float().cuda(), torch.sin(ang).float().cuda()
    x = qkv.double().cpu().view(T, H + 2 * K, D)
    want_qk = ref_rope(x[:, :H + K], pos.long(), n_rot, pairing, cos.cpu(), sin.cpu())
    got = qkv.clone()
    ops.rope_append(got, cos, sin, pos.cuda(), seq.cuda(), table, kp, vp, T, H, K, D, n_rot, pairing)
    g = got.double().cpu().view(T, H + 2 * K, D)
    close(g[:, :H], want_qk[:, :H], dtype, "q rotated in place")
    tb = table.cpu()
    for t in range(T):
        page, off = tb[seq[t], pos[t] // 64].item(), pos[t].item() % 64
        close(kp[page, :, off], want_qk[t, H:], dtype, f"k of token {t} in the cache")
        close(vp[page, :, off], x[t, H + K:], dtype, f"v of token {t} in the cache")
    # padding tokens are skipped
    got2, kp2 = qkv.clone(), torch.zeros_like(kp)
    ops.rope_append(got2, cos, sin, pos.cuda(), torch.full_like(seq, -1).cuda(), table, kp2, torch.zeros_like(vp),
                    T, H, K, D, n_rot, pairing)
    assert torch.equal(got2, qkv) and kp2.abs().sum().item() == 0


def ref_attention(q, k, v, pos_q, scale, window=0):
    """q [Tq,H,D], k/v [S,K,D] float64, pos_q: position of each query."""
    Tq, H, D = q.shape
    G = H // k.shape[1]
    out = torch.zeros(Tq, H, D, dtype=torch.float64)
    for t in range(Tq):
        p = int(pos_q[t])
        lo = max(0, p - window + 1) if window else 0
        for h in range(H):
            sc = (k[lo:p + 1, h // G] @ q[t, h]) * scale
            out[t, h] = torch.softmax(sc, 0) @ v[lo:p + 1, h // G]
    return out


def fill_cache(table, kp, vp, b, kk, vv):
    for s in range(kk.shape[0]):
        page = table[b, s // 64].item()
        kp[page, :, s % 64] = kk[s].to(kp.dtype)
        vp[page, :, s % 64] = vv[s].to(vp.dtype)


ATT_CASES = [(4, 4, 16), (6, 2, 32), (10, 5, 48), (8, 1, 64), (5, 5, 80), (4, 2, 128), (2, 1, 256), (14, 2, 96)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,K,D", ATT_CASES)
@pytest.mark.parametrize("window", [0, 37])
def test_attention_prefill_and_decode(dtype, H, K, D, window):
    """Three sequences in one launch: a prompt from position 0, a chunk on top of cached
    tokens, and a single decode token far into its sequence."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    lengths, q_lens = [75, 200, 301], [75, 40, 1]
    table, kp, vp = make_paged(lengths, 12, K, D, DT[dtype], seed=D)
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=DT[dtype], seed=7)
    ks = [rnd(n, K, D, dtype=DT[dtype], seed=8 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=DT[dtype], seed=11 + b) for b, n in enumerate(lengths)]
    for b in range(3):
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32)
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32)
    scale = D ** -0.5
    out = torch.empty(T, H * D, dtype=DT[dtype], device="cuda")
    cu = torch.tensor([0, 75, 115, 116], dtype=torch.int32).cuda()
    ctx = SimpleNamespace(tok_pos=pos.cuda(), tok_seq=seq.cuda(), n_tokens=T, n_seqs=3, cu_q=cu,
                          kv_len=torch.tensor(lengths, dtype=torch.int32).cuda(), is_decode=False,
                          host_q_lens=q_lens, host_kv_lens=lengths, max_q_len=75, max_kv_len=301, extras={})
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, scale, window)
    q = qkv.double().cpu().view(T, H + 2 * K, D)[:, :H]
    t0 = 0
    for b, (n, ql) in enumerate(zip(lengths, q_lens)):
        want = ref_attention(q[t0:t0 + ql], ks[b].double().cpu(), vs[b].double().cpu(), pos[t0:t0 + ql], scale, window)
        close(out[t0:t0 + ql].view(ql, H, D), want, dtype, f"sequence {b}")
        t0 += ql


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_finds_one_far_key(dtype):
    """Among hundreds of keys one, far back and on another page, matches the query: the
    output must be its value.  A kernel that skips, misplaces or masks that key shows here."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    H, K, D, n = 4, 2, 64, 700
    table, kp, vp = make_paged([n], 16, K, D, DT[dtype], seed=3)
    kk = rnd(n, K, D, seed=1) * 0.1
    vv = rnd(n, K, D, seed=2)
    qkv = torch.zeros(1, (H + 2 * K) * D, device="cuda")
    far = {0: 5, 1: 64, 2: 383, 3: 699}      # page starts, page ends, the first and the very last key
    for h, s in far.items():
        direction = torch.zeros(D, device="cuda")
        direction[h * 7] = 1.0
        kk[s, h // 2] = direction * 30.0
        qkv[0, h * D:(h + 1) * D] = direction * 30.0
    fill_cache(table.cpu(), kp, vp, 0, kk, vv)
    qkv = qkv.to(DT[dtype])
    out = torch.empty(1, H * D, dtype=DT[dtype], device="cuda")
    ctx = SimpleNamespace(tok_pos=torch.tensor([n - 1], dtype=torch.int32).cuda(),
                          tok_seq=torch.zeros(1, dtype=torch.int32).cuda(), n_tokens=1, n_seqs=1,
                          cu_q=torch.tensor([0, 1], dtype=torch.int32).cuda(),
                          kv_len=torch.tensor([n], dtype=torch.int32).cuda(), is_decode=True,
                          host_q_lens=[1], host_kv_lens=[n], max_q_len=1, max_kv_len=n, extras={})
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, 0)
    for h, s in far.items():
        want = vp[table[0, s // 64].item(), h // 2, s % 64].float()
        got = out[0, h * D:(h + 1) * D].float()
        assert (got - want).abs().max().item() < 2e-2, f"head {h} did not find key {s}"
    # with a window the far keys are cut off, except the last one, which lies inside it
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, 100)
    want = vp[table[0, 699 // 64].item(), 1, 699 % 64].float()
    assert (out[0, 3 * D:].float() - want).abs().max().item() < 2e-2
    # the window's edge: position n-100 is the first key inside, n-101 the last one outside
    kk2 = kk.clone()
    kk2[600, 0] = kk[5, 0]       # head 0's matching key, now on the edge
    kk2[599, 1] = kk[383, 1]     # head 2's matching key, now just outside (its old place 383 is outside too)
    fill_cache(table.cpu(), kp, vp, 0, kk2, vv)
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, 100)
    edge = vp[table[0, 600 // 64].item(), 0, 600 % 64].float()
    assert (out[0, :D].float() - edge).abs().max().item() < 2e-2, "the key on the window's edge was not seen"
    outside = vp[table[0, 599 // 64].item(), 1, 599 % 64].float()
    assert (out[0, 2 * D:3 * D].float() - outside).abs().max().item() > 0.1, "a key outside the window was seen"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,F", [(1, 160), (9, 264), (70, 1000)])
def test_swiglu(dtype, T, F):
    from alpacca_b200 import ops
    gate, up = rnd(T, F, seed=1) * 3, rnd(T, F, seed=2)
    gu = torch.cat([gate.view(T, F // 8, 8), up.view(T, F // 8, 8)], dim=2).reshape(T, 2 * F).to(DT[dtype])
    g, u = gu.view(T, F // 8, 2, 8)[:, :, 0].reshape(T, F).double(), gu.view(T, F // 8, 2, 8)[:, :, 1].reshape(T, F).double()
    out = torch.empty(T, F, dtype=DT[dtype], device="cuda")
    ops.swiglu(gu, out)
    close(out, g / (1 + torch.exp(-g)) * u, dtype)


@pytest.mark.parametrize("M,N,K", [(1, 72, 200), (5, 1003, 120), (70, 264, 333), (130, 64, 64)])
def test_gemm_f32(M, N, K):
    from alpacca_b200 import ops
    a, w, bias = rnd(M, K, seed=1), rnd(N, K, seed=2), rnd(N, seed=3)
    out = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, out, bias=bias)
    close(out, a.double() @ w.double().T + bias.double(), "float32")
    # a row's result does not depend on the rows beside it
    out1 = torch.empty(1, N, device="cuda")
    ops.gemm_f32(a[M // 2:M // 2 + 1].contiguous(), w, out1, bias=bias)
    assert torch.equal(out1[0], out[M // 2])


@pytest.mark.parametrize("K", [24, 250, 2048, 3000])
@pytest.mark.parametrize("N", [40, 129, 2100])
def test_gemm_f32_tiles(N, K):
    """Every tile height and both splits (K 250: rows that are not 16-byte aligned): the bits of a row do not depend on the
    number of rows, and are right.  Bound: each of the K additions of a sum rounds a partial sum, of about |a| |w| / sqrt(K)
    for random signs, by 2^-24 at most; even if all K rounded one way after a walk of sqrt(K) steps: 2^-24 |a| |w|; times 4."""
    from alpacca_b200 import ops
    a, w = rnd(230, K, seed=1), rnd(N, K, seed=2)
    want = a.double() @ w.double().T
    bound = 2.0 ** -22 * a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None]
    whole = torch.empty(230, N, device="cuda")
    ops.gemm_f32(a, w, whole)
    assert ((whole.double() - want).abs() <= bound).all()
    for M in (1, 8, 9, 16, 17, 32, 33, 64, 65, 200):
        out = torch.full((M + 1, N), 7.0, device="cuda")
        ops.gemm_f32(a[:M], w, out, n_rows=M)
        assert torch.equal(out[:M], whole[:M]) and (out[M] == 7.0).all(), M


@pytest.mark.parametrize("M,N,K", [(1, 72, 200), (3, 1003, 120), (8, 264, 328), (16, 520, 64), (70, 264, 336)])
@pytest.mark.parametrize("out_dtype", ["bfloat16", "float32"])
def test_linear_bf16(M, N, K, out_dtype):
    from alpacca_b200 import ops
    a, w = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2)
    out = torch.empty(M, N, dtype=DT[out_dtype], device="cuda")
    ops.linear_bf16(a, w, out)
    want = a.double() @ w.double().T
    close(out, want, out_dtype if out_dtype == "bfloat16" else "float32", "linear_bf16")


def test_add_bias():
    from alpacca_b200 import ops
    y, b = rnd(7, 72, dtype=torch.bfloat16), rnd(72, seed=4)
    want = y.float() + b
    ops.add_bias(y, b)
    close(y, want, "bfloat16")


def decode_ctx(lengths):
    from types import SimpleNamespace
    B = len(lengths)
    return SimpleNamespace(
        tok_pos=torch.tensor([n - 1 for n in lengths], dtype=torch.int32).cuda(),
        tok_seq=torch.arange(B, dtype=torch.int32).cuda(), n_tokens=B, n_seqs=B,
        cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_len=torch.tensor(lengths, dtype=torch.int32).cuda(),
        is_decode=True, host_q_lens=[1] * B, host_kv_lens=list(lengths), max_q_len=1, max_kv_len=max(lengths),
        extras={})


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,K,D", ATT_CASES + [(40, 2, 64)])
@pytest.mark.parametrize("window", [0, 130])
def test_attention_decode_batch(dtype, H, K, D, window):
    """One token per sequence, lengths from 1 to beyond a thousand keys (one to several chunks)."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    lengths = [1, 64, 65, 300, 700, 1025]
    table, kp, vp = make_paged(lengths, 40, K, D, DT[dtype], seed=D + H)
    B = len(lengths)
    qkv = rnd(B, (H + 2 * K) * D, dtype=DT[dtype], seed=17)
    ks = [rnd(n, K, D, dtype=DT[dtype], seed=18 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=DT[dtype], seed=31 + b) for b, n in enumerate(lengths)]
    for b in range(B):
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    ctx = decode_ctx(lengths)
    out = torch.empty(B, H * D, dtype=DT[dtype], device="cuda")
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window)
    q = qkv.double().cpu().view(B, H + 2 * K, D)[:, :H]
    for b, n in enumerate(lengths):
        want = ref_attention(q[b:b + 1], ks[b].double().cpu(), vs[b].double().cpu(), [n - 1], D ** -0.5, window)
        close(out[b].view(1, H, D), want, dtype, f"sequence of {n}")
    # a padded row (tok_seq -1) is skipped and leaves its output alone
    ctx.tok_seq[2] = -1
    out2 = torch.full_like(out, 7.0)
    ops.attention(qkv, out2, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window)
    assert torch.equal(out2[2], torch.full_like(out2[2], 7.0)) and torch.equal(out2[3], out[3])


@pytest.mark.parametrize("H,K,D", [(6, 2, 32), (8, 1, 64), (3, 3, 72)])
def test_attention_32bit_kernel_on_bfloat16(H, K, D):
    """The 32-bit kernel also serves bfloat16 tensors (head sizes the tensor-core kernel refuses)."""
    from alpacca_b200 import ops
    lengths = [5, 200]
    table, kp, vp = make_paged(lengths, 6, K, D, torch.bfloat16, seed=D)
    qkv = rnd(2, (H + 2 * K) * D, dtype=torch.bfloat16, seed=3)
    ks = [rnd(n, K, D, dtype=torch.bfloat16, seed=4 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=torch.bfloat16, seed=6 + b) for b, n in enumerate(lengths)]
    for b in range(2):
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    ctx = decode_ctx(lengths)
    out = torch.empty(2, H * D, dtype=torch.bfloat16, device="cuda")
    ops.attention_simt(qkv, out, kp, vp, table, ctx.tok_pos, ctx.tok_seq, 2, H, K, D, D ** -0.5, 0)
    q = qkv.double().cpu().view(2, H + 2 * K, D)[:, :H]
    for b, n in enumerate(lengths):
        want = ref_attention(q[b:b + 1], ks[b].double().cpu(), vs[b].double().cpu(), [n - 1], D ** -0.5)
        close(out[b].view(1, H, D), want, "bfloat16")


@pytest.mark.parametrize("M", [1, 5, 8, 13, 16, 27, 32])
@pytest.mark.parametrize("N,K", [(72, 200), (1003, 120), (2048, 2048), (264, 8200)])
def test_gemv_bf16(M, N, K):
    from alpacca_b200 import ops
    x, w, bias = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(N, seed=3)
    want = x.double() @ w.double().T + bias.double()
    for dt, tol in ((torch.float32, "float32"), (torch.bfloat16, "bfloat16")):
        out = torch.full((M, N), 9.0, dtype=dt, device="cuda")
        ops.gemv_bf16(x, w, out, bias=bias)
        close(out, want, tol, f"gemv {dt}")
    # fewer rows than the buffers hold: the rest is left alone
    if M > 1:
        out = torch.full((M, N), 9.0, dtype=torch.float32, device="cuda")
        ops.gemv_bf16(x, w, out, n_rows=M - 1)
        assert (out[M - 1] == 9.0).all()
        close(out[:M - 1], (x.double() @ w.double().T)[:M - 1], "float32")


@pytest.mark.parametrize("M,F,K", [(1, 160, 64), (7, 264, 120), (16, 1000, 328)])
def test_gemv_bf16_swiglu_epilogue(M, F, K):
    from alpacca_b200 import ops
    x = rnd(M, K, dtype=torch.bfloat16, seed=1)
    gate, up = rnd(F, K, dtype=torch.bfloat16, seed=2, scale=0.3), rnd(F, K, dtype=torch.bfloat16, seed=3, scale=0.3)
    bg, bu = rnd(F, seed=4), rnd(F, seed=5)
    w = torch.cat([gate.view(F // 8, 8, K), up.view(F // 8, 8, K)], dim=1).reshape(2 * F, K).contiguous()
    bias = torch.cat([bg.view(F // 8, 8), bu.view(F // 8, 8)], dim=1).reshape(2 * F).contiguous()
    g = x.double() @ gate.double().T + bg.double()
    u = x.double() @ up.double().T + bu.double()
    out = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    ops.gemv_bf16(x, w, out, bias=bias, swiglu=True)
    close(out, g / (1 + torch.exp(-g)) * u, "bfloat16", "swiglu epilogue")


@pytest.mark.parametrize("M", [1, 5, 8, 13, 32])
@pytest.mark.parametrize("E,K,N2,slices", [(72, 200, 88, 1), (2048, 264, 1003, 1), (200, 8200, 72, 1),
                                           (4104, 128, 160, 1), (264, 4096, 520, 3)])
def test_gemv_bf16_norm_between_two_products(M, E, K, N2, slices):
    """The residual epilogue (add to the 32-bit residual, bf16(residual * norm weight), partial sums of
    squares) and the product after it that applies the owed division by the rms: together they are
    product, residual add, RMS norm (alpacca/tensor.py:163-173), product; also with the activation."""
    from alpacca_b200 import ops
    eps = 3e-4
    x = rnd(M, K, dtype=torch.bfloat16, seed=1)
    w1, b1 = rnd(E, K, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(E, seed=3)
    res0 = rnd(M, E, seed=4, scale=2.0)
    nw = 1.0 + rnd(E, seed=5, scale=0.3)
    w2, b2 = rnd(N2, E, dtype=torch.bfloat16, seed=6, scale=0.1), rnd(N2, seed=7)
    want_res = res0.double() + x.double() @ w1.double().T + b1.double()
    rms = torch.sqrt((want_res ** 2).mean(-1, keepdim=True) + eps)
    normed = want_res / rms * nw.double()
    want = normed @ w2.double().T + b2.double()

    res = res0.clone()
    xw = torch.full((M, E), 9.0, dtype=torch.bfloat16, device="cuda")
    _, ss = ops.gemv_bf16(x, w1, xw, bias=b1, residual=res, norm_weight=nw, slices=slices)
    close(res, want_res, "float32", "residual after the product")
    assert tuple(ss.shape) == (M, -(-E // 16))
    close(ss.sum(-1), (want_res ** 2).sum(-1), "float32", "sums of squares")
    close(xw, want_res * nw.double(), "bfloat16", "residual times the norm weight")
    owed = (ss, E, eps)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((M, N2), 9.0, dtype=dt, device="cuda")
        ops.gemv_bf16(xw, w2, out, bias=b2, owed=owed)
        close(out, want, "bfloat16", f"product after the norm {dt}")
    if N2 % 16 == 0:
        F = N2 // 2
        g = want.view(M, F // 8, 2, 8)[:, :, 0].reshape(M, F)
        u = want.view(M, F // 8, 2, 8)[:, :, 1].reshape(M, F)
        out = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
        ops.gemv_bf16(xw, w2, out, bias=b2, swiglu=True, owed=owed)
        close(out, g / (1 + torch.exp(-g)) * u, "bfloat16", "activation after the norm")
    # fewer rows than the buffers hold: the rest of the residual is left alone
    if M > 1:
        res = res0.clone()
        ops.gemv_bf16(x, w1, xw, bias=b1, residual=res, norm_weight=nw, n_rows=M - 1)
        assert torch.equal(res[M - 1], res0[M - 1])
        close(res[:M - 1], want_res[:M - 1], "float32")


@pytest.mark.parametrize("M,N,K", [(3, 1003, 120), (8, 70, 64), (16, 2050, 264)])
def test_gemv_bf16_residual_epilogue_at_odd_widths(M, N, K):
    """The residual epilogue where the stream's width is no multiple of 4 (the tile of the residual is
    then read straight from memory, not staged) and the last slab is partial."""
    from alpacca_b200 import ops
    x, w, b = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(N, seed=3)
    res0, nw = rnd(M, N, seed=4, scale=2.0), 1.0 + rnd(N, seed=5, scale=0.3)
    want = res0.double() + x.double() @ w.double().T + b.double()
    res, xw = res0.clone(), torch.full((M, N), 9.0, dtype=torch.bfloat16, device="cuda")
    _, ss = ops.gemv_bf16(x, w, xw, bias=b, residual=res, norm_weight=nw)
    close(res, want, "float32", "residual")
    close(xw, want * nw.double(), "bfloat16", "residual times the norm weight")
    close(ss.sum(-1), (want ** 2).sum(-1), "float32", "sums of squares")


@pytest.mark.parametrize("M,N,K,swap,bn,slices", [
    (128, 256, 64, False, 256, 1), (300, 520, 328, False, 128, 1), (2048, 1024, 512, False, 256, 1),
    (8, 128, 128, True, 16, 1), (13, 1003, 200, True, 16, 1), (33, 520, 264, True, 64, 1),
    (64, 2048, 2048, True, 64, 4), (20, 264, 4096, True, 32, 3)])
def test_gemm_tc(M, N, K, swap, bn, slices):
    """The tcgen05 product in both orientations, with ragged edges, K slices and both output types."""
    from alpacca_b200 import ops
    x, w, bias = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(N, seed=3)
    want = x.double() @ w.double().T + bias.double()
    for dt, tol in ((torch.float32, "float32"), (torch.bfloat16, "bfloat16")):
        out = torch.full((M, N), 9.0, dtype=dt, device="cuda")
        ops.gemm_tc(x, w, out, bias=bias, swap=swap, bn=bn, slices=slices)
        close(out, want, tol, f"gemm_tc {dt}")
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("M,F,K,swap,bn", [(9, 160, 64, True, 16), (64, 264, 328, True, 64), (300, 1000, 200, False, 128),
                                           (128, 512, 256, False, 256)])
def test_gemm_tc_swiglu_epilogue(M, F, K, swap, bn):
    from alpacca_b200 import ops
    x = rnd(M, K, dtype=torch.bfloat16, seed=1)
    gate, up = rnd(F, K, dtype=torch.bfloat16, seed=2, scale=0.3), rnd(F, K, dtype=torch.bfloat16, seed=3, scale=0.3)
    bg, bu = rnd(F, seed=4), rnd(F, seed=5)
    w = torch.cat([gate.view(F // 8, 8, K), up.view(F // 8, 8, K)], dim=1).reshape(2 * F, K).contiguous()
    bias = torch.cat([bg.view(F // 8, 8), bu.view(F // 8, 8)], dim=1).reshape(2 * F).contiguous()
    g = x.double() @ gate.double().T + bg.double()
    u = x.double() @ up.double().T + bu.double()
    out = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc(x, w, out, bias=bias, swiglu=True, swap=swap, bn=bn, slices=1)
    close(out, g / (1 + torch.exp(-g)) * u, "bfloat16", "tcgen05 swiglu epilogue")
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("H,K,D", [(4, 4, 64), (8, 2, 64), (32, 8, 64), (16, 1, 64), (6, 6, 64), (6, 2, 64), (10, 2, 64),
                                   (4, 4, 128), (8, 2, 128), (16, 1, 128), (12, 2, 128), (7, 1, 128)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("growing", [False, True])
def test_attention_prefill_tcgen05(H, K, D, window, growing):
    """The tcgen05 prefill kernel (head sizes 64 and 128): whole prompts, a chunk on cached tokens,
    several sequences in one launch; against the float64 reference and against the mma.sync kernel.
    `growing`: the keys get longer with their position, so that the rows' maxima keep rising by large
    steps and the kernel has to move its references and rescale its output again and again."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    lengths, q_lens = [300, 150, 513], [300, 100, 130]
    table, kp, vp = make_paged(lengths, 20, K, D, torch.bfloat16, seed=H)
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=torch.bfloat16, seed=7)
    ks = [rnd(n, K, D, dtype=torch.bfloat16, seed=8 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=torch.bfloat16, seed=11 + b) for b, n in enumerate(lengths)]
    if growing:
        ks = [(k.float() * (1.0 + torch.arange(k.shape[0], device=k.device).view(-1, 1, 1) / 16.0)).to(torch.bfloat16)
              for k in ks]
    for b in range(3):
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32)
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32)
    cu = torch.tensor([0, 300, 400, 530], dtype=torch.int32).cuda()

    def run(use_tc):
        ctx = SimpleNamespace(tok_pos=pos.cuda(), tok_seq=seq.cuda(), n_tokens=T, n_seqs=3, cu_q=cu,
                              kv_len=torch.tensor(lengths, dtype=torch.int32).cuda(), is_decode=False,
                              host_q_lens=q_lens, host_kv_lens=lengths, max_q_len=300, max_kv_len=513, extras={})
        out = torch.zeros(T, H * D, dtype=torch.bfloat16, device="cuda")
        old = ops.USE_TCGEN05_ATTENTION
        ops.USE_TCGEN05_ATTENTION = use_tc
        try:
            ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window)
        finally:
            ops.USE_TCGEN05_ATTENTION = old
        return out
    got, other = run(True), run(False)
    assert ops.attention_tc_status() == 0
    q = qkv.double().cpu().view(T, H + 2 * K, D)[:, :H]
    t0 = 0
    for b, (n, ql) in enumerate(zip(lengths, q_lens)):
        want = ref_attention(q[t0:t0 + ql], ks[b].double().cpu(), vs[b].double().cpu(), pos[t0:t0 + ql], D ** -0.5, window)
        close(got[t0:t0 + ql].view(ql, H, D), want, "bfloat16", f"tcgen05, sequence {b}")
        close(other[t0:t0 + ql].view(ql, H, D), want, "bfloat16", f"mma.sync, sequence {b}")
        t0 += ql


@pytest.mark.parametrize("H,K", [(4, 4), (8, 2), (16, 1), (12, 2), (7, 1)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("growing", [False, True])
def test_attention_prefill_two_tiles(H, K, window, growing, monkeypatch):
    """The prompt kernel with two query tiles per CTA: second tiles that are full, partly filled, empty and at the step's end, a
    sequence of one new token, odd numbers of pages, keys that keep growing; against 64-bit arithmetic."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    monkeypatch.setattr(ops, "_pair_pays", lambda *a: True)
    D, lengths, q_lens = 128, [300, 150, 513, 65], [300, 1, 130, 65]
    table, kp, vp = make_paged(lengths, 20, K, D, torch.bfloat16, seed=H)
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=torch.bfloat16, seed=7)
    ks = [rnd(n, K, D, dtype=torch.bfloat16, seed=8 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=torch.bfloat16, seed=11 + b) for b, n in enumerate(lengths)]
    if growing:
        ks = [(k.float() * (1.0 + torch.arange(k.shape[0], device=k.device).view(-1, 1, 1) / 16.0)).to(torch.bfloat16) for k in ks]
    for b in range(4):
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32)
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32)
    cu = torch.tensor([0, 300, 301, 431, 496], dtype=torch.int32).cuda()
    ctx = SimpleNamespace(tok_pos=pos.cuda(), tok_seq=seq.cuda(), n_tokens=T, n_seqs=4, cu_q=cu, is_decode=False,
                          kv_len=torch.tensor(lengths, dtype=torch.int32).cuda(), host_q_lens=q_lens, host_kv_lens=lengths,
                          max_q_len=300, max_kv_len=513, extras={})
    out = torch.zeros(T, H * D, dtype=torch.bfloat16, device="cuda")
    ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window)
    assert ops.attention_pair_tc_status() == 0
    q = qkv.double().cpu().view(T, H + 2 * K, D)[:, :H]
    t0 = 0
    for b, ql in enumerate(q_lens):
        want = ref_attention(q[t0:t0 + ql], ks[b].double().cpu(), vs[b].double().cpu(), pos[t0:t0 + ql], D ** -0.5, window)
        close(out[t0:t0 + ql].view(ql, H, D), want, "bfloat16", f"sequence {b}")
        t0 += ql


@pytest.mark.parametrize("H,K,D,n_rot,pairing", [(4, 4, 16, 16, 0), (6, 2, 32, 32, 1), (10, 5, 48, 32, 1),
                                                 (32, 8, 64, 64, 1), (4, 2, 128, 64, 0), (40, 2, 64, 0, 0)])
@pytest.mark.parametrize("window", [0, 130])
@pytest.mark.parametrize("write_cache", [True, False])
def test_rope_attention_fused_decode(H, K, D, n_rot, pairing, window, write_cache):
    """Rotation, append and attention of a decode step in one kernel against the two kernels one
    after the other: the same outputs and the same cache, bit for bit; one to several chunks."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    lengths = [1, 64, 65, 300, 769, 1025, 1600]
    B = len(lengths)
    qkv0 = rnd(B, (H + 2 * K) * D, dtype=torch.bfloat16, seed=17)
    ang = rnd(1700, max(n_rot // 2, 1), seed=5, scale=3.0)
    rot = (torch.cos(ang).contiguous(), torch.sin(ang).contiguous(), n_rot, pairing) if n_rot else None
    results = []
    for fused in (False, True):
        table, kp, vp = make_paged(lengths, 70, K, D, torch.bfloat16, seed=D + H)
        for b, n in enumerate(lengths):
            # with write_cache off the step's own row is in the cache already (another layer's)
            fill_cache(table.cpu(), kp, vp, b, rnd(n, K, D, dtype=torch.bfloat16, seed=18 + b),
                       rnd(n, K, D, dtype=torch.bfloat16, seed=31 + b))
        ctx = decode_ctx(lengths)
        ctx.tok_seq[2] = -1                      # a padding row: no output, nothing appended
        qkv = qkv0.clone()
        out = torch.full((B, H * D), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.FUSE_ROPE_DECODE = fused
        try:
            ops.rope_attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window, rot,
                               write_cache=write_cache)
        finally:
            ops.FUSE_ROPE_DECODE = True
        results.append((out, kp, vp))
    (o1, k1, v1), (o2, k2, v2) = results
    assert torch.equal(o1, o2), f"outputs differ by {(o1.float() - o2.float()).abs().max().item()}"
    assert torch.equal(k1, k2) and torch.equal(v1, v2)
    assert (o1[3].float().abs() > 0).any() and torch.equal(o1[2], torch.full_like(o1[2], 7.0))


@pytest.mark.parametrize("H,K,D,B", [(8, 4, 64, 50), (8, 4, 64, 90), (4, 4, 128, 80), (2, 2, 256, 160), (24, 1, 64, 200)])
def test_attention_decode_many_sequences(H, K, D, B):
    """More (sequence, head) pairs than processors: the smaller CTAs, several rounds each; lengths
    from one key to several rounds' worth, with a window on top."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    lengths = [1 + (37 * b * b + 11 * b) % 700 for b in range(B)]
    table, kp, vp = make_paged(lengths, sum(-(-n // 64) for n in lengths) + 3, K, D, torch.bfloat16, seed=B)
    qkv = rnd(B, (H + 2 * K) * D, dtype=torch.bfloat16, seed=17)
    check = sorted(set([0, 1, B // 2, B - 1, max(range(B), key=lambda b: lengths[b])]))
    ks, vs = {}, {}
    for b, n in enumerate(lengths):
        kk, vv = rnd(n, K, D, dtype=torch.bfloat16, seed=18 + b), rnd(n, K, D, dtype=torch.bfloat16, seed=931 + b)
        fill_cache(table.cpu(), kp, vp, b, kk, vv)
        if b in check:
            ks[b], vs[b] = kk, vv
    ctx = decode_ctx(lengths)
    q = qkv.double().cpu().view(B, H + 2 * K, D)[:, :H]
    for window in (0, 100):
        out = torch.empty(B, H * D, dtype=torch.bfloat16, device="cuda")
        ops.attention(qkv, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5, window)
        for b in check:
            want = ref_attention(q[b:b + 1], ks[b].double().cpu(), vs[b].double().cpu(), [lengths[b] - 1], D ** -0.5, window)
            close(out[b].view(1, H, D), want, "bfloat16", f"sequence {b} of {lengths[b]}, window {window}")


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("M,N,K", [(2500, 2100, 328), (4000, 3000, 200), (130, 300, 4104), (256, 256, 64), (20000, 700, 520)])
def test_gemm_tc_persistent(M, N, K, pair):
    """The persistent form of the tcgen05 product: more tiles than processors (a CTA walks several,
    both accumulator buffers in turn), ragged edges in every direction, both output types; `pair`: on
    pairs of processors (tiles of 256 x 256 by `tcgen05.mma.cta_group::2`)."""
    from alpacca_b200 import ops
    x, w, bias = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(N, seed=3)
    want = x.double() @ w.double().T + bias.double()
    for dt, tol in ((torch.float32, "float32"), (torch.bfloat16, "bfloat16")):
        out = torch.full((M, N), 9.0, dtype=dt, device="cuda")
        ops.gemm_tc(x, w, out, bias=bias, swap=False, bn=256, slices=1, pair=pair)
        close(out, want, tol, f"persistent gemm_tc {dt}")
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("M,F,K", [(3000, 1304, 264), (1024, 512, 2048)])
def test_gemm_tc_persistent_swiglu(M, F, K, pair):
    from alpacca_b200 import ops
    x = rnd(M, K, dtype=torch.bfloat16, seed=1)
    gate, up = rnd(F, K, dtype=torch.bfloat16, seed=2, scale=K ** -0.5), rnd(F, K, dtype=torch.bfloat16, seed=3, scale=K ** -0.5)
    bg, bu = rnd(F, seed=4), rnd(F, seed=5)
    w = torch.cat([gate.view(F // 8, 8, K), up.view(F // 8, 8, K)], dim=1).reshape(2 * F, K).contiguous()
    bias = torch.cat([bg.view(F // 8, 8), bu.view(F // 8, 8)], dim=1).reshape(2 * F).contiguous()
    g = x.double() @ gate.double().T + bg.double()
    u = x.double() @ up.double().T + bu.double()
    out = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc(x, w, out, bias=bias, swiglu=True, swap=False, pair=pair)
    close(out, g / (1 + torch.exp(-g)) * u, "bfloat16", "persistent swiglu epilogue")
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("K", [1, 3, 16, 17, 33, 48, 513, 1021])
@pytest.mark.parametrize("M,N", [(5, 33), (20, 130), (70, 130), (200, 1100)])
def test_gemm_f32_ragged_k(M, N, K):
    """Last tiles of every fill, rows that are not 16-byte aligned, on every tile height.  Bound: as for the tiles' test."""
    from alpacca_b200 import ops
    a, w, bias = rnd(M, K, seed=1), rnd(N, K, seed=2), rnd(N, seed=3)
    want = a.double() @ w.double().T + bias.double()
    bound = 2.0 ** -22 * (a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] + bias.double().abs())
    out = torch.full((M + 1, N), 7.0, device="cuda")
    ops.gemm_f32(a, w, out, bias=bias, n_rows=M)
    assert ((out[:M].double() - want).abs() <= bound).all() and (out[M] == 7.0).all()


@pytest.mark.parametrize("M,K,largest", [(1, 96, True), (1, 96, False), (1, 2048, False), (16, 2048, True), (16, 2048, False),
                                         (40, 1100, True), (130, 513, True), (130, 513, False)])
def test_gemm_f32_extreme_numbers(M, K, largest):
    """Numbers that no bfloat16 holds (above its largest; with `largest`, in the first row), infinities and NaNs go where plain
    multiply-adds take them; numbers of very unlike sizes, and of one sign, keep the bound of the tiles' test."""
    from alpacca_b200 import ops
    N = 150
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2).abs()
    a *= torch.exp2(torch.randint(-30, 30, (M, K), generator=torch.Generator().manual_seed(3)).float()).cuda()
    a[:, 5], w[3, 7], w[4, 7] = 1.0, float("inf"), float("nan")
    if largest:
        a[0, 9], w[:, 9] = 3.4e38, 1e-3
    if M > 1:
        a[M // 2, 11] = float("-inf")
    out = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, out)
    want = a.double() @ w.double().T
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isposinf(), want.isposinf())
    assert torch.equal(out.isneginf(), want.isneginf())
    at = want.isfinite()
    bound = 2.0 ** -22 * a.double().nan_to_num(0, 0, 0).norm(dim=1)[:, None] * w.double().nan_to_num(0, 0, 0).norm(dim=1)[None]
    assert ((out.double() - want).abs() <= bound)[at].all() and at.any()
    assert ops.gemm_f32_status() == 0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("page", [1, 5, 8, 12, 20])
@pytest.mark.parametrize("window", [0, 11])
def test_attention_simt_any_page_size(dtype, page, window):
    """Pages that hold no multiple of the eight keys that a warp takes at a time, and the smallest that do."""
    from alpacca_b200 import ops
    H, K, D, lengths, q_lens = 4, 2, 40, [37, 3, 60], [9, 3, 1]
    table, kp, vp = make_paged(lengths, sum(-(-n // page) for n in lengths) + 2, K, D, DT[dtype], page=page, seed=page)
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=DT[dtype], seed=3)
    ks = [rnd(n, K, D, dtype=DT[dtype], seed=4 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=DT[dtype], seed=8 + b) for b, n in enumerate(lengths)]
    for b, n in enumerate(lengths):
        for i in range(n):
            where = int(table[b, i // page])
            kp[where, :, i % page], vp[where, :, i % page] = ks[b][i], vs[b][i]
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32).cuda()
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32).cuda()
    out = torch.zeros(T, H * D, dtype=DT[dtype], device="cuda")
    ops.attention_simt(qkv, out, kp, vp, table, pos, seq, T, H, K, D, D ** -0.5, window)
    q = qkv.double().cpu().view(T, H + 2 * K, D)[:, :H]
    at = 0
    for b, n in enumerate(q_lens):
        want = ref_attention(q[at:at + n], ks[b].double().cpu(), vs[b].double().cpu(), pos[at:at + n].cpu(), D ** -0.5, window)
        close(out[at:at + n].view(n, H, D), want, dtype, f"sequence {b}")
        at += n


@pytest.mark.parametrize("H,K,D", [(4, 1, 64), (16, 2, 128)])
@pytest.mark.parametrize("window", [0, 11, 70])
@pytest.mark.parametrize("lengths,q_lens", [([37, 3, 130], [9, 3, 1]), ([200], [200]), ([33, 64, 1, 7], [33, 8, 1, 7]), ([65, 1, 32], [1, 1, 1])])
def test_attention_32bit_of_four_heads_has_the_same_bits(H, K, D, window, lengths, q_lens):
    """Eight tokens, or the heads of one, that share their keys against a warp per row: every sum is in the same order.  Rows without
    a sequence stay as they are, and values that are not numbers stay with the rows that see them."""
    from alpacca_b200 import ops
    table, kp, vp = make_paged(lengths, sum(-(-n // 64) for n in lengths) + 2, K, D, torch.float32, seed=5)
    kp.copy_(rnd(*kp.shape, seed=6))
    vp.copy_(rnd(*vp.shape, seed=7))
    vp[table[0, (lengths[0] - 1) // 64].item(), :, (lengths[0] - 1) % 64] = float("nan")      # the first sequence's last key
    T = sum(q_lens)
    qkv = 3 * rnd(T + 1, (H + 2 * K) * D, seed=8)
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)] + [torch.zeros(1)]).to(torch.int32).cuda()
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)] + [torch.full((1,), -1)]).to(torch.int32).cuda()
    cu_q = torch.tensor([sum(q_lens[:b]) for b in range(len(q_lens) + 1)], dtype=torch.int32).cuda()
    want, got, one = (torch.full((T + 1, H * D), 7.0, device="cuda") for _ in range(3))
    ops.attention_simt(qkv, want, kp, vp, table, pos, seq, T + 1, H, K, D, D ** -0.5, window)
    ops.attention_simt(qkv, got, kp, vp, table, pos, seq, T + 1, H, K, D, D ** -0.5, window, cu_q=cu_q)
    ops.attention_simt(qkv, one, kp, vp, table, pos, seq, T + 1, H, K, D, D ** -0.5, window, single=True)
    assert want[:T].isnan().any() and not want[:T].isnan().all()
    for x in (got, one):
        assert torch.equal(x.view(torch.int32), want.view(torch.int32)) or torch.equal(x.nan_to_num(9.0), want.nan_to_num(9.0))


@pytest.mark.parametrize("form,H,K,D", [("plain", 32, 8, 64), ("plain", 4, 4, 64), ("plain", 8, 2, 128), ("latent", 16, 1, 256),
                                        ("latent", 4, 1, 64)])
def test_prompt_attention_waits_for_its_last_products(form, H, K, D):
    """A prompt of many tiles on top of a held one, again and again: the same bits every time, and every row right.  A warp that
    reads its rows before the last products have landed leaves out up to 128 of their keys, more than an eighth of a row's norm.
    Bound: weights and outputs are rounded to 8 bits, 2^-9 each; random rows add up to about three times that, times 2.5."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    lengths, q_lens = [2200, 1500], [1490, 1500]
    table, kp, vp = make_paged(lengths, 62, K, D, torch.bfloat16, seed=H)
    kp.copy_(rnd(*kp.shape, seed=1))
    vp.copy_(rnd(*vp.shape, seed=2))
    T = sum(q_lens)
    cu = torch.tensor([0, q_lens[0], T], dtype=torch.int32).cuda()
    pos = torch.cat([torch.arange(n - q, n) for n, q in zip(lengths, q_lens)]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(2), torch.tensor(q_lens)).to(torch.int32).cuda()
    ctx = SimpleNamespace(tok_pos=pos, tok_seq=seq, n_tokens=T, n_seqs=2, cu_q=cu, is_decode=False,
                          kv_len=torch.tensor(lengths, dtype=torch.int32).cuda(), host_q_lens=q_lens, host_kv_lens=lengths,
                          max_q_len=1500, max_kv_len=2200, extras={})
    x = rnd(T, (H + 2 * K if form == "plain" else H) * D, dtype=torch.bfloat16, seed=3)
    R = D // 8
    outs = []
    for _ in range(12):
        out = torch.zeros(T, H * D, dtype=torch.bfloat16, device="cuda")
        if form == "plain":
            ops.attention(x, out, KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5)
        else:
            ops.latent_attention_mma(x, out, KVLayerView(kp, None, table, None), ctx, H, D - R, R, D ** -0.5)
        outs.append(out.view(T, H, D) if form == "plain" else out.view(T, H, D)[..., :D - R])
    ops.check_tc_status()
    assert all(torch.equal(o, outs[0]) for o in outs)
    q = x.view(T, -1, D)[:, :H].double()
    for b in range(2):
        at = slice(int(cu[b]), int(cu[b + 1]))
        keys, values = (p[table[b].long()].transpose(1, 2).reshape(-1, K, D)[:lengths[b]].double()
                        for p in (kp, vp if form == "plain" else kp))
        hidden = torch.arange(lengths[b], device="cuda")[None] > pos[at, None]
        for h in range(H):
            p = torch.softmax((q[at, h] @ keys[:, h * K // H].T * D ** -0.5).masked_fill(hidden, -math.inf), -1)
            want = (p @ values[:, h * K // H])[:, :outs[0].shape[-1]]
            err = (outs[0][at, h].double() - want).norm(dim=1) / want.norm(dim=1)
            assert err.max().item() < 2.0 ** -6, (b, h)


@pytest.mark.parametrize("M,K", [(1, 96), (16, 2048), (40, 1100), (130, 513)])
@pytest.mark.parametrize("small,large", [(-105, 100), (-112, 100), (-120, 100), (-126, 120), (-140, 110), (-149, 60), (-65, -65), (-75, -70)])
def test_gemm_f32_small_numbers(M, K, small, large):
    """Numbers whose last bits lie below bfloat16's smallest, down to subnormal ones, times large ones, and products that are
    subnormal themselves.  Bound: that of the tiles' test, and half a last place of the smallest number for the result."""
    from alpacca_b200 import ops
    N = 150
    a, w = (rnd(M, K, seed=1).double() * 2.0 ** small).float(), (rnd(N, K, seed=2).double() * 2.0 ** large).float()
    a[:, ::5] = 0.0
    out = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, out)
    want = a.double() @ w.double().T
    bound = 2.0 ** -22 * a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] + 2.0 ** -150
    assert want.abs().max() > 0 and ((out.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("M,N", [(1, 40), (16, 129), (33, 300), (70, 64), (200, 1000)])
@pytest.mark.parametrize("K", [1, 2, 5, 16, 31, 40, 47])
def test_gemm_f32_of_few_k_rounds_as_its_chains_do(M, N, K):
    """Few k are two chains of multiply-adds, over the even and the odd k, added at the end: formed here in 64 bits (a product of
    two 32-bit numbers is exact there) and rounded after every step.  Only where that rounds twice may the last bit differ."""
    from alpacca_b200 import ops
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    a *= torch.exp2(torch.randint(-20, 20, (M, K), generator=torch.Generator().manual_seed(3)).float()).cuda()
    out, out1 = torch.empty(M, N, device="cuda"), torch.empty(1, N, device="cuda")
    ops.gemm_f32(a, w, out)
    ops.gemm_f32(a[M // 2:M // 2 + 1].contiguous(), w, out1)
    chain = [torch.zeros(M, N, device="cuda"), torch.zeros(M, N, device="cuda")]
    for k in range(K):
        chain[k % 2] = (chain[k % 2].double() + a[:, k, None].double() * w[None, :, k].double()).float()
    want = chain[0] + chain[1]
    assert torch.equal(out1[0], out[M // 2])
    assert (out != want).float().mean().item() < 1e-3 and (out - want).abs().max() <= 2.0 ** -20 * want.abs().max()


@pytest.mark.parametrize("M,N,K", [(1, 300, 2048), (16, 129, 96), (20, 300, 513), (33, 40, 250), (60, 2100, 2048), (97, 300, 1100),
                                   (130, 20000, 260), (200, 150, 64), (256, 2100, 2048)])
@pytest.mark.parametrize("every", [False, True])
def test_gemm_f32_forms_what_is_not_finite_again(M, N, K, every):
    """Rows of either operand with an infinity or a NaN, and a row whose sums are beyond 2^96, on every tile height, alone and
    shared by clusters: the former give what 64-bit sums give, the latter keep the tiles' test's bound, all others their bits.
    `every`: each row of A has a NaN or an infinity."""
    from alpacca_b200 import ops
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2).abs()
    clean, out = torch.empty(M, N, device="cuda"), torch.full((M + 1, N), 7.0, device="cuda")
    ops.gemm_f32(a, w, clean)
    w[N // 3, K // 2], w[N - 1, 0] = float("inf"), float("nan")
    touched = torch.zeros(M, dtype=torch.bool, device="cuda")
    touched[M // 2] = True
    a[M // 2] *= 2.0 ** 98
    if M > 2:
        a[0, K - 1], a[M - 1, 3] = float("-inf"), float("nan")
        touched[0] = touched[M - 1] = True
    if every:
        a[::2, 1], a[1::2, K // 3], touched[:] = float("nan"), float("inf"), True
    ops.gemm_f32(a, w, out, n_rows=M)
    want = a.double() @ w.double().T
    got = out[:M]
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and (out[M] == 7.0).all()
    assert torch.equal(got.isneginf(), want.isneginf())
    finite = want.isfinite()
    bound = 2.0 ** -22 * a.double().nan_to_num(0, 0, 0).norm(dim=1)[:, None] * w.double().nan_to_num(0, 0, 0).norm(dim=1)[None]
    assert ((got.double() - want).abs() <= bound)[finite].all()
    same = finite & ~touched[:, None]
    assert torch.equal(got[same], clean[same])
    assert ops.gemm_f32_status() == 0


@pytest.mark.parametrize("dtype,H,K,D", [("float32", 4, 1, 64), ("float32", 16, 2, 128), ("float32", 3, 3, 72), ("bfloat16", 6, 2, 72)])
@pytest.mark.parametrize("window", [0, 30])
def test_attention_32bit_of_scores_of_minus_infinity(dtype, H, K, D, window):
    """Keys whose score is -inf get no weight, also where they are the first ones, a whole run of eight or all but one; a row that
    sees no others is not a number.  The same in every form of the kernel, and what 64-bit arithmetic gives."""
    from alpacca_b200 import ops
    lengths, q_lens = [70, 20, 9], [70, 20, 9]
    table, kp, vp = make_paged(lengths, 5, K, D, DT[dtype], seed=2)
    ks = [rnd(n, K, D, dtype=DT[dtype], seed=4 + b) for b, n in enumerate(lengths)]
    vs = [rnd(n, K, D, dtype=DT[dtype], seed=7 + b) for b, n in enumerate(lengths)]
    for b, gone in enumerate([list(range(17)) + list(range(24, 40)) + [55], list(range(19)), [8]]):
        ks[b][gone, :, 0] = float("-inf")            # every query is positive there
        fill_cache(table.cpu(), kp, vp, b, ks[b], vs[b])
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, dtype=DT[dtype], seed=3)
    qkv.view(T, -1, D)[:, :, 0] = qkv.view(T, -1, D)[:, :, 0].abs() + 0.1
    pos = torch.cat([torch.arange(n) for n in lengths]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(3), torch.tensor(q_lens)).to(torch.int32).cuda()
    cu = torch.tensor([0, 70, 90, 99], dtype=torch.int32).cuda()
    outs = []
    for form in ({}, {"cu_q": cu}, {"single": True}):
        out = torch.empty(T, H * D, dtype=DT[dtype], device="cuda")
        ops.attention_simt(qkv, out, kp, vp, table, pos, seq, T, H, K, D, D ** -0.5, window, **form)
        outs.append(out.float().nan_to_num(9.0))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    q = qkv.double().cpu().view(T, -1, D)[:, :H]
    t0 = 0
    for b, n in enumerate(lengths):
        want = ref_attention(q[t0:t0 + n], ks[b].double().cpu(), vs[b].double().cpu(), pos[t0:t0 + n].cpu(), D ** -0.5, window)
        assert want.isnan().any() == (b < 2) and not want.isnan().all()
        close(outs[0][t0:t0 + n].view(n, H, D), want.nan_to_num(9.0), dtype, f"sequence {b}")
        t0 += n


@pytest.mark.parametrize("H,K,D", [(16, 4, 64), (16, 2, 128)])
@pytest.mark.parametrize("n,tokens,longest", [(9, 1, 100), (24, 1, 100), (48, 1, 100), (130, 1, 100), (150, 1, 9), (70, 2, 90),
                                              (70, 9, 60), (33, 4, 200), (12, 3, 200)])
def test_attention_32bit_forms_have_the_same_bits(H, K, D, n, tokens, longest):
    """Up to 148 blocks of one token, up to 444 and more; sequences of few tokens token by token or in runs, more of them than a
    warp has lanes; sequences of up to eight keys among the others: all as row by row."""
    from alpacca_b200 import ops
    lengths = [max(tokens, 1 + (longest * (7 * b + 3)) % (longest + 1)) for b in range(n)]
    q_lens = [max(1, tokens - b % 3) for b in range(n)]
    table, kp, vp = make_paged(lengths, sum(-(-x // 64) for x in lengths), K, D, torch.float32, seed=1)
    kp.copy_(rnd(*kp.shape, seed=2))
    vp.copy_(rnd(*vp.shape, seed=3))
    T = sum(q_lens)
    qkv = rnd(T, (H + 2 * K) * D, seed=4)
    pos = torch.cat([torch.arange(x - q, x) for x, q in zip(lengths, q_lens)]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(q_lens)).to(torch.int32).cuda()
    cu = torch.tensor([0] + torch.tensor(q_lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    outs = []
    for form in [{}, {"cu_q": cu}] + ([{"single": True}] if tokens == 1 else []):
        out = torch.full((T, H * D), 7.0, device="cuda")
        ops.attention_simt(qkv, out, kp, vp, table, pos, seq, T, H, K, D, D ** -0.5, 20 if longest == 60 else 0, **form)
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs) and not (outs[0] == 7.0).any()


@pytest.mark.parametrize("M,rows_per_tile", [(1, 16), (20, 32), (64, 64), (96, 96)])
@pytest.mark.parametrize("K,runs", [(1000, 8), (700, 6), (420, 4), (300, 3)])
def test_gemm_f32_bits_do_not_depend_on_how_runs_are_shared(M, rows_per_tile, K, runs):
    """All runs of a tile in one CTA (many tiles), where the sums of the runs before wait in tensor memory, against a run per CTA
    (few tiles): the same bits, and right.  Bound: that of the tiles' test."""
    import ctypes
    from alpacca_b200 import ops
    N, narrow = 32 * 4008, slice(17 * 128, 17 * 128 + 150)
    plans = []
    for cols in (N, 150):
        plan = (ctypes.c_int * 4)()
        ops._lib("gemm_f32").ab_gemm_f32_plan(M, cols, K, plan)
        plans.append(tuple(plan))
    assert plans[0][1:] == (rows_per_tile, 8, 1) and plans[1][1:] == (rows_per_tile, 1, runs), plans
    a, w = rnd(M, K, seed=1), rnd(4008, K, seed=2)
    wide, out = torch.empty(M, N, device="cuda"), torch.empty(M, 150, device="cuda")
    ops.gemm_f32(a, w.repeat(32, 1), wide)
    ops.gemm_f32(a, w[narrow].contiguous(), out)
    assert torch.equal(wide[:, narrow], out) and torch.equal(wide.view(M, 32, 4008), wide[:, None, :4008].expand(M, 32, 4008))
    wide = wide[:, :4008]
    bound = 2.0 ** -22 * a.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None]
    assert ((wide.double() - a.double() @ w.double().T).abs() <= bound).all()
    assert ops.gemm_f32_status() == 0


@pytest.mark.parametrize("n", [3, 40])
def test_attention_32bit_of_a_step_that_only_names_its_tokens(n):
    """The 32-bit attention needs of a step its tokens' sequences and positions, not where the sequences begin; steps of up to
    eight keys and longer ones give the bits of the same step with everything named."""
    from alpacca_b200 import ops
    from alpacca_b200.cache import KVLayerView
    from types import SimpleNamespace
    H, K, D = 8, 2, 64
    table, kp, vp = make_paged([n], 2, K, D, torch.float32, seed=1)
    kp.copy_(rnd(*kp.shape, seed=2))
    vp.copy_(rnd(*vp.shape, seed=3))
    qkv = rnd(n, (H + 2 * K) * D, seed=4)
    pos, seq = torch.arange(n, dtype=torch.int32).cuda(), torch.zeros(n, dtype=torch.int32).cuda()
    named = dict(is_decode=False, n_seqs=1, cu_q=torch.tensor([0, n], dtype=torch.int32).cuda(), max_kv_len=n)
    outs = []
    for more in ({}, named):
        ctx = SimpleNamespace(tok_pos=pos, tok_seq=seq, n_tokens=n, **more)
        outs.append(torch.empty(n, H * D, device="cuda"))
        ops.attention(qkv, outs[-1], KVLayerView(kp, vp, table, None), ctx, H, K, D, D ** -0.5)
    assert torch.equal(outs[0], outs[1])
    want = ref_attention(qkv.double().cpu().view(n, -1, D)[:, :H], *(p[table[0].long()].transpose(1, 2).reshape(-1, K, D)[:n].double().cpu()
                                                                     for p in (kp, vp)), pos.cpu(), D ** -0.5)
    close(outs[0].view(n, H, D), want, "float32")
