"""Edges of the ranges that the kernels' dispatch rules accept: remainders of tiles, smallest and largest sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from kch_b200 import synthetic as syn  # noqa: E402
from oracle import kch_oracle as orc  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module")
def kch():
    import kch_b200
    return kch_b200


def md(a, b):
    return float((a.double().cpu() - b.double().cpu()).abs().max()) if a.numel() else 0.0


@pytest.mark.parametrize("B,T,H,HV,K,V,chunk,gate", [
    (1, 65, 1, 2, 128, 128, 64, "decay"), (2, 200, 2, 2, 64, 64, 64, "decay"), (1, 130, 1, 1, 65, 20, 64, "decay"),
    (1, 64, 2, 4, 5, 3, 4, "decay"), (1, 63, 1, 1, 128, 130, 16, "decay"), (1, 7, 1, 1, 16, 8, 3, "decay"),
    (1, 150, 1, 1, 128, 64, 64, "mixed"), (1, 100, 1, 1, 32, 32, 64, "clamped")])
def test_kda_chunk_fp32_edges(kch, B, T, H, HV, K, V, chunk, gate):
    """The fp32 chunk kernels pad to 64 tokens, 64 / 128 channels and 8 value columns.  Sums of at most 128 + 64 fp32
    products per chunk step: 2e-5 of values around 1, as for the golden cases."""
    q, k, v, g, beta, S0 = syn.kda_inputs(5 * T + K, B, T, H, K, V, HV, torch.float32, with_state=True)
    if gate == "mixed":           # one chunk with a growing gate takes the pair-by-pair exponents
        g[:, 70:80] = 0.02
    if gate == "clamped":         # far below the clamp: every factor underflows
        g = g * 40
    o_ref, s_ref = orc.recurrent_kda(*(x.double() for x in (q, k, v, g, beta)), initial_state=S0.double())
    o, s = kch.naive_chunk_kda(*(x.to(DEV) for x in (q, k, v, g, beta)), initial_state=S0.to(DEV), output_final_state=True,
                               chunk_size=chunk)
    assert md(o, o_ref) <= 2e-5 and md(s, s_ref) <= 2e-5, (md(o, o_ref), md(s, s_ref))


@pytest.mark.parametrize("T,K,chunk,lo,hi,growth", [
    (100, 64, 16, 10, 60, 1.0), (130, 64, 64, 0, 64, 1.0), (150, 64, 48, 20, 110, 0.6), (64, 16, 64, 0, 40, 2.0),
    (100, 64, 32, 10, 60, 1.5), (70, 64, 3, 0, 60, 1.0)])
def test_kda_chunk_fp32_growing_gate(kch, T, K, chunk, lo, hi, growth):
    """Where half of the channels grow for a while, exponents are clamped within a chunk of min(chunk_size, 64, K) tokens and
    exact between chunks, whatever the kernels pack together.  Values reach 1e32; the chunk form in 32 bits on the CPU is up to
    1.5e-6 (2-norm, relative) from 64 bits here, ten times that is allowed."""
    q, k, v, g, beta, S0 = syn.kda_inputs(3, 1, T, 1, K, 8, 1, torch.float32, with_state=True)
    g[:, lo:hi, :, :K // 2] = growth
    o_ref, s_ref = orc.chunk_kda(*(x.double() for x in (q, k, v, g, beta)), initial_state=S0.double(), chunk_size=min(chunk, 64, K))
    o, s = kch.naive_chunk_kda(*(x.to(DEV) for x in (q, k, v, g, beta)), initial_state=S0.to(DEV), output_final_state=True,
                               chunk_size=chunk)
    for got, want in ((o, o_ref), (s, s_ref)):
        assert float((got.double().cpu() - want).norm() / want.norm()) <= 1.5e-5


def _attend_ref(q, comp, sel, win, m, t0, nvis, window, sink, scale, win_t0):
    """One softmax over the selected (or all visible) rows, the window and the sink, in 64 bits on the GPU."""
    B, T, nh, c = q.shape
    n = comp.shape[1]
    q, comp, win, out = q.double(), comp.double(), win.double(), torch.zeros(B, T, nh, c, dtype=torch.float64, device=DEV)
    q = q / q.norm(dim=-1, keepdim=True).clamp_min(1e-12)
    for t in range(T):
        v = min(n, nvis if nvis >= 0 else (t0 + t + 1) // m)
        lo = max(0, t + win_t0 - window + 1)
        for b in range(B):
            ids = torch.arange(v, device=DEV) if sel is None else sel[b, t][(sel[b, t] >= 0) & (sel[b, t] < v)].long()
            keys = torch.cat([comp[b, ids], win[b, lo:t + win_t0 + 1] if window else comp[b, :0]])
            s = torch.cat([q[b, t] @ keys.T * scale, sink.double()[:, None]], 1)
            out[b, t] = torch.softmax(s, -1)[:, :-1] @ keys if len(keys) else 0
    return out.reshape(B, T, nh * c)


@pytest.mark.parametrize("B,T,nh,n,topk,m,t0,nvis,window,scale,odd", [
    (1, 70, 16, 300, 40, 1, 200, -1, 128, 1.0, None), (2, 33, 8, 130, 130, 4, 400, -1, 16, 1.0, None),
    (1, 17, 5, 64, 7, 4, 0, -1, 8, 4.0, None), (1, 9, 12, 65, 65, 1, 0, 65, 0, 1.0, None),
    (2, 40, 16, 2500, 30, 1, 900, -1, 20, 1.0, None), (1, 24, 16, 96, 20, 2, 100, -1, 32, 1.0, "nan"),
    (1, 24, 8, 96, 20, 2, 100, -1, 32, 1.0, "inf")])
def test_selection_as_mask_matches_gather(kch, B, T, nh, n, topk, m, t0, nvis, window, scale, odd):
    """A selection list applied as a bit mask over key tiles (few visible rows per selected one) or gathered (the case of 2500
    rows): operator outputs within 2e-3 of the 64-bit softmax, as everywhere.  Rows that a query does not attend do not reach
    it even when they are not finite."""
    from kch_b200.csa import attend
    g = torch.Generator(device=DEV).manual_seed(T * nh + n)
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s, generator=g, device=DEV), dim=-1).bfloat16()  # noqa: E731
    win_t0 = 3
    q, comp, win = torch.randn(B, T, nh, 128, generator=g, device=DEV).bfloat16(), unit(B, n, 128), unit(B, T + win_t0, 128)
    sink = torch.randn(nh, generator=g, device=DEV)
    sel = torch.full((B, T, topk), -1, dtype=torch.int32, device=DEV)
    for t in range(T):
        v = min(n, nvis if nvis >= 0 else (t0 + t + 1) // m)
        for b in range(B):
            ids = torch.randperm(v, generator=g, device=DEV)[:topk]
            sel[b, t, :len(ids)] = ids.int()
    bad = None
    if odd:                                   # a row that half of the queries select, and a token's window row
        bad = (sel == 5).any(-1)[0]
        comp[0, 5] = float(odd)
        win[0, 20] = float(odd)
        bad |= (torch.arange(T, device=DEV) + win_t0 >= 20) & (torch.arange(T, device=DEV) + win_t0 < 20 + window)
    kw = dict(nh=nh, c=128, sel=sel, m=m, t0=t0, n_visible=nvis, q_normalize=True, win=win, sliding_window=window, sink=sink,
              scale=scale, out_dtype=torch.bfloat16, win_t0=win_t0)
    a = attend(q.reshape(B, T, nh * 128), comp, sel_distinct=True, **kw)
    b = attend(q.reshape(B, T, nh * 128), comp, **kw)
    ref = _attend_ref(q, comp, sel, win, m, t0, nvis, window, sink, scale, win_t0)
    if odd:
        assert 0 < int(bad.sum()) < T
        assert not torch.isfinite(a[:, bad].float()).all(-1).any() and torch.isfinite(a[:, ~bad].float()).all()
        a, b, ref = a[:, ~bad], b[:, ~bad], ref[:, ~bad]
    assert md(a, ref) <= 2e-3 and md(b, ref) <= 2e-3, (md(a, ref), md(b, ref))
    if odd:                                   # without a list: a row that only the later half of the queries sees
        late = (t0 + T // 2) // m + 1
        comp = unit(B, n, 128)
        comp[0, late] = float(odd)
        pos = torch.arange(T, device=DEV)
        bad = ((t0 + pos + 1) // m > late) | ((pos + win_t0 >= 20) & (pos + win_t0 < 20 + window))
    dense = attend(q.reshape(B, T, nh * 128), comp, **dict(kw, sel=None))
    dref = _attend_ref(q, comp, None, win, m, t0, nvis, window, sink, scale, win_t0)
    if odd:
        assert 0 < int(bad.sum()) < T
        assert not torch.isfinite(dense[:, bad].float()).all(-1).any() and torch.isfinite(dense[:, ~bad].float()).all()
        dense, dref = dense[:, ~bad], dref[:, ~bad]
    assert md(dense, dref) <= 2e-3, md(dense, dref)


def test_selection_split_between_mask_and_gather(kch):
    """Enough queries to fill the chip, of which the first see few rows and the others many: the former take the mask, the
    latter the gather, in two launches.  Each form is within 2e-3 of the 64-bit softmax, so 4e-3 of each other."""
    from kch_b200.csa import attend
    B, T, nh, topk = 4, 4096, 16, 256
    g = torch.Generator(device=DEV).manual_seed(2)
    q = torch.randn(B, T, nh, 128, generator=g, device=DEV).bfloat16()
    comp = torch.nn.functional.normalize(torch.randn(B, T, 128, generator=g, device=DEV), dim=-1).bfloat16()
    sink = torch.randn(nh, generator=g, device=DEV)
    pos = torch.arange(T, device=DEV)
    score = torch.rand(B, T, T, generator=g, device=DEV).masked_fill_(pos[None, :] > pos[:, None], -1.0)
    top = score.topk(topk, -1)
    sel = torch.where(top.values >= 0, top.indices, -1).int()
    kw = dict(nh=nh, c=128, m=1, q_normalize=True, sink=sink, scale=1.0, out_dtype=torch.bfloat16)
    a, b = (attend(q.reshape(B, T, nh * 128), comp, sel=sel, sel_distinct=d, **kw) for d in (True, False))
    assert md(a, b) <= 4e-3, md(a, b)
    for t0 in (0, 6 * topk - 8, T - 8):                      # the line between the two lies at six visible rows per selected one
        ref = _attend_ref(q[:, t0:t0 + 8], comp, sel[:, t0:t0 + 8], comp[:, :0], 1, t0, -1, 0, sink, 1.0, 0)
        assert md(a[:, t0:t0 + 8], ref) <= 2e-3, md(a[:, t0:t0 + 8], ref)


@pytest.mark.parametrize("M,N", [(1, 256), (7, 400), (33, 6288), (64, 256)])
def test_decode_gemm_l2norm_rows(kch, M, N):
    """The 128-wide decode tiles deal their rows out over the CTAs of a cluster by the real row count."""
    from kch_b200 import _lib
    from kch_b200.csa import linear
    g = torch.Generator(device=DEV).manual_seed(M)
    x, W = torch.randn(M, 1, 2048, generator=g, device=DEV).bfloat16(), (torch.randn(N, 2048, generator=g, device=DEV) * 0.02).bfloat16()
    tail = N % 128
    segs = [(N - tail, _lib.ACT_SILU_L2NORM, 0.0)] + ([(tail, _lib.ACT_SIGMOID, 0.0)] if tail else [])
    y = linear(x, W, epilogue=segs, group=128)
    p = (x.double() @ W.double().T).bfloat16().double()
    ref = torch.nn.functional.silu(p[..., :N - tail]).bfloat16().double().unflatten(-1, (-1, 128))
    ref = (ref / ref.norm(dim=-1, keepdim=True).bfloat16().double()).flatten(-2)
    ref = torch.cat([ref, torch.sigmoid(p[..., N - tail:])], -1)
    # products within one bf16 rounding, then the rounding of the activation: 2^-7 of the value in all
    assert bool(((y.double() - ref).abs() <= 2 ** -7 * ref.abs() + 2e-3).all()), md(y, ref)


@pytest.mark.parametrize("B,nb,topk,quant", [(1, 40, 16, None), (3, 700, 300, "fp8"), (8, 1500, 1024, None), (70, 64, 64, "int8"),
                                             (2, 5000, 4500, None)])
def test_decode_attention_split_or_cluster(kch, B, nb, topk, quant):
    """Few entries per sequence are merged inside a cluster, many by a second launch; the indexer deals its key rows out by
    the batch.  Against the oracle of the cache: 2e-4 with bf16 rows, 2e-3 with 8-bit rows, as for the golden streams."""
    c, cI, m, win, nh, nI = 128, 64, 4, 32, 16, 4
    g = torch.Generator().manual_seed(nb)
    T = nb * m + 1
    w = [(torch.randn(B, T, x, generator=g)).bfloat16() for x in (c, c, c, c, cI, cI)]
    Ba, Bb, Bi = ((torch.randn(m, x, generator=g) * 0.02).bfloat16() for x in (c, c, cI))
    cache = kch.CSADecodingCache(B, c, cI, m, win, DEV, torch.bfloat16, kv_quant=quant)
    ref = orc.CSACacheOracle(B, c, cI, m, win, torch.bfloat16, quant)
    dw, db = [x.to(DEV) for x in w], [x.to(DEV) for x in (Ba, Bb, Bi)]
    cache.append_step(*(x[:, :-1] for x in dw), *db)
    cache.append_step(*(x[:, -1:] for x in dw), *db)
    ref.append(*(x[:, :-1] for x in w), Ba, Bb, Bi)
    ref.append(*(x[:, -1:] for x in w), Ba, Bb, Bi)
    q = torch.nn.functional.normalize(torch.randn(B, 1, nh, c, generator=g), dim=-1)
    qi, wi, sink = torch.randn(B, 1, nI, cI, generator=g), torch.randn(B, 1, nI, generator=g), torch.randn(nh, generator=g)
    out, sel = cache.forward_step(q.to(DEV), qi.to(DEV), wi.to(DEV), topk=topk, nh=nh, nIh=nI, scale=1.0, sink_logits=sink.to(DEV),
                                  use_ste=False, _return_indices=True)
    want = ref.step(q, qi, wi, topk=topk, sink_logits=sink, scale=1.0)
    assert (sel.sort(-1).values[:, 0, 1:] > sel.sort(-1).values[:, 0, :-1]).all()
    assert md(out, want) <= (2e-3 if quant else 2e-4), md(out, want)


@pytest.mark.parametrize("M,N,K", [(512, 136, 64), (513, 264, 128), (700, 776, 2048), (1153, 2304, 128), (640, 1016, 192)])
def test_large_gemm_bulk_store_edges(kch, M, N, K):
    """The bulk-tensor store clips rows beyond M and columns beyond N of a 256 x 256 tile; nothing around C is touched.  Products
    within one bf16 rounding of the 64-bit value."""
    from kch_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, W = torch.randn(M, K, generator=g, device=DEV).bfloat16(), (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    ref = x.double() @ W.double().T
    for ldc in (N, N + 24):
        C = torch.full((M + 2, ldc), 7.0, device=DEV, dtype=torch.bfloat16)
        lib = _lib.load()
        _lib.check(lib.kch_linear(_lib.ptr(x), _lib.ptr(W), C.data_ptr() + 2 * ldc, None, M, N, K, K, K, ldc, 0, _lib.KCH_BF16,
                                  _lib.stream()))
        got = C[1:-1, :N].double()
        assert bool(((got - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()), md(got, ref)
        assert bool((C[0] == 7).all() and (C[-1] == 7).all() and (C[1:-1, N:] == 7).all())


@pytest.mark.parametrize("M,N", [(520, 520), (1100, 400)])
def test_large_gemm_residual_and_activation_edges(kch, M, N):
    """Residual tiles arrive and leave by the copy engine; 128-column groups of one activation take its epilogue, mixed ones the
    general loop.  Product, activation and sum each round once to bf16."""
    from kch_b200 import _lib
    from kch_b200.csa import linear
    g = torch.Generator(device=DEV).manual_seed(M)
    x, W = torch.randn(M, 256, generator=g, device=DEV).bfloat16(), (torch.randn(N, 256, generator=g, device=DEV) / 16).bfloat16()
    R = torch.randn(M, N + 8, generator=g, device=DEV).bfloat16()[:, :N]
    p = (x.double() @ W.double().T).bfloat16().double()
    y = linear(x, W, residual=R)
    assert bool(((y.double() - (p + R.double())).abs() <= 2 ** -7 * (p.abs() + R.double().abs()) + 1e-5).all())
    segs = [(128, _lib.ACT_SILU_L2NORM, 0.0), (160, _lib.ACT_SILU, 0.0), (N - 288 - 16, 0, 0.0), (16, _lib.ACT_SIGMOID, 0.0)]
    if (N - 16) % 32:
        segs = [(128, _lib.ACT_SILU_L2NORM, 0.0), (160, _lib.ACT_SILU, 0.0), (N - 288, _lib.ACT_SIGMOID, 0.0)]
    y = linear(x, W, epilogue=segs, group=128)
    h = torch.nn.functional.silu(p[:, :128]).bfloat16().double()
    want = [h / h.norm(dim=-1, keepdim=True).bfloat16().double(), torch.nn.functional.silu(p[:, 128:288])]
    rest = p[:, 288:]
    want.append(torch.cat([rest[:, :-16], torch.sigmoid(rest[:, -16:])], 1) if len(segs) == 4 else torch.sigmoid(rest))
    want = torch.cat(want, 1)
    # the fp32 product may round to the neighbouring bf16 value (2^-7 of it), then silu, norm and result round (2^-9 to 2^-8 each)
    assert bool(((y.double() - want).abs() <= 2 ** -6 * want.abs() + 2e-3).all()), md(y, want)


@pytest.mark.parametrize("M,N", [(520, 520), (1100, 384)])
@pytest.mark.parametrize("act", ["SIGMOID", "NEG_SOFTPLUS"])
def test_large_gemm_wide_activation(kch, M, N, act):
    """Column groups of 128 with one elementwise activation leave by the copy engine, the ragged rest of N too.  Product,
    activation and result round to bf16 (2^-7 of the product, at most as much of the value, then 2^-8 each)."""
    from kch_b200 import _lib
    from kch_b200.csa import linear
    g = torch.Generator(device=DEV).manual_seed(M)
    x, W = torch.randn(M, 128, generator=g, device=DEV).bfloat16(), (torch.randn(N, 128, generator=g, device=DEV) / 6).bfloat16()
    p = (x.double() @ W.double().T).bfloat16().double()
    for cut in (N, 256):                     # all columns, or a second group without an activation
        segs = [(cut, getattr(_lib, "ACT_" + act), 0.5)] + ([(N - cut, 0, 0.0)] if cut < N else [])
        want = torch.sigmoid(p[:, :cut]) if act == "SIGMOID" else -0.5 * torch.nn.functional.softplus(p[:, :cut])
        want = torch.cat([want, p[:, cut:]], 1)
        y = linear(x, W, epilogue=segs)
        assert bool(((y.double() - want).abs() <= 2 ** -6 * want.abs() + 1e-4).all()), md(y, want)


@pytest.mark.parametrize("B,T,dtype", [(2, 131, "bf16"), (1, 517, "bf16"), (3, 130, "fp32"), (1, 9, "bf16"), (2, 3, "fp32")])
def test_ragged_lengths_without_padding(kch, B, T, dtype):
    """Lengths that are no multiple of a block (4 and 64 tokens) or of the indexer's query tile: same as the oracle, which pads.
    Operator outputs within 2e-3 (bf16) / 2e-5 (fp32); CSA on the kernel's own selection."""
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    kw = dict(nh=8, c=128, dc=64, nIh=4, c_I=64, m=4)
    w, sink, H = syn.csa_inputs(T, B, T, 256, **kw, dtype=dt, random_sink=True)
    args = dict(kw, topk=24, sliding_window=16, normalize_qk=True)
    dw = {k: v.to(DEV) for k, v in w.items()}
    out, idx = kch.naive_csa(H.to(DEV), *dw.values(), **args, sink_logits=sink.to(DEV), use_ste=False, _return_indices=True)
    ref = orc.csa_forward(H, *w.values(), **args, sink_logits=sink,
                          indices_override=torch.cat([idx.long().cpu(), idx.new_full((B, -T % 4, 24), -1).long().cpu()], 1))
    assert out.shape == ref.shape and md(out, ref) <= (2e-3 if dtype == "bf16" else 2e-5), md(out, ref)
    vis = (torch.arange(T) + 1) // 4
    assert bool(((idx.cpu() >= 0).sum(-1) == vis.clamp(max=24)).all()) and bool((idx.cpu() < vis[None, :, None].clamp(min=1)).all())
    w, sink, H = syn.hca_inputs(T + 1, B, T, 256, nh=8, c=128, dc=64, m2=64, dtype=dt, random_sink=True)
    kw = dict(m2=64, nh=8, c=128, dc=64, sliding_window=16)
    out = kch.naive_hca(H.to(DEV), *(v.to(DEV) for v in w.values()), **kw, sink_logits=sink.to(DEV))
    ref = orc.hca_forward(H, *w.values(), **kw, sink_logits=sink)
    assert out.shape == ref.shape and md(out, ref) <= (2e-3 if dtype == "bf16" else 2e-5), md(out, ref)


@pytest.mark.parametrize("B,win,quant,dtype,runs", [(1, 8, None, "bf16", (3, 2, 40, 3, 2)), (3, 5, "int8", "bf16", (1, 7, 3, 6)),
                                                    (2, 16, None, "fp32", (2, 130, 2, 9)), (2, 0, "fp8", "bf16", (5, 11))])
def test_bulk_append_leaves_the_cache_of_the_oracle(kch, B, win, quant, dtype, runs):
    """Runs that close no, one or many blocks, with and without an open one, shorter and longer than the window: what is copied
    is the same to the bit, rows within one rounding of the storage dtype (fp32: 4 ulp of the softmax sums)."""
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    c, cI, m, m2 = 128, 64, 4, 8
    rel = 2 ** -7 if dt == torch.bfloat16 else 2e-6          # neighbouring bf16 values are up to 2^-7 of the value apart
    g = torch.Generator().manual_seed(B)
    Ba, Bb, Bi, Bh = (torch.randn(r, x, generator=g).mul(0.1).to(dt) for r, x in ((m, c), (m, c), (m, cI), (m2, c)))
    csa, hca = kch.CSADecodingCache(B, c, cI, m, win, DEV, dt, kv_quant=quant), kch.HCADecodingCache(B, c, m2, win, DEV, dt, kv_quant=quant)
    rc, rh = orc.CSACacheOracle(B, c, cI, m, win, dt, quant), orc.HCACacheOracle(B, c, m2, win, dt, quant)
    for i, T in enumerate(runs):
        wide = torch.randn(B, T, 4 * c + 2 * cI, generator=g).to(dt)         # slices of one projection, as a module passes them
        if i % 2:
            wide = wide.transpose(0, 1).contiguous().transpose(0, 1)
        dev = wide.to(DEV)
        csa.append_step(*dev.split([c] * 4 + [cI] * 2, -1), *(x.to(DEV) for x in (Ba, Bb, Bi)))
        rc.append(*wide.split([c] * 4 + [cI] * 2, -1), Ba, Bb, Bi)
        hca.append_step(dev[..., :c], dev[..., 2 * c:3 * c], Bh.to(DEV))
        rh.append(wide[..., :c], wide[..., 2 * c:3 * c], Bh)
        for cache, ref, mm in ((csa, rc, m), (hca, rh, m2)):
            st, nb, rest = cache.export_state(), ref.tokens // mm, ref.tokens % mm
            assert (st["n_blocks"], st["acc_len"], st["n_tokens_seen"]) == (nb, rest, ref.tokens)
            assert cache._ctr.tolist()[:5] == [rest, nb, ref.tokens if win else 0, int(cache is csa and nb > 0), ref.tokens]
            assert all(torch.equal(a[:, :rest].cpu(), r) for a, r in zip(st["acc"], ref.acc))
            if win:
                k = min(win, ref.tokens)
                slots = torch.arange(ref.tokens - k, ref.tokens) % win
                got, want = st["ring"].cpu()[:, slots].float(), ref.window.float()
                assert bool(((got - want).abs() <= rel * want.abs() + 1e-7).all())
            if nb:
                if not quant:
                    got, want = st["comp"].cpu().float(), ref.C_comp.float()
                    assert bool(((got - want).abs() <= rel * want.abs() + 2e-6).all()), md(got, want)
                    assert bool(((st["norms"].cpu() - got.norm(dim=-1)).abs() <= 2e-6 * st["norms"].cpu()).all())
                if cache is csa:
                    assert torch.equal(st["prev"][0].cpu(), ref.prev_Cb) and torch.equal(st["prev"][1].cpu(), ref.prev_Zb)
                    got, want = st["kcomp"].cpu().float(), ref.K_IComp.float()
                    assert bool(((got - want).abs() <= rel * want.abs() + 2e-6).all())
                    assert bool(((st["kcomp_norms"].cpu() - got.norm(dim=-1)).abs() <= 2e-6 * got.norm(dim=-1)).all())


@pytest.mark.parametrize("M", [1, 7, 64])
@pytest.mark.parametrize("N,K", [(256, 64), (2304, 128), (2048, 2048)])
def test_settled_weights_give_the_same_product(kch, M, N, K):
    """Weights fetched before the launch before has finished, or after it: the same product to the bit."""
    from kch_b200.csa import linear
    g = torch.Generator(device=DEV).manual_seed(M + N)
    W, R = (torch.randn(N, K, generator=g, device=DEV) * 0.05).bfloat16(), torch.randn(M, 1, N, generator=g, device=DEV).bfloat16()
    for _ in range(5):
        x = torch.randn(M, 1, K, generator=g, device=DEV).bfloat16()
        assert torch.equal(linear(x, W, residual=R, w_settled=True), linear(x, W, residual=R))


_STEP_CFG = dict(d_model=512, n_heads_qk=4, n_heads_v=4, head_dim_k=128, head_dim_v=128, kda_chunk_size=64, csa_m=4, csa_topk=8,
                 csa_nh=16, csa_c=128, csa_dc=128, csa_nIh=4, csa_cI=64, csa_sliding_window=16, hca_m2=16, hca_nh=16, hca_c=128,
                 hca_dc=128, hca_sliding_window=16)


@pytest.mark.parametrize("names", [("q_proj", "W_aKV", "W_KV"), ("g_up",), ("W_UQ",), ("o_proj",), ("parametrised",)])
def test_weights_changed_between_one_token_steps(kch, names):
    """A step right after a change of weights in place (members of a fused projection, or read as they lie), or with weights
    computed when they are read, is the step of a model built with those weights, to the bit."""
    from torch.nn.utils import parametrize
    cfg = kch.HybridConfig(**_STEP_CFG)

    def model_of(params):
        with torch.device(DEV):
            m = kch.HybridKCHAttention(cfg, 5)
        m = m.bfloat16().eval()
        m.load_state_dict(params, strict=True)
        return m
    params = {k: v.to(DEV) for k, v in syn.hybrid_params(7, cfg, 5, dtype=torch.bfloat16).items()}
    x = syn.hidden_states(8, 3, 48, cfg.d_model, torch.bfloat16).to(DEV)

    class Twice(torch.nn.Module):
        def forward(self, w):
            return w * 2
    with torch.no_grad():
        model = model_of(params)
        a = kch.HybridDecoding(model=model)
        a.reset()
        a(x[:, :32])
        a(x[:, 32:33])
        for t in range(33, 41):
            st = a.export_state()
            st = {k: (v.clone() if torch.is_tensor(v) else v) for k, v in st.items()}
            if names == ("parametrised",):
                if t == 33:
                    for layer in model.layers:
                        for n in ("g_up", "W_UQ", "o_proj"):
                            if n in dict(layer.named_children()):
                                parametrize.register_parametrization(getattr(layer, n), "weight", Twice(), unsafe=True)
                changed = {k: v * 2 if k.split(".")[-2] in ("g_up", "W_UQ", "o_proj") else v for k, v in params.items()}
            else:
                changed = {k: v * (-1.5) ** (t - 32) if k.split(".")[-2] in names else v for k, v in params.items()}
                for k, w in model.named_parameters():
                    if k.split(".")[-2] in names:
                        w.copy_(changed[k])
            got = a(x[:, t:t + 1])
            b = kch.HybridDecoding(model=model_of(changed))
            b.import_state(st)
            assert torch.equal(got, b(x[:, t:t + 1])), t


@pytest.mark.parametrize("M,N,K,off", [(1, 1, 4, 0), (31, 63, 28, 4), (32, 64, 32, 0), (33, 65, 36, 0), (662, 840, 256, 0),
                                       (97, 128, 300, 8), (50, 130, 33, 0), (40, 64, 64, 1)])
@pytest.mark.parametrize("form", ["plain", "residual", "act", "norm"])
def test_linear_fp32_edges(kch, M, N, K, off, form):
    """Tiles of 32 x 64 with steps of 32 in K, operands that 16-byte copies cannot read (odd K, odd offset), and the activation
    segments in the epilogue.  A chain of K fused multiply-adds is off by at most K 2^-24 sum |a||w|; silu, sigmoid and
    softplus have slopes below 1.1 and add a few units in the last place of values below max(1, |x|)."""
    from kch_b200 import _lib
    from kch_b200.csa import linear
    gen = torch.Generator(device=DEV).manual_seed(M + N + K)
    wide = torch.randn(M, K + 2 * off + (-(K + 2 * off)) % (4 if off != 1 else 1), generator=gen, device=DEV)
    x = wide[:, off:off + K]
    W = torch.randn(N, K, generator=gen, device=DEV) * K ** -0.5
    y = x.double() @ W.double().T
    bound = 1.1 * K * 2.0 ** -24 * (x.double().abs() @ W.double().abs().T) + 2.0 ** -21 * y.abs().clamp_min(1.0)
    if form == "plain":
        got, ref = linear(x, W), y
    elif form == "residual":
        r = torch.randn(M, N, generator=gen, device=DEV)
        got, ref = linear(x, W, residual=r), y + r.double()
        bound = bound + 2.0 ** -23 * r.double().abs()
    elif form == "act":
        if N < 4:
            pytest.skip("four segments")
        c = [0, N // 4, N // 2, N // 2 + 1, N]
        acts = [(_lib.ACT_SILU, 0.0), (0, 0.0), (_lib.ACT_SIGMOID, 0.0), (_lib.ACT_NEG_SOFTPLUS, 0.1)]
        got = linear(x, W, epilogue=[(c[i + 1] - c[i], *acts[i]) for i in range(4)])
        ref = y.clone()
        ref[:, :c[1]] = torch.nn.functional.silu(y[:, :c[1]])
        ref[:, c[2]:c[3]] = torch.sigmoid(y[:, c[2]:c[3]])
        ref[:, c[3]:] = -0.1 * torch.nn.functional.softplus(y[:, c[3]:])
    else:
        if N % 64:
            pytest.skip("whole groups")
        for group in (64, 32, 16, 4):
            got = linear(x, W, epilogue=[(64, _lib.ACT_SILU_L2NORM, 0.0)] + ([(N - 64, _lib.ACT_SILU, 0.0)] if N > 64 else []), group=group)
            s = torch.nn.functional.silu(y)
            nrm = s[:, :64].unflatten(-1, (-1, group)).norm(dim=-1, keepdim=True)
            ref = s.clone()
            ref[:, :64] = (s[:, :64].unflatten(-1, (-1, group)) / nrm).flatten(1)
            # a quotient moves by the error of its numerator and of the norm, each relative to the norm
            e = bound[:, :64].unflatten(-1, (-1, group))
            b = bound.clone()
            b[:, :64] = ((e + e.norm(dim=-1, keepdim=True)) / nrm).flatten(1) + group * 2.0 ** -23
            assert bool(((got.double() - ref).abs() <= b).all()), group
        return
    assert bool(((got.double() - ref).abs() <= bound).all()), float(((got.double() - ref).abs() - bound).max())


@pytest.mark.parametrize("B,T,H,HV,K,V,dtype,off", [
    (2, 130, 4, 4, 128, 128, torch.float32, 0), (3, 70, 2, 4, 64, 100, torch.float32, 0), (2, 65, 4, 8, 64, 36, torch.bfloat16, 0),
    (1, 90, 2, 2, 64, 64, torch.bfloat16, 2), (1, 90, 1, 2, 128, 36, torch.float32, 1), (1, 67, 1, 1, 62, 38, torch.float32, 0)])
def test_kda_chunk_generic_columns(kch, B, T, H, HV, K, V, dtype, off):
    """Four or eight value columns per CTA of the scan (by the number of CTAs), columns that fill neither, and operands that loads
    of four elements cannot read (odd widths, an odd offset).  Bounds as in test_kda_chunk_fp32_edges; bf16 adds the rounding
    of the output."""
    ins = list(syn.kda_inputs(9 * T + V, B, T, H, K, V, HV, dtype, with_state=True))
    S0 = ins.pop()
    o_ref, s_ref = orc.recurrent_kda(*(x.double() for x in ins), initial_state=S0.double())
    if off:                       # the same values behind an odd offset
        ins = [torch.cat([x.new_zeros(off), x.flatten()]).to(DEV)[off:].view(x.shape) for x in ins]
    o, s = kch.naive_chunk_kda(*(x.to(DEV) for x in ins), initial_state=S0.to(DEV), output_final_state=True, chunk_size=64)
    assert md(s, s_ref) <= 2e-5, md(s, s_ref)
    d = (o.double().cpu() - o_ref).abs()
    assert bool((d <= 2e-5 + (o_ref.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0.0)).all()), float(d.max())


@pytest.mark.parametrize("B,T,H,HV,state,gate", [
    (1, 2049, 2, 2, True, "model"), (1, 3000, 1, 2, False, "model"), (1, 2500, 2, 2, True, "op"), (2, 1700, 1, 1, True, "mixed"),
    (1, 2049, 1, 2, True, "clamped"), (1, 2200, 1, 1, True, "grows"), (1, 129, 1, 1, True, "op"), (1, 2048, 1, 1, True, "none")])
def test_kda_chunk_segments(kch, B, T, H, HV, state, gate):
    """Few heads and many chunks: the segments of a sequence are scanned side by side.  Gates from the model's (-0.1 softplus)
    over the operator's own (a chunk decays by 2^-74 on average, past the half-way centre in some channels) to the clamp,
    none at all, and one that grows for 300 tokens (e^6: its segments run as one chain).  Operands in two bf16 terms: 2^-16
    relative to the values, which stay around 1 but for the growing gate; the output is rounded to bf16 once."""
    q, k, v, g, beta, S0 = syn.kda_inputs(T + HV, B, T, H, 128, 128, HV, torch.bfloat16, with_state=True)
    S0 = S0 if state else None
    gf = g.float()
    if gate == "model":
        gf = gf * 0.1
    elif gate == "mixed":                      # a run beyond 2^-192 a chunk, which the mma.sync stage prepares
        gf = gf * 0.3
        gf[:, 500:900] *= 12.0
    elif gate == "clamped":
        gf = gf * 40.0
    elif gate == "grows":
        gf = gf * 0.1
        gf[:, 700:1000] = 0.02
    elif gate == "none":
        gf = gf * 0.0
    g = gf.bfloat16()
    o_ref, s_ref = orc.recurrent_kda(*(x.double() for x in (q, k, v, g, beta)), initial_state=None if S0 is None else S0.double())
    o, s = kch.naive_chunk_kda(*(x.to(DEV) for x in (q, k, v, g, beta)), initial_state=None if S0 is None else S0.to(DEV),
                               output_final_state=True, chunk_size=64)
    assert kch._lib.device_status() == 0
    assert float((s.double().cpu() - s_ref).norm() / s_ref.norm()) <= 1e-4
    d = (o.double().cpu() - o_ref).abs()
    assert bool((d <= o_ref.abs() * 2.0 ** -8 + 5e-4 * o_ref.abs().max().clamp_min(1.0)).all()), float(d.max())


@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16),
                                       (torch.float32, torch.float32)])
@pytest.mark.parametrize("rows,c,ld,off", [(1, 8, 8, 0), (33, 16, 40, 0), (67, 128, 128, 0), (5, 256, 264, 8), (9, 264, 264, 0), (7, 24, 24, 0),
                                           (31, 128, 130, 0), (31, 128, 136, 1)])
def test_rownorm_rows(kch, dtype, out, rows, c, ld, off):
    """Rows of 8 to 256 elements on 16-byte boundaries (several rows a warp) and the others (a warp a row).  fp32 arithmetic: a sum
    of c squares, a root and a division, 2^-23 * (c / 8 + 8) of the value at most; a bf16 result is rounded once (eight
    significant bits: half a unit in the last place is up to 2^-8 of the value)."""
    from kch_b200 import _lib
    x = torch.randn(rows * ld + off, generator=torch.Generator().manual_seed(c)).to(dtype).to(DEV)[off:].view(rows, ld)
    x[rows // 2] = 0.0
    y, norms = torch.empty(rows, c, dtype=out, device=DEV), torch.empty(rows, device=DEV)
    _lib.check(_lib.load().kch_rownorm(_lib.ptr(x), ld, _lib.ptr(y), _lib.ptr(norms), rows, c, _lib.dtype_tag(dtype), _lib.dtype_tag(out), 0))
    torch.cuda.synchronize()
    ref_n = x[:, :c].double().norm(dim=-1).clamp_min(1e-12)
    ref, eps = x[:, :c].double() / ref_n.unsqueeze(-1), 2.0 ** -23 * (c / 8 + 8)
    assert bool(((norms.double() - ref_n).abs() <= eps * ref_n).all())
    assert bool(((y.double() - ref).abs() <= ref.abs() * (eps + (2.0 ** -8 if out == torch.bfloat16 else 0.0))).all())


@pytest.mark.parametrize("T,c,m", [(64, 33, 8), (7 * 9, 31, 9), (130, 1, 65), (21, 70, 7), (128, 32, 128), (9472, 32, 16), (9600, 5, 8)])
def test_compress_subsets(kch, T, c, m):
    """Blocks whose rows eight warps share (m >= 64, or m >= 8 and at most 1184 groups of 32 channels) and, on either side of that
    line, those that a thread walks; widths that fill no group.  Bound as in test_compress_matches_oracle, by the values: 2e-6."""
    g = torch.Generator().manual_seed(T + c)
    t = [torch.randn(2, T, c, generator=g) for _ in range(4)]
    t[2][0, :m], t[3][0, :m] = -1e30, 40.0
    Ba, Bb = [torch.randn(m, c, generator=g) * 0.3 for _ in range(2)]
    a = kch.csa_compress_kv_overlapped(*[x.to(DEV) for x in t], Ba.to(DEV), Bb.to(DEV), m)
    assert md(a, orc.compress_kv_overlapped(*t, Ba, Bb, m)) <= 2e-6
    b = kch.csa_compress_kv(t[0].to(DEV), t[2].to(DEV), Ba.to(DEV), m)
    assert md(b, orc.compress_kv(t[0], t[2], Ba, m)) <= 2e-6



@pytest.mark.parametrize("geometry,dtype,B,T", [
    ("small", torch.float32, 2, 97), ("small", torch.bfloat16, 1, 130), ("small", torch.float32, 1, 64), ("small", torch.bfloat16, 2, 20),
    ("wide", torch.bfloat16, 2, 203), ("wide", torch.bfloat16, 1, 129), ("wide", torch.float32, 1, 70), ("narrow", torch.float32, 1, 150)])
@pytest.mark.parametrize("path", ["stack", "prompt", "op"])
def test_layer_calls_match_the_steps(kch, monkeypatch, geometry, dtype, B, T, path):
    """The one-call form of the layers against the same launches issued one by one: the same kernels with the same arguments, so
    the same bits.  Lengths below and above the blocks and chunks, ragged ones, and a geometry whose widths are not multiples
    of 8 (which the calls leave to the steps)."""
    from kch_b200 import layers
    geo = {"small": dict(d_model=64, n_heads_qk=2, n_heads_v=4, head_dim_k=32, head_dim_v=16, csa_nh=4, csa_c=32, csa_dc=24, csa_nIh=2,
                         csa_cI=16, csa_m=16, csa_topk=3, csa_sliding_window=5, hca_m2=32, hca_nh=2, hca_c=32, hca_dc=16,
                         hca_sliding_window=0),
           "wide": dict(d_model=256, n_heads_qk=2, n_heads_v=2, head_dim_k=128, head_dim_v=128, csa_nh=4, csa_c=128, csa_dc=64, csa_nIh=2,
                        csa_cI=64, csa_m=4, csa_topk=16, csa_sliding_window=16, hca_m2=16, hca_nh=4, hca_c=128, hca_dc=64,
                        hca_sliding_window=16),
           "narrow": dict(d_model=36, n_heads_qk=1, n_heads_v=1, head_dim_k=12, head_dim_v=20, csa_nh=1, csa_c=12, csa_dc=10, csa_nIh=1,
                          csa_cI=6, csa_m=8, csa_topk=4, csa_sliding_window=3, hca_m2=16, hca_nh=1, hca_c=12, hca_dc=10,
                          hca_sliding_window=3)}[geometry]
    cfg = kch.HybridConfig(**geo)
    params = syn.hybrid_params(3, cfg, 5, dtype=dtype, random_sink=True)
    x = syn.hidden_states(4, B, T, cfg.d_model, dtype).to(DEV)
    model = kch.HybridKCHAttention(cfg, 5)
    model.load_state_dict(params, strict=True)
    model = model.to(dtype).to(DEV).eval()

    def run():
        if path == "stack":
            y, S, lbs = model.forward_functional(x, None, [None] * 3)
            return [y, S, *lbs, *model.forward_functional(x[:, : T // 2 + 2].contiguous(), S, lbs)[:2]]
        if path == "op":
            csa, hca = model.layers[3], model.layers[4]
            w = {k: getattr(csa, k).weight for k in ("W_aKV", "W_bKV", "W_aZ", "W_bZ")}
            got = kch.naive_csa(x, *w.values(), csa.Ba, csa.Bb, csa.W_DQ.weight, csa.W_UQ.weight, csa.W_IUQ.weight, csa.W_w.weight,
                                csa.W_KV_idx.weight, csa.W_Z_idx.weight, csa.B_idx, m=cfg.csa_m, topk=cfg.csa_topk, nh=cfg.csa_nh,
                                nIh=cfg.csa_nIh, c=cfg.csa_c, c_I=cfg.csa_cI, dc=cfg.csa_dc, sliding_window=cfg.csa_sliding_window,
                                sink_logits=csa.sink, use_ste=False, normalize_qk=True, return_projections=True)
            got2 = kch.naive_hca(x, hca.W_KV.weight, hca.W_Z.weight, hca.B_pos, hca.W_DQ.weight, hca.W_UQ.weight, m2=cfg.hca_m2,
                                 nh=cfg.hca_nh, c=cfg.hca_c, dc=cfg.hca_dc, sliding_window=cfg.hca_sliding_window, sink_logits=hca.sink,
                                 return_projections=True)
            return [got[0], *got[1], got2[0], *got2[1], csa(x)[0], hca(x, residual=x)[0]]
        dec = kch.HybridDecoding(model=model)
        dec.reset()
        out = [dec(x[:, : T - 7]), dec(x[:, T - 7: T - 1]), dec(x[:, T - 1:]), model._kda_state]
        for c in dec._caches.values():
            st = c.export_state()
            out += [t for t in (*st["acc"], st["comp"], st["norms"], st["ring"], *st.get("prev", []), st.get("kcomp"), c._ctr) if t is not None]
        return out
    with torch.no_grad():
        calls = {}
        for name in ("csa_layer", "hca_layer", "kda_layer"):
            def spy(*a, _f=getattr(layers, name), _n=name, **kw):
                got = _f(*a, **kw)
                calls[_n] = calls.get(_n, 0) + (got is not None)
                return got
            monkeypatch.setattr(layers, name, spy)
        one = run()
        if geometry != "narrow" and T >= 64:
            assert all(calls.get(n, 0) > 0 for n in (("csa_layer", "hca_layer") if path == "op" else ("csa_layer", "hca_layer", "kda_layer"))), calls
        for name in ("csa_layer", "hca_layer", "kda_layer"):
            monkeypatch.setattr(layers, name, lambda *a, **kw: None)
        steps = run()
    assert len(one) == len(steps)
    for a, b in zip(one, steps):
        assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b), (a.shape, float((a.double() - b.double()).abs().max()))


@pytest.mark.parametrize("B,H,HV,state,stride,settled", [(1, 1, 1, False, 0, True), (2, 4, 8, True, 8, False), (37, 8, 8, True, 0, True),
                                                         (37, 2, 4, True, 136, True), (18, 16, 16, False, 24, False)])
def test_kda_step_gate(kch, B, H, HV, state, stride, settled):
    """One token whose gate is projected in the same launch: from one head to the 296 that take that form, grouped heads, gate
    inputs that lie inside a wider row.  The pre-activation (|t| <= 5 here), its softplus and their product
    with the scale are rounded to bf16 each: the gate is within 7 * 2^-8 of itself, exp(gate) within 0.37 of that; the
    intrinsic exponential and logarithm stay far below a rounding."""
    from kch_b200.kda import step_gate, step_gate_supported
    assert step_gate_supported(B, HV, 128, 128, torch.bfloat16) and not step_gate_supported(297, 1, 128, 128, torch.bfloat16)
    q, k, v, _, beta, S0 = (x.to(DEV) for x in syn.kda_inputs(B + HV, B, 1, H, 128, 128, HV, torch.bfloat16, with_state=True))
    gen = torch.Generator().manual_seed(B)
    x = torch.randn(B, 1, 128 + stride, generator=gen).bfloat16().to(DEV)[..., stride // 16 * 8:][..., :128]
    W = (torch.randn(HV * 128, 128, generator=gen) * 0.08).bfloat16().to(DEV)
    S0 = S0 if state else None
    o, S = step_gate(q, k, v, x, W, beta, scale=128 ** -0.5, initial_state=S0, state_out=None, gate_scale=0.3, w_settled=settled)
    t = x.double() @ W.double().T
    assert float(t.abs().max()) <= 5.0
    decay = torch.exp((-0.3 * torch.nn.functional.softplus(t)).clamp(min=-10.0)).view(B, HV, 128, 1)
    qd, kd = (y.double()[:, 0].repeat_interleave(HV // H, 1) for y in (q, k))
    vd, bd = v.double()[:, 0], beta.double()[:, 0].unsqueeze(-1)
    prev = (torch.zeros(B, HV, 128, 128, device=DEV, dtype=torch.float64) if S0 is None else S0.double()) * decay
    S_ref = prev + kd.unsqueeze(-1) * (bd * (vd - torch.einsum("bhk,bhkv->bhv", kd, prev))).unsqueeze(-2)
    off = 0.37 * 7 * 2.0 ** -8 * (torch.zeros_like(prev) if S0 is None else S0.double().abs())
    off = off + kd.abs().unsqueeze(-1) * (bd * torch.einsum("bhk,bhkv->bhv", kd.abs(), off)).unsqueeze(-2)
    assert bool(((S.double() - S_ref).abs() <= off + 1e-5).all()), float(((S.double() - S_ref).abs() - off).max())
    o_ref = torch.einsum("bhk,bhkv->bhv", qd, S_ref) * 128 ** -0.5
    off = torch.einsum("bhk,bhkv->bhv", qd.abs(), off) * 128 ** -0.5 + o_ref.abs() * 2.0 ** -8
    assert bool(((o[:, 0].double() - o_ref).abs() <= off + 1e-5).all())
