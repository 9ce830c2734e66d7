"""Which path a call takes, and that it is the same call on every one of them: the forms that a dispatch rule chooses between,
layers whose parts a program has replaced or watches, sizes at which a launch runs into a limit, host threads."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from kch_b200 import synthetic as syn  # noqa: E402
from oracle import kch_oracle as orc  # noqa: E402

DEV = "cuda:0"


@pytest.fixture(scope="module")
def kch():
    import kch_b200
    from kch_b200 import _lib
    _lib.load()
    yield kch_b200
    assert _lib.device_status() == 0, "a bounded device-side wait expired"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("c", [8, 16, 32, 64, 128, 256])
def test_row_norms_do_not_depend_on_the_form(kch, dtype, c):
    """Rows on 16-byte boundaries (several a warp) and the same rows elsewhere (a warp a row): the squares are summed in one order, so
    norms and quotients have the same bits."""
    from kch_b200 import _lib
    lib = _lib.load()
    rows = 1003
    x = torch.randn(rows, c, generator=torch.Generator().manual_seed(c)).to(dtype).to(DEV)
    wide = torch.zeros(rows, c + 9, dtype=dtype, device=DEV)
    wide[:, :c] = x
    got = []
    for t, ld in ((x, c), (wide, c + 9)):
        y, n = torch.empty(rows, c, device=DEV), torch.empty(rows, device=DEV)
        _lib.check(lib.kch_rownorm(_lib.ptr(t), ld, _lib.ptr(y), _lib.ptr(n), rows, c, _lib.dtype_tag(dtype), _lib.KCH_F32, 0))
        got.append((y, n))
    torch.cuda.synchronize()
    assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][0], got[1][0])


def _many_heads(seed, T=4096):
    ins = list(syn.kda_inputs(seed, 4, T, 16, 128, 128, 16, torch.bfloat16, with_state=True))
    ins[3] = (ins[3].float() * 0.1).bfloat16()
    return [x.to(DEV) for x in ins]


def _chunk(kch, ins):
    return kch.naive_chunk_kda(*ins[:5], initial_state=ins[5], output_final_state=True, chunk_size=64)


def test_kda_parts_from_several_threads(kch):
    """Calls that go in parts over the side stream, from three host threads on streams of their own: each gets its own results."""
    import threading
    ins = [_many_heads(70 + i) for i in range(3)]
    want = [_chunk(kch, x) for x in ins]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(12):
                    o, s = _chunk(kch, ins[i])
                    if not (torch.equal(o, want[i][0]) and torch.equal(s, want[i][1])):
                        bad.append(i)
        except Exception as e:      # noqa: BLE001 (reported by the assertion below)
            bad.append(repr(e))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_kda_parts_beside_a_capture(kch):
    """A call in parts is captured, and before the capture ends another stream makes the same kind of call: that one runs at once, the
    captured one when it is replayed."""
    import threading
    a, b = _many_heads(80), _many_heads(81)
    want = [_chunk(kch, x) for x in (a, b)]
    torch.cuda.synchronize()
    graph, got, err = torch.cuda.CUDAGraph(), [], []

    def beside():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got.append(_chunk(kch, b))
        except Exception as e:      # noqa: BLE001
            err.append(repr(e))
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        first = _chunk(kch, a)
        t = threading.Thread(target=beside)
        t.start()
        t.join()
        second = _chunk(kch, a)
    torch.cuda.synchronize()
    assert not err, err
    assert torch.equal(got[0][0], want[1][0]) and torch.equal(got[0][1], want[1][1])
    graph.replay()
    torch.cuda.synchronize()
    for r in (first, second):
        assert torch.equal(r[0], want[0][0]) and torch.equal(r[1], want[0][1])


@pytest.mark.parametrize("B,H,HV,gate_scale", [(1, 1, 1, 0.1), (3, 2, 4, 0.1), (37, 8, 8, 1.0)])
def test_kda_step_gate_matches_the_two_launches(kch, B, H, HV, gate_scale):
    """The step that projects its gate against the recurrence on the gate of the same products, rounded at the layer's three points.
    The only liberty is the order of the 128 products: a pre-activation within 2^-17 (128 x 2^-24) of the middle between two
    bf16 values may round to the other one.  Channels whose pre-activation is not that close agree as two fp32 recurrences do:
    1e-5 of values below 10."""
    from kch_b200.kda import step_gate
    q, k, v, _, beta, S0 = (x.to(DEV) for x in syn.kda_inputs(B + HV, B, 1, H, 128, 128, HV, torch.bfloat16, with_state=True))
    gen = torch.Generator().manual_seed(B)
    x = torch.randn(B, 1, 128, generator=gen).bfloat16().to(DEV)
    W = (torch.randn(HV * 128, 128, generator=gen) * 0.08).bfloat16().to(DEV)
    t = (x.double() @ W.double().T).view(B, 1, HV, 128)
    tr = t.bfloat16()                                     # one rounding of the exact sum
    ulp = torch.ldexp(torch.ones_like(t), (torch.frexp(t).exponent - 8).int())
    away = (t - tr.double()).abs()
    close = (ulp * 0.5 - away) <= 2.0 ** -17 * (x.double().abs() @ W.double().abs().T).view_as(t)
    sp = torch.nn.functional.softplus(tr.double())
    spr = sp.bfloat16()
    ulp2 = torch.ldexp(torch.ones_like(sp), (torch.frexp(sp).exponent - 8).int())
    close |= (ulp2 * 0.5 - (sp - spr.double()).abs()) <= 2.0 ** -20 * sp.clamp_min(1.0)      # (the intrinsic logarithm)
    g = (-spr.float() * gate_scale).bfloat16()
    g = torch.where(close, torch.zeros_like(g), g)
    # channels that may go either way leave the comparison: no state, no key, no query there
    keep = ~close.any(dim=2, keepdim=True)                # [B, 1, 1, 128]
    q, k = q * keep, k * keep
    S0 = S0 * keep.view(B, 1, 128, 1)
    assert float(keep.float().mean()) > 0.5
    o, S = step_gate(q, k, v, x, W, beta, scale=128 ** -0.5, initial_state=S0, state_out=None, gate_scale=gate_scale)
    o2, S2 = kch.naive_recurrent_kda(q, k, v, g, beta, scale=128 ** -0.5, initial_state=S0, output_final_state=True)
    assert float((S - S2).abs().max()) <= 1e-5, float((S - S2).abs().max())
    assert bool(((o.float() - o2.float()).abs() <= 1e-5 + o2.float().abs() * 2.0 ** -8).all())


@pytest.mark.parametrize("state", [True, False])
def test_kda_parts_of_many_heads(kch, state):
    """64 heads and 65 chunks: too many heads for segments side by side, so the sequence goes in four parts, prepared on the caller's
    stream and scanned on another, the state carried through memory (the caller's final state, or the workspace where none is
    wanted).  Bounds as in test_kda_chunk_segments: operands in two bf16 terms."""
    B, T, H = 4, 4100, 16
    ins = list(syn.kda_inputs(64, B, T, H, 128, 128, H, torch.bfloat16, with_state=True))
    S0 = ins.pop() if state else (ins.pop(), None)[1]
    ins[3] = (ins[3].float() * 0.1).bfloat16()
    d = [x.to(DEV) for x in ins]
    S0d = None if S0 is None else S0.to(DEV)
    o, s = kch.naive_chunk_kda(*d, initial_state=S0d, output_final_state=True, chunk_size=64)
    o_only, none = kch.naive_chunk_kda(*d, initial_state=S0d, output_final_state=False, chunk_size=64)
    assert none is None and torch.equal(o, o_only)

    def check(o, s, o_ref, s_ref):
        assert float((s.double() - s_ref).norm() / s_ref.norm()) <= 1e-4
        e = (o.double() - o_ref).abs()
        assert bool((e <= o_ref.abs() * 2.0 ** -7 + 5e-4 * o_ref.abs().max().clamp_min(1.0)).all()), float(e.max())
    o2, s2 = kch.naive_recurrent_kda(*d, initial_state=S0d, output_final_state=True)
    check(o, s, o2.double(), s2.double())
    for b, h in ((0, 0), (3, 15)):                        # heads do not meet: two of them against the oracle in 64 bits
        one = [x[b:b + 1, :, h:h + 1].double() for x in ins]
        o_ref, s_ref = orc.chunk_kda(*one, initial_state=None if S0 is None else S0[b:b + 1, h:h + 1].double(), chunk_size=64)
        check(o[b:b + 1, :, h:h + 1].cpu(), s[b:b + 1, h:h + 1].cpu(), o_ref, s_ref)


def test_kda_chain_and_segments_agree(kch, tmp_path):
    """512 chunks of two heads as one chain (KCH_KDA_SPLIT=0 in a child process) and in segments: both against the oracle."""
    import os
    import subprocess
    import sys
    B, T, H = 1, 32768, 2
    q, k, v, g, beta = syn.kda_inputs(512, B, T, H, 128, 128, H, torch.bfloat16)
    g = (g.float() * 0.1).bfloat16()
    ins, outs = tmp_path / "in.pt", tmp_path / "out.pt"
    torch.save((q, k, v, g, beta), ins)
    code = ("import sys, torch\nsys.path.insert(0, sys.argv[3])\nimport kch_b200\n"
            "t = [x.cuda() for x in torch.load(sys.argv[1])]\n"
            "o, s = kch_b200.naive_chunk_kda(*t, output_final_state=True, chunk_size=64)\n"
            "assert kch_b200._lib.device_status() == 0\ntorch.save((o.cpu(), s.cpu()), sys.argv[2])\n")
    pkg = os.path.dirname(os.path.dirname(kch.__file__))
    subprocess.run([sys.executable, "-c", code, str(ins), str(outs), pkg], check=True, env=dict(os.environ, KCH_KDA_SPLIT="0"), timeout=300)
    o_ref, s_ref = orc.chunk_kda(*(x.double() for x in (q, k, v, g, beta)), chunk_size=64)
    seg = kch.naive_chunk_kda(*(x.to(DEV) for x in (q, k, v, g, beta)), output_final_state=True, chunk_size=64)
    for o, s in (torch.load(outs), [x.cpu() for x in seg]):
        assert float((s.double() - s_ref).norm() / s_ref.norm()) <= 1e-4
        e = (o.double() - o_ref).abs()
        assert bool((e <= o_ref.abs() * 2.0 ** -8 + 5e-4 * o_ref.abs().max().clamp_min(1.0)).all()), float(e.max())


@pytest.mark.parametrize("B,T,H", [(4, 4096, 16), (1, 8175, 64), (1, 4033, 50)])
def test_kda_chunks_over_and_over(kch, B, T, H):
    """The scan's hand-overs between its warps hold whatever a warp is held up by: many calls back to back, beside the prepare stage of
    their next part or call, with the same bits from each and no wait that expires."""
    ins = list(syn.kda_inputs(90 + H, B, T, H, 128, 128, H, torch.bfloat16, with_state=True))
    ins[3] = (ins[3].float() * 0.1).bfloat16()
    d = [x.to(DEV) for x in ins]
    want = _chunk(kch, d)
    for _ in range(8):
        got = [_chunk(kch, d) for _ in range(8)]
        torch.cuda.synchronize()
        assert kch._lib.device_status() == 0
        assert all(torch.equal(o, want[0]) and torch.equal(s, want[1]) for o, s in got)


@pytest.mark.parametrize("total", [95.5, 96.5, 150.0, 191.0, 193.0])
@pytest.mark.parametrize("growth", [0.0, 1e-5, 0.02])
def test_kda_chunks_at_the_lines_of_the_centre(kch, total, growth):
    """Chunks whose decay (2^-total in every second channel, a few units in the others) lies on either side of where the exponents are
    centred half way and of where that is not enough, with a gate that never grows, hardly, or does for 20 tokens.  Two chunks
    and a tail, 64 heads (one chain).  Bounds as in test_kda_chunk_segments."""
    B, T, H = 2, 150, 32
    q, k, v, g, beta, S0 = syn.kda_inputs(int(total), B, T, H, 128, 128, H, torch.bfloat16, with_state=True)
    gf = g.float() * 0.1
    gf[..., ::2] = -total * 0.6931471805599453 / 64
    if growth:
        gf[:, 70:90, :, 1::4] = growth
    g = gf.bfloat16()
    o, s = kch.naive_chunk_kda(*(x.to(DEV) for x in (q, k, v, g, beta)), initial_state=S0.to(DEV), output_final_state=True, chunk_size=64)
    for b, h in ((0, 0), (1, 31)):
        one = [x[b:b + 1, :, h:h + 1].double() for x in (q, k, v, g, beta)]
        o_ref, s_ref = orc.recurrent_kda(*one, initial_state=S0[b:b + 1, h:h + 1].double())
        assert float((s[b:b + 1, h:h + 1].double().cpu() - s_ref).norm() / s_ref.norm()) <= 1e-4
        e = (o[b:b + 1, :, h:h + 1].double().cpu() - o_ref).abs()
        assert bool((e <= o_ref.abs() * 2.0 ** -8 + 5e-4 * o_ref.abs().max().clamp_min(1.0)).all()), float(e.max())


@pytest.mark.parametrize("c,m,blocks", [(128, 64, 300), (128, 100, 300), (33, 128, 600), (33, 100, 600), (64, 64, 600), (65, 72, 400)])
def test_compression_of_many_long_blocks(kch, c, m, blocks):
    """More than 1184 groups of 32 channels, blocks on either side of the lengths from which their rows are shared between warps, with
    the overlap and without, and widths that leave lanes idle.  Bound as in test_compress_subsets."""
    g = torch.Generator().manual_seed(c + m)
    t = [torch.randn(2, blocks * m, c, generator=g) for _ in range(4)]
    t[2][1, -m:], t[3][0, m:2 * m] = -1e30, 40.0
    Ba, Bb = [torch.randn(m, c, generator=g) * 0.3 for _ in range(2)]
    a = kch.csa_compress_kv_overlapped(*[x.to(DEV) for x in t], Ba.to(DEV), Bb.to(DEV), m)
    assert float((a.double().cpu() - orc.compress_kv_overlapped(*t, Ba, Bb, m).double()).abs().max()) <= 2e-6
    b = kch.csa_compress_kv(t[0].to(DEV), t[2].to(DEV), Ba.to(DEV), m)
    assert float((b.double().cpu() - orc.compress_kv(t[0], t[2], Ba, m).double()).abs().max()) <= 2e-6


def _small(kch, seed=3, T=70):
    cfg = kch.HybridConfig(d_model=64, n_heads_qk=2, n_heads_v=2, head_dim_k=32, head_dim_v=32, csa_nh=2, csa_c=32, csa_dc=32, csa_nIh=2,
                           csa_cI=16, csa_m=4, csa_topk=4, csa_sliding_window=8, hca_m2=16, hca_nh=2, hca_c=32, hca_dc=32,
                           hca_sliding_window=8)
    model = kch.HybridKCHAttention(cfg, 5)
    model.load_state_dict(syn.hybrid_params(seed, cfg, 5, dtype=torch.float32, random_sink=True), strict=True)
    return model.to(DEV).eval(), syn.hidden_states(seed + 1, 2, T, cfg.d_model, torch.float32).to(DEV)


def _served(kch, model, x):
    dec = kch.HybridDecoding(model=model)
    dec.reset()
    return torch.cat([dec(x[:, :60]), dec(x[:, 60:69]), dec(x[:, 69:])], 1)


@pytest.mark.parametrize("where", [0, 3, 4])
def test_a_layer_whose_forward_is_replaced_is_called_as_it_always_was(kch, where):
    """A ``forward`` put on one layer of the stack: it gets the arguments that it got before the layers' own keywords came, for CSA
    and HCA the normalised input, and its result is the sub-layer's."""
    model, x = _small(kch)
    want = model(x)
    layer, seen = model.layers[where], []
    plain = type(layer).forward if where else type(layer).forward_functional
    if where == 0:          # the stack calls a KDA layer's functional form
        def functional(x, state, lookback, *, residual=None, norm=None):
            seen.append(x)
            return plain(layer, x, state, lookback, residual=residual, norm=norm)
        layer.forward_functional = functional
    else:
        def forward(x, state=None, residual=None):
            seen.append(x)
            return plain(layer, x, state, residual)
        layer.forward = forward
    model.reset_state()
    got = model(x)
    assert len(seen) == 1 and torch.equal(got, want)


def test_a_kda_layer_whose_projection_is_replaced(kch):
    """``project`` put on a KDA layer is what its passes run, over several tokens and over one."""
    model, x = _small(kch)
    layer, calls = model.layers[1], []
    own = type(layer).project
    want = _served(kch, model, x)

    def project(x, conv_lookback, lookback_in_place=False, norm=None, raw_gate=False):
        calls.append(x.shape[1])
        return own(layer, x, conv_lookback, lookback_in_place, norm, raw_gate)
    layer.project = project
    got = _served(kch, model, x)
    assert calls == [60, 9, 1] and torch.equal(got, want)


@pytest.mark.parametrize("how", ["instance", "hook", "pre_hook", "every"])
@pytest.mark.parametrize("path", ["stack", "served"])
def test_a_watched_or_replaced_norm_runs(kch, how, path):
    """The pre-norms of the CSA and HCA layers, replaced on the instance, hooked, or hooked for all modules: what the program put there
    takes part in every pass."""
    model, x = _small(kch)
    run = (lambda: model(x)) if path == "stack" else (lambda: _served(kch, model, x))
    base = run()
    model.reset_state()
    calls, handles = [], []
    for norm in (model.norms[3], model.norms[4]):
        if how == "instance":
            def forward(h, _n=norm):
                calls.append(h.shape[1])
                return type(_n).forward(_n, h) * 2.0
            norm.forward = forward
        elif how == "hook":
            handles.append(norm.register_forward_hook(lambda mod, a, out: (calls.append(a[0].shape[1]), out * 2.0)[1]))
        elif how == "pre_hook":
            handles.append(norm.register_forward_pre_hook(lambda mod, a: (calls.append(a[0].shape[1]), (a[0].flip(-1),))[1]))
    if how == "every":
        watched = {id(model.norms[3]), id(model.norms[4])}
        handles.append(torch.nn.modules.module.register_module_forward_hook(
            lambda mod, a, out: (calls.append(a[0].shape[1]), out * 2.0)[1] if id(mod) in watched else None))
    try:
        got = run()
    finally:
        for h in handles:
            h.remove()
    assert calls == ([70, 70] if path == "stack" else [60, 60, 9, 9, 1, 1])
    assert float((got - base).abs().max()) > 1e-3


def test_hooks_for_all_modules_see_the_layers(kch):
    """A hook registered for all modules meets the CSA and HCA layers with the input they always had, the normalised one."""
    model, x = _small(kch)
    want, seen = model(x), []
    model.reset_state()
    types = (type(model.layers[3]), type(model.layers[4]))
    h = torch.nn.modules.module.register_module_forward_pre_hook(lambda mod, a: seen.append(a[0]) if isinstance(mod, types) else None)
    try:
        got = model(x)
    finally:
        h.remove()
    assert torch.equal(got, want) and len(seen) == 2
    for s in seen:
        assert float(s.mean(-1).abs().max()) <= 1e-5 and abs(float(s.var(-1, unbiased=False).mean()) - 1.0) <= 1e-3


@pytest.mark.parametrize("T", [1, 5, 70])
def test_an_unknown_kda_backend_is_refused_for_every_length(kch, T):
    """A backend set after the configuration was made is named by the first pass, over one token, few or many."""
    model, x = _small(kch)
    model.cfg.kda_backend = "fla"
    with pytest.raises(ValueError, match="kda_backend='fla'"):
        model(x[:, :T])


def _peak(f):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    f()
    torch.cuda.synchronize()
    return torch.cuda.max_memory_allocated() - base


@pytest.mark.parametrize("kind", ["kda", "csa", "hca"])
@pytest.mark.parametrize("B,T", [(1, 4096), (2, 16384)])
def test_layer_calls_hold_no_more_memory_than_the_steps(kch, monkeypatch, kind, B, T):
    """A layer of width 1024 as one call and step by step.  The one call allocates its output before its intermediate results instead
    of behind them, and rounds each of those (a dozen) up to 512 bytes: that much more at its peak and no further; calls whose
    intermediate results pass the limit of the one-call form hold what the steps hold."""
    from kch_b200 import layers
    cfg = kch.HybridConfig(d_model=1024, n_heads_qk=8, n_heads_v=8, head_dim_k=128, head_dim_v=128, csa_nh=8, csa_c=128, csa_dc=128,
                           csa_nIh=4, csa_cI=64, csa_m=4, csa_topk=512, csa_sliding_window=128, hca_m2=128, hca_nh=8, hca_c=128,
                           hca_dc=128, hca_sliding_window=128)
    model = kch.HybridKCHAttention(cfg, 5).bfloat16().to(DEV).eval()
    i = {"kda": 0, "csa": 3, "hca": 4}[kind]
    layer, norm = model.layers[i], model.norms[i]
    x = syn.hidden_states(5, B, T, cfg.d_model, torch.bfloat16).to(DEV)

    def run():
        with torch.no_grad():
            if kind == "kda":
                return layer.forward_functional(x, None, None, residual=x, norm=norm)
            return layer(x, None, residual=x, norm=norm)
    run()
    names = ("csa_layer", "hca_layer", "kda_layer")
    own, taken = {n: getattr(layers, n) for n in names}, []
    for n in names:
        monkeypatch.setattr(layers, n, lambda *a, _f=own[n], **kw: (lambda got: (taken.append(got is not None), got)[1])(_f(*a, **kw)))
    one = _peak(run)
    for n in names:
        monkeypatch.setattr(layers, n, lambda *a, **kw: None)
    steps = _peak(run)
    assert one <= steps + (B * T * cfg.d_model * 2 + 16 * 512 if taken[0] else 0), (one, steps, taken)
    if (B, T) == (2, 16384):
        for n in names:
            monkeypatch.setattr(layers, n, own[n])
        monkeypatch.setattr(layers, "WORKSPACE_LIMIT", 1 << 20)
        assert _peak(run) <= steps


def test_bench_line_has_the_products():
    """The bench line's ``roofline`` is that of the products of a pass: five layers have three (KDA: projection, gate, output) or
    three (CSA, HCA: input, queries, output) each, whichever way the layers are issued."""
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, os.path.join(root, "bench.py"), "--batch", "1", "--seq-len", "512", "--steps", "2", "--warmup", "3",
                        "--no-decode", "--no-cpu-baseline"], capture_output=True, text=True, timeout=300, check=True)
    roof = json.loads(r.stdout.strip().splitlines()[-1])["roofline"]
    assert roof["launches"] == 2 * 15 and roof["achieved"] > 0 and sum(s["launches"] for s in roof["shapes"]) == roof["launches"]
    # 131072 tokens of the default workload have 131072 / 512 times these
    per_token = sum(2.0 * n * k for n, k in [(6288, 2048), (2048, 128), (2048, 2048)] * 3)
    assert roof["flops_per_step"] > 512 * per_token


@pytest.mark.parametrize("T", [64, 131])
@pytest.mark.parametrize("change", [
    dict(csa_nh=17, hca_nh=17), dict(csa_nh=16, hca_nh=16), dict(csa_c=64, hca_c=64), dict(csa_c=12, hca_c=20, csa_nh=1), dict(csa_cI=32),
    dict(csa_topk=0), dict(csa_topk=200), dict(csa_sliding_window=0, hca_sliding_window=0), dict(d_model=264), dict(d_model=2304),
    dict(d_model=512, dtype="fp32"), dict(head_dim_k=64, head_dim_v=64), dict(kda_chunk_size=16), dict(kda_decay_scale=0.0), dict(scale=16.5)],
    ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_the_rules_of_the_one_call_layers_are_those_of_the_steps(kch, monkeypatch, change, T):
    """Which key type, which form of the queries, of the norm and of the gate a layer takes is decided once in Python and once in the
    library: on both sides of each of those lines the one call gives the bits of the steps."""
    from kch_b200 import layers
    change = dict(change)
    dtype = torch.float32 if change.pop("dtype", "") == "fp32" else torch.bfloat16
    scale = change.pop("scale", 1.0)
    geo = dict(d_model=256, n_heads_qk=1, n_heads_v=2, head_dim_k=128, head_dim_v=128, csa_nh=2, csa_c=128, csa_dc=64, csa_nIh=2, csa_cI=64,
               csa_m=4, csa_topk=16, csa_sliding_window=16, hca_m2=16, hca_nh=2, hca_c=128, hca_dc=64, hca_sliding_window=16)
    cfg = kch.HybridConfig(**{**geo, **change})
    model = kch.HybridKCHAttention(cfg, 5)
    model.load_state_dict(syn.hybrid_params(7, cfg, 5, dtype=dtype, random_sink=True), strict=True)
    model = model.to(dtype).to(DEV).eval()
    x = syn.hidden_states(8, 2, T, cfg.d_model, dtype).to(DEV)
    c, h = model.layers[3], model.layers[4]

    def run():
        y, S, lbs = model.forward_functional(x, None, [None] * 3)
        ws = [getattr(c, n).weight for n in ("W_aKV", "W_bKV", "W_aZ", "W_bZ")]
        a = kch.naive_csa(x, *ws, c.Ba, c.Bb, c.W_DQ.weight, c.W_UQ.weight, c.W_IUQ.weight, c.W_w.weight, c.W_KV_idx.weight, c.W_Z_idx.weight,
                          c.B_idx, m=cfg.csa_m, topk=cfg.csa_topk, nh=cfg.csa_nh, nIh=cfg.csa_nIh, c=cfg.csa_c, c_I=cfg.csa_cI, dc=cfg.csa_dc,
                          scale=scale, sliding_window=cfg.csa_sliding_window, use_ste=False, normalize_qk=True)
        b = kch.naive_hca(x, h.W_KV.weight, h.W_Z.weight, h.B_pos, h.W_DQ.weight, h.W_UQ.weight, m2=cfg.hca_m2, nh=cfg.hca_nh, c=cfg.hca_c,
                          dc=cfg.hca_dc, scale=scale, sliding_window=cfg.hca_sliding_window, sink_logits=h.sink)
        return [y, S, *lbs, a, b]
    with torch.no_grad():
        one = run()
        for name in ("csa_layer", "hca_layer", "kda_layer"):
            monkeypatch.setattr(layers, name, lambda *a, **kw: None)
        steps = run()
    for got, want in zip(one, steps):
        assert torch.equal(got, want), float((got.double() - want.double()).abs().max())


@pytest.mark.parametrize("what", ["kda.forward_functional", "kda.project", "csa.forward", "csa.core", "hca.forward", "hca.core", "norm.forward"])
@pytest.mark.parametrize("path", ["stack", "served"])
def test_methods_replaced_on_the_class_run(kch, monkeypatch, what, path):
    """The same for a method that a program replaces on the class, with the arguments that it had before the layers' own keywords."""
    if path == "served" and what in ("csa.forward", "hca.forward"):
        pytest.skip("a served session calls the operators of these layers")
    model, x = _small(kch)
    run = (lambda: model(x)) if path == "stack" else (lambda: _served(kch, model, x))
    want = run()
    model.reset_state()
    kind, name = what.split(".")
    cls = type(model.norms[0] if kind == "norm" else model.layers[{"kda": 0, "csa": 3, "hca": 4}[kind]])
    own, calls = getattr(cls, name), []
    if name == "core":
        def method(self, x, *, return_projections=False, q_rows=None):
            calls.append(x.shape[1])
            return own(self, x, return_projections=return_projections, q_rows=q_rows)
    elif name == "project":
        def method(self, x, conv_lookback, lookback_in_place=False, norm=None, raw_gate=False):
            calls.append(x.shape[1])
            return own(self, x, conv_lookback, lookback_in_place, norm, raw_gate)
    elif name == "forward_functional":
        def method(self, x, state, lookback, *, residual=None, state_out=None, lookback_in_place=False, norm=None):
            calls.append(x.shape[1])
            return own(self, x, state, lookback, residual=residual, state_out=state_out, lookback_in_place=lookback_in_place, norm=norm)
    elif kind == "norm":
        def method(self, x):
            calls.append(x.shape[1])
            return own(self, x)
    else:
        def method(self, x, state=None, residual=None):
            calls.append(x.shape[1])
            return own(self, x, state, residual)
    monkeypatch.setattr(cls, name, method)
    got = run()
    assert torch.equal(got, want)
    per = {"kda": 3, "csa": 1, "hca": 1, "norm": 5}[kind]
    lengths = [70] if path == "stack" else [60] if name == "core" else [60, 9, 1]      # (a later chunk does not call `core`)
    if kind == "norm":                                     # fp32: LayerNorm and conv are two kernels, so all five norms run
        assert sorted(calls) == sorted(lengths * per)
    else:
        assert calls == [n for n in lengths for _ in range(per)]
