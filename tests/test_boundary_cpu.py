"""Host-side checks that need no GPU: the C-ABI library loads and exports every symbol the header
declares, host validation rejects bad arguments with the reference's exception types before any
launch, CPU tensors are refused (no fallback), and the backend installer is reversible."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _header_symbols():
    src = open(os.path.join(ROOT, "include", "kch_b200.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(kch_[a-z0-9_]+)\s*\(", src)))


def test_library_exports_every_declared_symbol():
    from kch_b200 import _lib
    lib = _lib.load()
    syms = _header_symbols()
    assert len(syms) >= 18
    for s in syms:
        assert hasattr(lib, s), f"{s} declared in include/kch_b200.h but not exported"
        assert s in _lib.PROTOTYPES, f"{s} has no ctypes prototype"
    assert sorted(_lib.PROTOTYPES) == syms
    assert lib.kch_abi_version() == 1


def test_argument_errors_come_back_as_codes_without_a_gpu():
    from kch_b200 import _lib
    lib = _lib.load()
    # every one of these is rejected on the host before any CUDA call
    rc = lib.kch_compress_kv(None, None, None, None, 1, 10, 8, 0, 8, 10, 0, 0, 0, None)
    assert rc < 0 and b"m=0" in lib.kch_last_error()
    rc = lib.kch_compress_kv(None, None, None, None, 1, 10, 8, 4, 8, 10, 0, 0, 0, None)
    assert rc < 0 and b"divisible" in lib.kch_last_error()
    rc = lib.kch_kda_recurrent(*([None] * 8), 1, 4, 2, 3, 8, 8, 1.0, -10.0, 0, 0, 0, 0, 0, None)
    assert rc < 0 and b"HV=3" in lib.kch_last_error()
    rc = lib.kch_indexer_topk(None, None, None, None, 1, 4, 4, 2, 0, 3, 1.0, 4, 0, -1, 0, 0, None, 0, None)
    assert rc < 0 and b"c_I" in lib.kch_last_error()
    rc = lib.kch_linear(None, None, None, None, 4, 4, 4, 2, 4, 4, 0, 0, None)
    assert rc < 0 and b"lda" in lib.kch_last_error()
    with pytest.raises(ValueError, match="lda"):
        _lib.check(rc)
    assert lib.kch_kda_chunk_workspace_bytes(4, 32768, 16, 128, 128, 64) > 0
    assert lib.kch_indexer_workspace_bytes(1, 4096, 1024, 4, 32) == 4096 * 1024 * 4
    assert lib.kch_indexer_workspace_bytes(1, 4096, 1024, 4, 64) > 4096 * 1024 * 4


def test_cpu_tensors_are_refused_not_silently_computed():
    import kch_b200
    q = torch.randn(1, 4, 2, 8)
    with pytest.raises(RuntimeError, match="CUDA"):
        kch_b200.naive_recurrent_kda(q, q, q, q, torch.rand(1, 4, 2))
    with pytest.raises(RuntimeError, match="CUDA"):
        kch_b200.kda_forward(q, q, q, q, torch.rand(1, 4, 2))
    H = torch.randn(1, 8, 16)
    W = torch.randn(4, 16)
    with pytest.raises(RuntimeError, match="CUDA"):
        kch_b200.naive_hca(H, W, W, torch.zeros(4, 4), torch.randn(4, 16), torch.randn(8, 4), m2=4, nh=2, c=4, dc=4)
    with pytest.raises(RuntimeError, match="CUDA"):
        kch_b200.CSADecodingCache(1, 8, 4, 4, 4, "cpu", torch.float32)


def test_validation_matches_reference_types_and_names():
    import kch_b200
    q = torch.randn(1, 4, 2, 8)
    with pytest.raises(ValueError, match="rank"):
        kch_b200.naive_recurrent_kda(q[0], q, q, q, torch.rand(1, 4, 2))
    with pytest.raises(ValueError, match="beta"):
        kch_b200.naive_chunk_kda(q, q, q, q, torch.rand(1, 4, 3))
    with pytest.raises(ValueError, match="kda_backend"):
        kch_b200.kda_forward(q, q, q, q, torch.rand(1, 4, 2), backend="fla")
    with pytest.raises(TypeError):
        kch_b200.kda_forward(q, q, q, q, torch.rand(1, 4, 2), g_clamp_min="x")
    with pytest.raises(ValueError, match="m=0"):
        kch_b200.csa_compress_kv(torch.zeros(1, 4, 4), torch.zeros(1, 4, 4), torch.zeros(1, 4), 0)
    with pytest.raises(ValueError, match="topk"):
        kch_b200.csa_lightning_indexer(torch.zeros(1, 2, 1, 4), torch.zeros(1, 2, 4), None, -1)
    with pytest.raises(NotImplementedError):
        kch_b200.csa_lightning_indexer(torch.zeros(1, 2, 1, 4), torch.zeros(1, 2, 4), None, 1, ste_mode="aux_contrastive")
    with pytest.raises(ValueError, match="n_heads_v"):
        kch_b200.HybridConfig(n_heads_qk=3, n_heads_v=4)
    with pytest.raises(ValueError, match="kda_backend"):
        kch_b200.HybridConfig(kda_backend="triton")
    with pytest.raises(ValueError, match="win"):
        kch_b200.CSADecodingCache(1, 8, 4, 4, -1, "cuda", torch.float32)
    with pytest.raises(TypeError):
        kch_b200.HCADecodingCache(1, 8, 4, 4, "cuda", torch.int32)


def test_module_tree_uses_reference_state_dict_names():
    import kch_b200
    from kch_b200 import synthetic as syn
    cfg = kch_b200.HybridConfig(d_model=32, n_heads_qk=2, n_heads_v=2, head_dim_k=8, head_dim_v=8, csa_c=8, csa_dc=8,
                                csa_cI=4, csa_nh=2, hca_c=8, hca_dc=8, hca_nh=2, csa_m=4, hca_m2=8)
    model = kch_b200.HybridKCHAttention(cfg, total_layers=5)
    assert model.layout == ["kda", "kda", "kda", "csa", "hca"]
    params = syn.hybrid_params(1, cfg, 5, dtype=torch.float32)
    assert set(params) == set(model.state_dict())
    model.load_state_dict(params, strict=True)


def test_install_is_reversible_when_reference_is_importable():
    import sys
    # a checkout named by the environment, else the offline install of the reference under baseline/_ref
    ref = os.environ.get("KCH_REFERENCE_DIR") or os.path.join(ROOT, "baseline", "_ref")
    if not os.path.isfile(os.path.join(ref, "ops_fused.py")):
        pytest.skip("the reference is not installed (baseline/_ref) and KCH_REFERENCE_DIR is not set")
    sys.path.insert(0, ref)
    try:
        import kch_b200
        import ops_fused
        import ops_kda_backend
        before = (ops_kda_backend.kda_forward, ops_fused.naive_csa, ops_fused.naive_hca)
        done = kch_b200.install()
        assert "ops_kda_backend.kda_forward" in done and "ops_fused.naive_csa" in done
        assert "ops_csa.naive_csa" in done and "ops_hca.naive_hca" in done and "ops_fused.kda_forward" in done
        assert ops_kda_backend.validate_kda_backend("b200") == "b200"
        cfg = ops_fused.HybridConfig(kda_backend="b200")
        assert cfg.kda_backend == "b200"
        # CPU tensors still reach the reference implementation through the rebound globals
        q = torch.nn.functional.normalize(torch.randn(1, 4, 2, 8), dim=-1)
        o, _ = ops_kda_backend.kda_forward(q, q, q, -torch.rand(1, 4, 2, 8), torch.rand(1, 4, 2), backend="reference")
        assert o.shape == (1, 4, 2, 8)
        with pytest.raises(RuntimeError, match="CUDA"):
            ops_kda_backend.kda_forward(q, q, q, -torch.rand(1, 4, 2, 8), torch.rand(1, 4, 2), backend="b200")
        kch_b200.uninstall()
        assert (ops_kda_backend.kda_forward, ops_fused.naive_csa, ops_fused.naive_hca) == before
        with pytest.raises(ValueError):
            ops_kda_backend.validate_kda_backend("b200")
    finally:
        sys.path.remove(ref)


def test_ring_tail_does_not_alias_the_ring_storage():
    """The window keys a chunked prefill takes from the ring before appending its own chunk must survive that
    append: while the ring is not yet full its contents are a view of the storage, and a chunk that wraps around
    overwrites the very slots the view shows."""
    from types import SimpleNamespace
    from kch_b200.decoding_cache import _SlidingWindowRingBuffer
    from kch_b200.fused import HybridDecoding
    for first, second in ((6, 6), (1, 9), (3, 20)):
        ring = _SlidingWindowRingBuffer(1, 8, 2, "cpu", torch.float32)
        rows = torch.arange(1, first + second + 1, dtype=torch.float32).view(1, -1, 1).expand(1, -1, 2)
        ring.append(rows[:, :first])
        tail = HybridDecoding._ring_tail(SimpleNamespace(_sw=ring), 8)
        want = rows[:, max(0, first - 7):first].clone()
        ring.append(rows[:, first:])
        assert torch.equal(tail, want), (first, second, tail[0, :, 0].tolist())
        assert torch.equal(ring.get(), rows[:, -8:])


def test_projection_slices_are_read_in_place():
    """Column slices of a fused projection reach the KDA kernels without a copy, also for a single token per
    sequence (where PyTorch reports an arbitrary stride for the size-1 time axis)."""
    from kch_b200.kda import _token_stride
    for B, T in ((64, 1), (1, 1), (2, 5), (1, 7)):
        proj = torch.zeros(B, T, 6288, dtype=torch.bfloat16)
        q, k, v, gd, beta = proj.split([2048, 2048, 2048, 128, 16], dim=-1)
        for t, inner in ((q.unflatten(-1, (16, 128)), 2048), (v.unflatten(-1, (16, 128)), 2048), (beta, 16)):
            t2, ld = _token_stride(t)
            assert t2.data_ptr() == t.data_ptr()
            assert ld == (6288 if B * T > 1 else inner)
    odd = torch.zeros(2, 3, 100, dtype=torch.bfloat16)[..., 1:65].unflatten(-1, (2, 32))   # misaligned start
    t2, ld = _token_stride(odd)
    assert t2.is_contiguous() and ld == 64


def test_new_entry_points_validate_on_the_host():
    from kch_b200 import _lib
    lib = _lib.load()
    rc = lib.kch_cache_advance(None, 4, None)
    assert rc < 0 and b"counters" in lib.kch_last_error()
    assert lib.kch_attend_decode_splits(64) >= 1 and lib.kch_attend_decode_splits(1) <= 32
    assert lib.kch_attend_decode_workspace_bytes(64, 16, 128) == 64 * lib.kch_attend_decode_splits(64) * 16 * 130 * 4
    assert lib.kch_decode_indexer_workspace_bytes(64, 32770) == 64 * 32772 * 4
    a = _lib.AttendDecodeArgs()
    a.B, a.nh, a.c = 4, 16, 64
    rc = lib.kch_attend_decode(a, None)
    assert rc < 0 and b"c == 128" in lib.kch_last_error()
    rc = lib.kch_decode_indexer_topk(None, 0, 0, None, 1, None, None, 0, 0, None, 2, 16, 4, 64, 0, 1, 1.0, 4, None, None, 0, None)
    assert rc < 0 and b"topk" in lib.kch_last_error()
    rc = lib.kch_layernorm_short_conv(None, None, None, 1e-5, None, None, None, None, None, 1, 8, 100, 1, 1, None)
    assert rc < 0 and b"d=100" in lib.kch_last_error()
    rc = lib.kch_indexer_topk_ex(None, 2, 64, 0, None, None, None, 1, 4, 4, 1, 64, 4, 1.0, 4, 0, -1, 0, 0, None, 0, None)
    assert rc < 0 and b"q_dtype" in lib.kch_last_error()
    assert lib.kch_kda_chunk_gate_supported(128, 128, 64, -10.0, _lib.KCH_BF16) == 1
    assert lib.kch_kda_chunk_gate_supported(64, 128, 64, -10.0, _lib.KCH_BF16) == 0
    assert lib.kch_kda_chunk_gate_supported(128, 128, 64, -10.0, _lib.KCH_F32) == 0


def test_bench_accounting():
    import importlib.util
    spec = importlib.util.spec_from_file_location("kch_bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    fpt = bench.algorithmic_flops_per_token(bench.C4, 32768)
    assert abs(fpt - 145.86e6) / 145.86e6 < 1e-3
    nbytes = bench.decode_state_bytes(bench.C4, 64, 131072, 2)
    assert 0.80e9 < nbytes < 0.90e9          # indexer keys counted at their stored width (bf16 + fp32 norm per row)
    assert bench.decode_state_bytes(bench.C4, 64, 131072, 1.0625) < nbytes


def _cpu_cache(cls, **fields):
    """A cache object without its CUDA requirement: enough for what append_step decides on the host."""
    cache = object.__new__(cls)
    cache.__dict__.update(B=2, c=8, win=4, device=torch.device("cpu"), dtype=torch.float32, kv_quant=None, _kind=None,
                          _normalize_qk=True, **fields)
    cache.reset()
    return cache


@pytest.mark.parametrize("T", [1, 5])
@pytest.mark.parametrize("cut", ["narrow", "wide", "batch of one", "larger batch", "flat"])
def test_append_refuses_a_stream_of_another_shape(T, cut):
    """The append kernels read every stream with the width and batch of the cache: a stream of another shape is refused before
    anything is grown or stored, and so is a bias with fewer rows than a block."""
    import kch_b200
    x = lambda w: torch.zeros(2, T, w)  # noqa: E731

    def bad(t):
        return {"narrow": t[..., :-1], "wide": torch.cat([t, t], -1), "batch of one": t[:1], "larger batch": torch.cat([t, t]),
                "flat": t.flatten(1)[:, None].expand(-1, T, -1)[..., :1]}[cut]
    csa = _cpu_cache(kch_b200.CSADecodingCache, c_I=4, m=4)
    biases = [torch.zeros(4, 8), torch.zeros(4, 8), torch.zeros(4, 4)]
    for i in range(1, 6):
        streams = [x(8)] * 4 + [x(4)] * 2
        streams[i] = bad(streams[i])
        with pytest.raises(ValueError):
            csa.append_step(*streams, *biases)
    for i in range(3):
        with pytest.raises(ValueError, match="must hold"):
            csa.append_step(*[x(8)] * 4, *[x(4)] * 2, *(b[:-1] if i == j else b for j, b in enumerate(biases)))
    hca = _cpu_cache(kch_b200.HCADecodingCache, m2=4)
    with pytest.raises(ValueError):
        hca.append_step(x(8), bad(x(8)), torch.zeros(4, 8))
    with pytest.raises(ValueError, match="must hold"):
        hca.append_step(x(8), x(8), torch.zeros(3, 8))
    for cache in (csa, hca):
        assert (cache._n_tokens_seen, cache._n_blocks, cache._acc_len, cache._comp) == (0, 0, 0, None)


def test_compression_refuses_streams_of_different_shapes():
    import kch_b200
    C, b = torch.zeros(2, 8, 6), torch.zeros(4, 6)
    for other in (C[:1], C[..., :5], C[:, :4]):
        with pytest.raises(ValueError, match="shape"):
            kch_b200.csa_compress_kv(C, other, b, 4)
        for i in range(3):
            streams = [C, C, C]
            streams[i] = other
            with pytest.raises(ValueError, match="shape"):
                kch_b200.csa_compress_kv_overlapped(C, *streams, b, b, 4)
    with pytest.raises(ValueError, match="must hold"):
        kch_b200.csa_compress_kv(C, C, b[:3], 4)
    with pytest.raises(ValueError, match="must hold"):
        kch_b200.csa_compress_kv_overlapped(C, C, C, C, b, b[:3], 4)
    with pytest.raises(ValueError, match="prev_Cb"):
        kch_b200.csa_compress_kv_overlapped(C, C, C, C, b, b, 4, prev_Cb=C[:, :3], prev_Zb=C[:, :4])


def test_bulk_append_refuses_incomplete_arguments():
    """kch_cache_append_rows: what one stream needs is there, or the call is refused on the host (the pointers below are never
    followed: every call is wrong in one respect)."""
    from kch_b200 import _lib
    lib = _lib.load()

    def call(T=4, ring_n=0, seen=0, bs_c=32, **change):
        a = _lib.CacheAppendArgs()
        a.B, a.c, a.c_I, a.m, a.win, a.dtype, a.ld_c, a.ld_i = 1, 8, 4, 4, 4, _lib.KCH_F32, 8, 4
        for name in ("Ca Cb Za Zb K_idx Z_idx acc_Ca acc_Cb acc_Za acc_Zb acc_K_idx acc_Z_idx prev_Cb prev_Zb ring counters").split():
            setattr(a, name, 4096)
        for name, value in change.items():
            setattr(a, name, value)
        rc = lib.kch_cache_append_rows(a, T, bs_c, 16, ring_n, seen, None)
        return rc, lib.kch_last_error().decode()
    for name in "Zb acc_Cb acc_Zb prev_Cb prev_Zb Cb".split():
        rc, why = call(**{name: None})
        assert rc < 0 and "Cb goes with" in why, (name, why)
    for name in "Z_idx acc_K_idx acc_Z_idx K_idx".split():
        rc, why = call(**{name: None})
        assert rc < 0 and "K_idx goes with" in why, (name, why)
    rc, why = call(c_I=0)
    assert rc < 0 and "c_I" in why
    rc, why = call(ring=None)
    assert rc < 0 and "ring" in why
    for kw in (dict(ld_c=-8), dict(ld_i=-1), dict(bs_c=-1)):
        rc, why = call(**kw)
        assert rc < 0 and "stride" in why, why
    for kw in (dict(seen=2 ** 31 - 4), dict(ring_n=2 ** 31 - 4), dict(n_blocks=2 ** 31 - 2), dict(T=2 ** 31), dict(seen=-1)):
        rc, why = call(**kw)
        assert rc < 0 and "out of range" in why, (kw, why)


def test_attend_refuses_queries_of_another_width():
    """The kernels read nh * c query channels per token (naive_hca with a W_UQ of fewer rows arrives here)."""
    from kch_b200.csa import attend
    comp = torch.zeros(1, 2, 8)
    for q in (torch.zeros(1, 3, 24), torch.zeros(1, 3, 40), torch.zeros(1, 3, 3, 8)):
        with pytest.raises(RuntimeError, match="shape"):
            attend(q, comp, nh=4, c=8, m=1, q_normalize=True)


def test_chained_kernels_take_tensor_memory_before_they_trigger():
    """A kernel started early may allocate tensor memory before its wait, so the kernel before it has to hold its own by then:
    in every kernel with both, no trigger stands before the allocation."""
    csrc = os.path.join(ROOT, "kda-csa-hca-fusion_b200", "csrc")
    both = []
    for name in sorted(os.listdir(csrc)):
        for body in open(os.path.join(csrc, name)).read().split("__global__")[1:]:
            if "chain_trigger()" in body and "tcgen05.alloc" in body:
                both.append(name)
                assert body.index("chain_trigger()") > body.index("tcgen05.alloc"), name
    assert both == ["gemm_decode.cu", "indexer_decode_tc5.cu"]


def test_fused_weights_say_whether_this_call_launched_the_copy():
    """The early weight fetch of a one-token step rests on it: False on the call that concatenates (first, or after a change in
    place), True on the next, and the answer is the caller's own, whatever another thread asks in between."""
    from torch import nn
    from kch_b200.fused import _at_rest, _FusedWeights
    a, b = nn.Linear(4, 3, bias=False), nn.Linear(4, 5, bias=False)
    f = _FusedWeights()
    W, settled = f.get_settled(a.weight, b.weight)
    again = f.get_settled(a.weight, b.weight)          # another caller, between the first one's get and its launch
    assert not settled and again[1] and again[0] is W and f.get(a.weight, b.weight) is W
    with torch.no_grad():
        b.weight.mul_(2)
    W2, settled = f.get_settled(a.weight, b.weight)
    assert not settled and torch.equal(W2[3:], b.weight.detach()) and f.get_settled(a.weight, b.weight)[1]
    assert not hasattr(f, "settled")
    # a parametrised weight is computed when it is read: the launch before the product writes it

    class Twice(nn.Module):
        def forward(self, w):
            return w * 2
    assert _at_rest(a.weight)
    nn.utils.parametrize.register_parametrization(a, "weight", Twice())
    assert not _at_rest(a.weight)


def test_epilogue_segments_are_taken_by_value(monkeypatch):
    """A parameter given as a tensor and changed in place between two products is read anew."""
    from kch_b200 import _lib, csa
    seen = []

    class Lib:
        def kch_linear_ex(self, *a):
            seen.append([a[12].seg_param[i] for i in range(a[12].n_segments)])
            return 0
    monkeypatch.setattr(_lib, "load", lambda: Lib())
    monkeypatch.setattr(_lib, "require_cuda", lambda *t, fn="": None)
    monkeypatch.setattr(_lib, "device", lambda dev: _lib._SAME_DEVICE)
    monkeypatch.setattr(_lib, "stream", lambda: 0)
    scale, x, W = torch.tensor(0.5), torch.zeros(2, 8), torch.zeros(4, 8)
    for value in (0.5, 2.0):
        scale.fill_(value)
        csa.linear(x, W, epilogue=[(4, _lib.ACT_NEG_SOFTPLUS, scale)])
    assert seen == [[0.5], [2.0]]


def test_layer_calls_refuse_on_the_host():
    """The structures of the one-call layers reach the library field by field (sizes and messages depend on the last ones), and
    calls that are wrong in one respect are refused before anything is launched (the pointers are never followed)."""
    from kch_b200 import _lib
    lib = _lib.load()

    def csa(**kw):
        a = _lib.CsaLayerArgs()
        a.l.B, a.l.T, a.l.d, a.l.dtype, a.l.x, a.l.ld_x, a.l.out = 2, 100, 64, _lib.KCH_BF16, 4096, 64, 4096
        a.c, a.c_I, a.dc, a.nh, a.nIh, a.m, a.topk, a.sliding_window, a.T_blocks, a.scale = 32, 16, 24, 4, 2, 16, 3, 5, 6, 1.0
        a.W = a.Wq = a.Ba = a.Bb = a.B_idx = 4096
        a.n_w, a.n_q, a.ld_w, a.ld_wq = 192, 160, 64, 24
        for k, v in kw.items():
            setattr(a.l if k in ("B", "norm_w", "W_o", "out") else a, k, v)
        return a
    full = lib.kch_csa_layer_workspace_bytes(csa())
    assert full - lib.kch_csa_layer_workspace_bytes(csa(proj=4096)) == 2 * 100 * 192 * 2
    assert full - lib.kch_csa_layer_workspace_bytes(csa(comp=4096)) == 2 * 6 * 32 * 4
    assert full - lib.kch_csa_layer_workspace_bytes(csa(kcomp=4096)) == 2 * 6 * 16 * 4
    assert lib.kch_csa_layer_workspace_bytes(csa(W=None)) - full == 192 * 64 * 2
    for kw, why in ((dict(), "workspace"), (dict(B=0), "B=0"), (dict(T_blocks=5), "T_blocks=5"), (dict(n_w=180), "fused widths"),
                    (dict(norm_w=4096), "come together"), (dict(m=0), "m=0"), (dict(B_idx=None), "biases"), (dict(W_o=4096, out=None), "`out`")):
        assert lib.kch_csa_layer(csa(**kw), None) < 0 and why in lib.kch_last_error().decode(), (kw, lib.kch_last_error())

    def hca(**kw):
        a = _lib.HcaLayerArgs()
        a.l.B, a.l.T, a.l.d, a.l.dtype, a.l.x, a.l.ld_x, a.l.out = 1, 70, 64, _lib.KCH_F32, 4096, 64, 4096
        a.c, a.dc, a.nh, a.m2, a.sliding_window, a.T_blocks, a.scale, a.n_w, a.W, a.Wq, a.B_pos = 32, 16, 2, 32, 0, 2, 1.0, 80, 4096, 4096, 4096
        for k, v in kw.items():
            setattr(a, k, v)
        return a
    full = lib.kch_hca_layer_workspace_bytes(hca())
    assert full - lib.kch_hca_layer_workspace_bytes(hca(comp=4096)) == 256 and full - lib.kch_hca_layer_workspace_bytes(hca(proj=4096)) == 22528
    for kw, why in ((dict(), "workspace"), (dict(T_blocks=1), "T_blocks=1"), (dict(n_w=79), "fused width"), (dict(B_pos=None), "fused width")):
        assert lib.kch_hca_layer(hca(**kw), None) < 0 and why in lib.kch_last_error().decode(), (kw, lib.kch_last_error())

    def kda(**kw):
        a = _lib.KdaLayerArgs()
        a.l.B, a.l.T, a.l.d, a.l.dtype, a.l.x, a.l.ld_x, a.l.out, a.l.W_o = 1, 40, 64, _lib.KCH_F32, 4096, 64, 4096, 4096
        a.H, a.HV, a.K, a.V, a.chunk_size, a.n_w, a.scale, a.decay_scale, a.g_clamp_min = 2, 2, 16, 16, 64, 120, 0.25, 0.1, -10.0
        a.W = a.W_gup = a.conv_w = a.conv_b = a.lookback_out = 4096
        for k, v in kw.items():
            setattr(a.l if k in ("T",) else a, k, v)
        return a
    assert lib.kch_kda_layer_workspace_bytes(kda()) == 4 * 40 * (64 + 120 + 32 + 32)       # every piece a multiple of 256 here
    for kw, why in ((dict(), "workspace"), (dict(T=1), "T=1"), (dict(HV=3), "HV=3"), (dict(n_w=113), "fused width"), (dict(lookback_out=None), "fused width")):
        assert lib.kch_kda_layer(kda(**kw), None) < 0 and why in lib.kch_last_error().decode(), (kw, lib.kch_last_error())
    a = _lib.CacheAppendArgs()
    a.B, a.c, a.c_I, a.m, a.dtype, a.comp_kind, a.acc_len = 1, 8, 4, 4, _lib.KCH_F32, _lib.KCH_F32, 1
    assert lib.kch_cache_append_prompt(a, 8, 64, 32, 0, 0, None, None, None, 0, None) < 0 and b"open block" in lib.kch_last_error()
    a.acc_len = 0
    a.comp_kind = _lib.KCH_FP8_E4M3
    assert lib.kch_cache_append_prompt(a, 8, 64, 32, 0, 0, None, None, None, 0, None) < 0 and b"8-bit" in lib.kch_last_error()
    a.comp_kind = _lib.KCH_F32
    assert lib.kch_cache_append_prompt(a, 8, 64, 32, 0, 0, None, None, None, 0, None) < 0 and b"no room" in lib.kch_last_error()
    assert lib.kch_cache_append_prompt_workspace_bytes(a, 8) == 512
