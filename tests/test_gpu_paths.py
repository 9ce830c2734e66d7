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
