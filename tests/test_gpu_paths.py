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
