"""Edges of the ranges that the kernels' dispatch rules accept: remainders of tiles, smallest and largest sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from kch_b200 import synthetic as syn  # noqa: E402
from oracle import kch_oracle as orc  # noqa: E402

DEV = "cuda"


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
