"""TRANSPORT and REINITIALIZATION of a column whose band is more than one interface's: a vapour slab
has 32 cells on the layers the stages work on, which takes them off the registers and through the
window -- against the oracle, bit for bit, and the two-cells-a-layer band beside it in the same batch."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_lvs import Case, coupled_psi, run

pytestmark = pytest.mark.gpu

N = 64


def slab(za, zb):
    """Vapour between za and zb, liquid below and above."""
    a, b = O.lvs_init(N, 1.0, za), O.lvs_init(N, 1.0, zb)
    assert not np.any((a["layer"] > 0) & (b["layer"] > 0))
    st = {"n": N, "length": 1.0, "phi": b["phi"] - a["phi"], "layer": a["layer"] + b["layer"],
          "psif": (1.0 - a["psif"]) + b["psif"], "wo": a["wo"]}
    st["vol_tot_ori"] = float(np.sum((1.0 - st["psif"][1:2 * N + 1]) / (2 * N)))
    return st


@pytest.mark.parametrize("iphs,mf_amp", [(1, 0.02), (2, 0.0)])
def test_transport_of_a_slab(iphs, mf_amp):
    case = Case(N, [0.3, 0.45], seed=5, wscale=0.4, iphs=iphs, mf_amp=mf_amp)
    case.states[0] = slab(0.3, 0.62)
    case.pcs[0], case.pzs[0] = coupled_psi(case.states[0]["psif"])
    run(case, 4)
    assert (case.states[0]["layer"] > 0).sum() > 32 >= (case.states[1]["layer"] > 0).sum()


def test_reinitialization_of_a_slab():
    from lica_boiling1d_b200 import routines
    st = slab(0.25, 0.7)
    k = np.arange(st["phi"].shape[0])
    start = st["phi"] * (1.0 + 0.2 * np.sin(0.7 * k))
    ref = O.reinitialization(N, 1.0, start.copy(), st["layer"].copy(), 8)
    got = start[None].copy()
    assert not np.any(routines.reinitialization(N, 1.0, got, st["layer"][None].copy(), 8))
    assert np.any(ref != start)
    np.testing.assert_array_equal(got[0], ref)
