"""The force kernels that give eight lanes to a molecule, at the sizes where such a
kernel can go wrong, against the FP64 oracle at the parity gates (FP64 form: forces
1e-10, energy 1e-11; FP32 form: forces and torques 1e-5 on liquid-density systems,
3e-5 on the small confined ones, energy 1e-6 / 3e-6)."""
import copy

import numpy as np
import pytest

from oracle import oracle as O
from remd_b200 import engine as E
from remd_b200 import systems as S
from tests.common import rel

pytestmark = pytest.mark.gpu
GATES = {"fp64": (1e-10, 1e-11), "fp32": (1e-5, 1e-6), "fp32 small": (3e-5, 3e-6)}


def _check(spec, st, prec, gate=None):
    eng = E.REMDGPU([S.Ensemble("g", spec, 1, 1, np.array([st.T]), np.array([st.P]), [st])], precision=prec)
    g = eng.ConvertVariablesToHost(0)
    orc = O.Oracle(spec, st)
    orc.initialize_property()
    tf, te = GATES[gate or prec]
    assert rel(g["f"], orc.f) < tf and rel(g["n"], orc.n) < tf
    assert g["pot"] == pytest.approx(orc.prop()["pot"], rel=te)
    assert rel(g["vir"], orc.prop()["vir"]) < tf
    assert abs(eng.pair_count() - orc.prop()["npairs"]) <= (0 if prec == "fp64" else 1)
    eng.close()


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("nmol", [2, 3, 5, 15, 16, 17, 33])
def test_edges_of_groups_warps_and_blocks(nmol, prec):
    """Molecule counts around a warp (4 molecules), a block (16) and a tile (32)."""
    e = S.small_ensemble("tip4p", 1, nmol=nmol, ntemp=1, npress=1, seed=300 + nmol, wall=7.0)
    _check(e.spec, e.states[0], prec, "fp32 small" if prec == "fp32" else None)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("model", ["tip3p", "tip5p"])
def test_more_pairs_than_one_partial_sum(model, prec):
    """A lane's FP32 sums, and the FP64 form's shared rows, close after 256 pairs of a
    molecule: a bulk box at 1.2 times liquid density has about 290 within 12 A."""
    e = S.make_ensemble("dense", model, 0, 1000, 0.0, 12.0, 10.0, 1, 1, 300, 300, 0.1e6, 0.1e6, 310)
    st = e.states[0]
    st.L = st.L * 0.94
    _check(e.spec, st, prec)


@pytest.mark.parametrize("model", ["tip3p", "tip4p", "tip5p"])
def test_charges_other_than_the_water_models_ratios(model):
    """Any charged sites are accepted: without the ratios that the pair kernel has as
    constants it reads them."""
    e = S.make_ensemble("q", model, 0, 512, 0.0, 10.0, 9.0, 1, 1, 300, 300, 0.1e6, 0.1e6, 320)
    spec = copy.deepcopy(e.spec)
    q = spec.moltype.charge
    first = int(np.nonzero(q)[0][0])
    q[first] *= 0.9
    q[-1] -= q.sum()
    _check(spec, e.states[0], "fp32")


@pytest.mark.parametrize("model,charges", [("tip3p", (-0.834, 1e-24, 0.834)), ("tip4p", (0.0, 0.52, 1e-24, -0.52)),
                                           ("tip5p", (0.0, 0.241, 1e-24, -0.12, -0.121))])
def test_charges_far_apart(model, charges):
    """A charged site that is switched off by a tiny charge (a zero is refused): no
    charge may be taken in units of another, their ratio's square overflows."""
    e = S.make_ensemble("far", model, 0, 512, 0.0, 10.0, 9.0, 1, 1, 300, 300, 0.1e6, 0.1e6, 321)
    spec = copy.deepcopy(e.spec)
    spec.moltype.charge[:] = charges
    _check(spec, e.states[0], "fp32")


def test_fp64_form_with_cell_lists():
    """A tube long enough to be cut into cells: the FP64 form takes the list rebuild
    of the FP32 form and tests its entries in FP64."""
    e = S.make_ensemble("cells", "tip4p", 1, 1500, 7.0, 9.0, 8.0, 1, 1, 300, 300, 0.1e6, 0.1e6, 330)
    _check(e.spec, e.states[0], "fp64")


def test_mixed_models_in_one_handle_equal_each_alone():
    """More models than one kernel is compiled for share a launch (one chain): the
    forces are those of the per-model kernels, bit for bit."""
    ens = [S.small_ensemble(m, 1, nmol=n, ntemp=1, npress=1, seed=340, interval=5)
           for m, n in (("tip3p", 70), ("tip4p", 65), ("tip5p", 80))]
    both = E.REMDGPU(ens, precision="fp32")
    both.execute_nsteps(5)
    for k, e in enumerate(ens):
        alone = E.REMDGPU([e], precision="fp32")
        alone.execute_nsteps(5)
        a, b = alone.ConvertVariablesToHost(0), both.ConvertVariablesToHost(k)
        assert all(np.array_equal(a[x], b[x]) for x in ("r", "v", "q", "p", "f", "n"))
        alone.close()
    both.close()
