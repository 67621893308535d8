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


def _counts(spec, st):
    """Per molecule: neighbours within rcut, and those of them that are near pairs
    (their site vectors may cross half a box length)."""
    d = st.r[:, None] - st.r[None]
    d = (d - np.round(d)) * st.L
    within = (d ** 2).sum(-1) <= spec.rcut ** 2
    np.fill_diagonal(within, False)
    reach = np.linalg.norm(spec.moltype.r, axis=1).max()
    near = within & (np.abs(d) >= 0.5 * st.L - 2.0 * reach - 1e-3).any(-1)
    return within.sum(1), near.sum(1)


def _dense(model, nmol, scale, seed, moved=0.15):
    """A bulk box denser than the liquid, the molecules moved a little off their lattice."""
    e = S.make_ensemble("dense", model, 0, nmol, 0.0, 12.0, 10.0, 1, 1, 300, 300, 0.1e6, 0.1e6, seed)
    st = e.states[0]
    st.L = st.L * scale
    rng = np.random.default_rng(seed)
    st.r = (st.r + rng.normal(size=st.r.shape) * (moved / st.L)) % 1.0
    return copy.deepcopy(e.spec), st


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("model", ["tip3p", "tip5p"])
def test_more_pairs_than_one_partial_sum(model, prec):
    """A lane's FP32 sums, and the FP64 form's shared rows, close after 256 pairs of a
    molecule: a box where molecules of one warp lie on both sides of that."""
    spec, st = _dense(model, 1000, 0.968, 310)
    pairs, near = _counts(spec, st)
    warps = pairs.reshape(-1, 4)
    assert ((warps > 256).any(1) & (warps <= 256).any(1)).sum() > 20 and near.max() == 0
    _check(spec, st, prec)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_near_pairs_beside_several_partial_sums(prec):
    """A box little above 2 rcut: some near pairs beside more than 256 far ones."""
    spec, st = _dense("tip3p", 729, 0.935, 312)
    pairs, near = _counts(spec, st)
    assert pairs.min() > 256 and 0 < near.mean() < 64
    _check(spec, st, prec)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_more_near_pairs_than_one_partial_sum(prec):
    """A weak charge far from its molecule's centre makes nearly every pair near.  The
    energy gate needs terms that do not cancel: the FP32 form's Lennard-Jones and
    Coulomb energies are good to some 8e-7 and 4e-7, which is 6e-7 of their sum here."""
    spec, st = _dense("tip4p", 729, 0.935, 312, moved=0.05)
    spec.moltype.r[1] *= 5.0
    spec.moltype.charge[:] = (0.0, 1e-6, 1.04, -1.04)
    pairs, near = _counts(spec, st)
    assert near.min() > 256 and (pairs > near).all()
    _check(spec, st, prec)


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


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("nmol", [511, 512, 1500, 2100])
def test_cell_lists_and_their_smallest_replica(nmol, prec):
    """A tube long enough to be cut into cells, from 512 molecules on; 2100 take two
    windows of the rebuild's bitmap.  Both forms share the rebuild, and the FP64 form
    tests its entries in FP64.  (A cutoff off the lattice: at 9.0 A every molecule has
    a neighbour exactly at it.)"""
    e = S.make_ensemble("cells", "tip4p", 1, nmol, 7.0, 9.1, 8.1, 1, 1, 300, 300, 0.1e6, 0.1e6, 330)
    _check(e.spec, e.states[0], prec, "fp32 small" if prec == "fp32" else None)


@pytest.mark.parametrize("prec,charges", [("fp32", "water"), ("fp64", "water"), ("fp32", "other")])
def test_mixed_models_in_one_handle_equal_each_alone(prec, charges):
    """The first forces of a handle come from one launch over all its models, for which
    the kernels choose per block (alone, the kernel compiled for the model); then the
    chains of the interval graph, one model each: both give the bits of each alone."""
    ens = [S.small_ensemble(m, 1, nmol=n, ntemp=1, npress=1, seed=340, interval=5)
           for m, n in (("tip3p", 70), ("tip4p", 65), ("tip5p", 80))]
    if charges == "other":
        ens = copy.deepcopy(ens)
        for e in ens:
            q = e.spec.moltype.charge
            q[int(np.nonzero(q)[0][0])] *= 0.9
            q[-1] -= q.sum()
    def run(e):
        eng = E.REMDGPU(e, precision=prec)
        first = [eng.ConvertVariablesToHost(k) for k in range(eng.nrep)]
        eng.ExecuteSteps(eng.T, eng.P)
        graph = [eng.ConvertVariablesToHost(k) for k in range(eng.nrep)]
        eng.execute_nsteps(5)
        last = [eng.ConvertVariablesToHost(k) for k in range(eng.nrep)]
        eng.close()
        return first, graph, last
    both = run(ens)
    for k, e in enumerate(ens):
        for a, b in zip(run([e]), both):
            assert all(np.array_equal(a[0][x], b[k][x]) for x in ("r", "v", "q", "p", "f", "n"))
