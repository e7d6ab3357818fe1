"""Envelope value rows whose sum is carried by small terms beside large ones: every orbital has weight on its own nucleus
alone, so that an electron's largest coefficients (its nearest nucleus') meet zero weights in all other orbitals.  Half of
the walkers crowd their electrons around the first two nuclei: the determinants are then products of the small values.
Bounds as in the parity tests: the rounding of the determinants in FP64, 3e-5 of log|psi| in FP32 and mixed."""
import numpy as np
import pytest

from sparse_wf_gb300 import params as P, systems

pytestmark = pytest.mark.gpu


def _localized(mol):
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    for spin in ("up", "dn"):
        pi = np.zeros_like(p[f"env_{spin}_pi"])
        rng = np.random.default_rng(1)
        for o in range(mol.n_el):
            pi[o, :, :, o] = rng.normal(1, 0.2, pi[o, :, :, o].shape)
        p[f"env_{spin}_pi"] = pi
    blob, offs = P.pack_params(dims, p, np.float32)
    return P.unpack_params(dims, blob, offs)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n,spacing", [(6, 6.0), (12, 4.0)])
def test_localized_envelopes(n, spacing, precision):
    from oracle import fire_oracle as O

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol = systems.hydrogen_chain(n, spacing)
    p = _localized(mol)
    rng = np.random.default_rng(2)
    r = np.zeros((8, n, 3), np.float32)
    for w in range(8):
        centers = mol.R[[0, 1] + list(rng.integers(0, n, n - 2))] if w % 2 else mol.R[rng.integers(0, 2, n)]
        r[w] = centers + rng.normal(0, 0.7, (n, 3))
    prob = O.Problem(mol.R, mol.Z, systems.spin_counts(mol)[0])
    want = np.array([O.logpsi(prob, p, x.astype(np.float64))[1] for x in r])
    wf = FireWaveFunction(mol, precision=precision)
    static = wf.get_static_input(r)
    tol = (1e-10 if precision == "fp64" else 3e-5) * np.maximum(1.0, np.abs(want))
    value = wf.signed(p, r, static)[1].double().cpu().numpy()
    assert np.all(np.abs(value - want) <= tol), np.abs(value - want).max()
    energy = wf.local_energy_full(p, r, static)[1]["logpsi"].double().cpu().numpy()
    assert np.all(np.abs(energy - want) <= tol), np.abs(energy - want).max()
