"""The sliced tensor-core contractions (csrc/fire_sliced.cu) through the entry points, at the edges of their tiles: row
counts around 128, spins of different and of no electrons, envelope lengths K = 8 n_nuc that are no multiple of 16, that
cross the 256-long chunks of the exact sums, column counts around one tile (80 and 64)."""
import numpy as np
import pytest

from sparse_wf_gb300 import params as P, systems

pytestmark = pytest.mark.gpu

# (molecule, walkers): electron rows 2, 126, 128, 130 (one and two row tiles), three electrons (2 up, 1 down), K8 = 40 and
# 24 (K % 16 = 8), 4 n = 40 .. 84 columns, 33 nuclei (K8 = 264: the second chunk holds 8 values)
CASES = [("h2", lambda: systems.hydrogen_chain(2, 1.8), 1), ("h2", lambda: systems.hydrogen_chain(2, 1.8), 63),
         ("h2", lambda: systems.hydrogen_chain(2, 1.8), 64), ("h2", lambda: systems.hydrogen_chain(2, 1.8), 65),
         ("h3", lambda: systems.hydrogen_chain(3, 1.8), 43), ("h5", lambda: systems.hydrogen_chain(5, 1.8), 26),
         ("h21", lambda: systems.hydrogen_chain(21, 1.8), 7), ("ch4", lambda: systems.alkane(1), 13),
         ("h33", lambda: systems.hydrogen_chain(33, 1.8), 2)]


def _inputs(make, walkers):
    from oracle import fire_oracle as O

    mol = make()
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    blob, offs = P.pack_params(dims, p, np.float32)
    return mol, P.unpack_params(dims, blob, offs), systems.init_electrons(mol, walkers, 77), O.Problem(mol.R, mol.Z, n_up)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("name,make,walkers", CASES)
def test_sliced_edges(name, make, walkers, precision):
    from oracle import fire_oracle as O

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol, p, r, prob = _inputs(make, walkers)
    wf = FireWaveFunction(mol, precision=precision)
    static = wf.get_static_input(r)
    sign, logpsi = wf.signed(p, r, static)
    eloc, aux = wf.local_energy_full(p, r, static, debug=True)
    pick = range(0, walkers, max(1, walkers // 6))
    ref = [O.logpsi(prob, p, r[w].astype(np.float64)) for w in pick]
    got = logpsi.double().cpu().numpy()[list(pick)]
    # FP64: the rounding of the determinants; FP32 and mixed: the parity bound of log|psi|
    tol = 1e-10 if precision == "fp64" else 3e-5
    want = np.array([x[1] for x in ref])
    assert np.all(np.abs(got - want) <= tol * np.maximum(1.0, np.abs(want))), np.max(np.abs(got - want))
    assert np.array_equal(sign.cpu().numpy()[list(pick)], np.array([x[0] for x in ref]))
    e = eloc.double().cpu().numpy()
    for w in pick:
        rw = r[w].astype(np.float64)
        _, g, lap = O.logpsi_fl(prob, p, rw)
        v = O.potential_energy(rw, mol.R, mol.Z)
        scale = 0.5 * (abs(lap) + g @ g) + abs(v)  # the magnitude of the terms E_loc sums
        bound = {"fp64": 1e-9, "fp32": 1e-5, "mixed": 1e-4}[precision]
        assert abs(e[w] - (-0.5 * (lap + g @ g) + v)) <= bound * scale, (w, e[w])
