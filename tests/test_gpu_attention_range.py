"""Attention norms far from 1: all electrons within the cutoff of one another and of every nucleus, so that the embeddings are
large and the norms (oracle) reach 10^14 to 10^22, where their cube, for the largest their square, is beyond FP32's range.
Tolerance as for the positions per dependency (test_gpu_tiles.py): 2e-5 of the terms' magnitude and ten times what a rounding
of the positions makes of E_loc."""
import numpy as np
import pytest

from sparse_wf_gb300 import params as P, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("n", [42, 43, 48, 50])
def test_large_attention_norms(n, precision):
    from oracle import fire_oracle as O

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol = systems.hydrogen_chain(n, 4.0 / n)
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    blob, offs = P.pack_params(dims, p, np.float32)
    p = P.unpack_params(dims, blob, offs)
    prob = O.Problem(mol.R, mol.Z, n_up)
    wf = FireWaveFunction(mol, precision=precision)
    r = systems.init_electrons(mol, 2, 11)
    eloc, aux = wf.local_energy_full(p, r, wf.get_static_input(r), debug=True)
    e, grad = eloc.double().cpu().numpy(), aux["debug"]["grad"].double().cpu().numpy()

    def oracle(x):
        _, g, lap = O.logpsi_fl(prob, p, x)
        v = O.potential_energy(x, mol.R, mol.Z)
        return -0.5 * (lap + g @ g) + v, 0.5 * (abs(lap) + g @ g) + abs(v), g

    rng = np.random.default_rng(n)
    for w in range(2):
        x = r[w].astype(np.float64)
        want, scale, g = oracle(x)
        moved = [oracle(x * (1 + 6e-8 * rng.choice([-1, 1], x.shape))) for _ in range(2)]
        tol = 2e-5 * scale + 10 * max(abs(m[0] - want) for m in moved)
        assert abs(e[w] - want) <= tol, (w, e[w], want, scale)
        gtol = 1e-4 * np.abs(g).max() + 10 * max(np.abs(m[2] - g).max() for m in moved)
        assert np.all(np.abs(grad[w].ravel() - g) <= gtol), w


@pytest.mark.parametrize("n", [43, 48, 50])
def test_gradient_at_large_attention_norms(n):
    """Rows of the FP32 gradient against the FP64 build's: 10^-3 of the row's norm (the logits of 50 round to 3 10^-6 of the
    weights; the rows of the other tests agree to 10^-4)."""
    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol = systems.hydrogen_chain(n, 4.0 / n)
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    blob, offs = P.pack_params(dims, p, np.float32)
    p = P.unpack_params(dims, blob, offs)
    r = systems.init_electrons(mol, 2, 11)
    rows = []
    for precision in ("fp32", "fp64"):
        wf = FireWaveFunction(mol, precision=precision)
        rows.append(wf.logpsi_grad(p, r, wf.get_static_input(r))[0].double().cpu().numpy())
    assert np.all(np.linalg.norm(rows[0] - rows[1], axis=1) <= 1e-3 * np.linalg.norm(rows[1], axis=1))
