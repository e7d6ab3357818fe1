"""Where a contraction, the determinant Laplacian or the refinement changes its tile, its instance or its route with the
size, against the oracle or against the same walkers in a batch of another size."""
import ctypes as C

import numpy as np
import pytest
import torch

from sparse_wf_gb300 import params as P, systems

pytestmark = pytest.mark.gpu


def _model(mol, precision):
    from oracle import fire_oracle as O

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    blob, offs = P.pack_params(dims, p, np.float32)
    return FireWaveFunction(mol, precision=precision), P.unpack_params(dims, blob, offs), O.Problem(mol.R, mol.Z, n_up)


def _oracle(prob, p, mol, r):
    """E_loc and the magnitude of the terms it sums"""
    from oracle import fire_oracle as O

    _, g, lap = O.logpsi_fl(prob, p, r)
    v = O.potential_energy(r, mol.R, mol.Z)
    return -0.5 * (lap + g @ g) + v, 0.5 * (abs(lap) + g @ g) + abs(v)


# All electrons see one another, so that a dependency has up to n positions: the instances end at 20, 44 and 64 positions, the
# tile heights change in between; the eliminations' block sizes at 32 and 33 orbitals.
@pytest.mark.parametrize("n,precision", [(n, p) for n in (2, 5, 11, 16, 20, 21, 32, 33, 44, 46, 64) for p in ("fp32", "fp64")] +
                         [(45, "fp64")])
def test_positions_per_dependency(n, precision):
    mol = systems.hydrogen_chain(n, 4.0 / n)
    wf, p, prob = _model(mol, precision)
    r = systems.init_electrons(mol, 2, 11)
    eloc, _ = wf.local_energy_full(p, r, wf.get_static_input(r))
    e = eloc.double().cpu().numpy()
    rng = np.random.default_rng(n)
    for w in range(2):
        rw = r[w].astype(np.float64)
        want, scale = _oracle(prob, p, mol, rw)
        # the conditioning of the walker: what a perturbation of the positions by the precision's rounding makes of E_loc
        eps = 1e-15 if precision == "fp64" else 6e-8
        moved = max(abs(_oracle(prob, p, mol, rw * (1 + eps * rng.choice([-1, 1], rw.shape)))[0] - want) for _ in range(2))
        tol = (1e-9 if precision == "fp64" else 2e-5) * scale + 10 * moved
        assert abs(e[w] - want) <= tol, (w, e[w], want, scale)


def test_tiles_of_batch_sizes():
    """10000 walkers of 4 electrons take the 128 x 128 and the 64 x 64 tiles, 8 the 32 x 32 ones: every output is the same
    sum, so that the energies differ by what the order of the per-center sums leaves (FP32 rounding of the terms)."""
    mol = systems.hydrogen_chain(4, 1.8)
    wf, p, prob = _model(mol, "fp32")
    r = systems.init_electrons(mol, 10000, 3)
    big, _ = wf.local_energy_full(p, r, wf.get_static_input(r))
    few, _ = wf.local_energy_full(p, r[:8], wf.get_static_input(r[:8]))
    for w in range(8):
        want, scale = _oracle(prob, p, mol, r[w].astype(np.float64))
        assert abs(float(big[w]) - float(few[w])) <= 1e-5 * scale
        assert abs(float(big[w]) - want) <= 2e-5 * scale


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_parts_of_column_tiles(precision):
    """log|psi| of 16, 200 and 2000 walkers of 10 electrons: column tiles in parts of one and of two pieces, and whole; the
    sums are exact either way, so that the walkers' values agree to the rounding of their type."""
    mol = systems.hydrogen_chain(10, 1.8)
    wf, p, _ = _model(mol, precision)
    r = systems.init_electrons(mol, 2000, 13)
    a, b, c = (wf.signed(p, r[:w], wf.get_static_input(r[:w]))[1][:16].double().cpu().numpy() for w in (16, 200, 2000))
    tol = (1e-12 if precision == "fp64" else 1e-6) * np.maximum(1.0, np.abs(a))
    assert np.all(np.abs(b - a) <= tol) and np.all(np.abs(c - a) <= tol)


@pytest.mark.parametrize("walkers", [1, 3, 40])
def test_every_walker_refined(walkers):
    """More walkers refined than the first pass's room (a quarter of the batch): the call runs again with room for all."""
    mol = systems.hydrogen_chain(6, 1.8)
    wf, p, prob = _model(mol, "fp32")
    wf.refine_kappa = 1e-3  # no matrix's condition number is below 1
    r = systems.init_electrons(mol, walkers, 21)
    eloc, aux = wf.local_energy_full(p, r, wf.get_static_input(r))
    assert aux["refined"] == walkers
    for w in range(0, walkers, max(1, walkers // 4)):
        want, scale = _oracle(prob, p, mol, r[w].astype(np.float64))
        assert abs(float(eloc[w]) - want) <= 1e-5 * scale


@pytest.mark.parametrize("M,N,K", [(1, 16, 8), (127, 132, 40), (129, 256, 256), (20001, 324, 72), (300, 4, 64)])
def test_mixed_rows_at_16_bytes(cuda_lib, M, N, K):
    """Rows that are 16- but not 32-byte aligned, row and column remainders, more row tiles than SMs."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M * K + 4, device="cuda", generator=g)[4:].view(M, K)
    W = torch.randn(K, N, device="cuda", generator=g) / K**0.5
    out = torch.full((M, N), float("nan"), device="cuda")
    ws = torch.empty(32768 * -(-N // 128) * -(-K // 64) + 4 * N, dtype=torch.uint8, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    ptr = [C.c_void_p(t.data_ptr()) for t in (A, W, out, ws, status)]
    rc = cuda_lib.fire_gemm_mixed(C.c_void_p(torch.cuda.current_stream().cuda_stream), M, N, K, ptr[0], ptr[1], ptr[2], ptr[3],
                                  C.c_size_t(ws.numel()), ptr[4])
    assert rc == 0
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    ref = A.double() @ W.double()
    # a row's and a column's elements err by 2^-20 of their largest: the product by that times K largest by largest
    bound = 2.0**-19 * K * A.abs().amax(1, keepdim=True).double() * W.abs().amax(0, keepdim=True).double()
    assert bool(((out.double() - ref).abs() <= bound).all())


def test_gradients_of_batch_sizes():
    """60 walkers at once put their pair rows through the warp-per-row contraction, two at a time through the tiles."""
    mol = systems.hydrogen_chain(10, 1.8)
    wf, p, _ = _model(mol, "fp32")
    r = systems.init_electrons(mol, 60, 9)
    static = wf.get_static_input(r)
    a, b = (wf.logpsi_grad(p, r, static, chunk=c)[0].double().cpu().numpy() for c in (60, 2))
    # FP32 sums in another order: 10^-5 of the row's norm
    assert np.all(np.linalg.norm(a - b, axis=1) <= 1e-5 * np.linalg.norm(b, axis=1))
