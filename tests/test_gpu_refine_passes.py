"""The refinement of a local energy in several passes: capacity 30 of 40 walkers beside passes of 6 (refined by at most 6 at a
time, as the workspace holds), 15 of them flagged, so that some passes are full, one is partly filled and some are empty.
Every walker is compared with the same walkers refined in one pass, the refined ones with the oracle; eagerly, where the FP64
values run on a stream beside the FP32 planes, and captured, where everything is in one order."""
import ctypes as C

import numpy as np
import pytest
import torch

from sparse_wf_gb300 import _lib, params as P, systems

pytestmark = pytest.mark.gpu

WALKERS, FLAGGED, ROOM, CHUNK = 40, 15, 30, 6


@pytest.fixture(scope="module", params=["fp32", "mixed"])
def case(request, cuda_lib):
    """The wavefunction with the condition number that flags FLAGGED walkers, and the energies in one pass."""
    from oracle import fire_oracle as O

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol = systems.hydrogen_chain(6, 1.8)
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    blob, offs = P.pack_params(dims, p, np.float32)
    p = P.unpack_params(dims, blob, offs)
    wf = FireWaveFunction(mol, precision=request.param)
    wf.refine_ratio = wf.refine_ks = wf.refine_kscond = 1e30
    r = wf._electrons(systems.init_electrons(mol, WALKERS, 21))
    static = wf.get_static_input(r)
    wf.refine_kappa = 1e30
    cond = wf.local_energy_full(p, r, static, debug=True)[1]["debug"]["cond"].cpu().numpy()
    order = np.sort(cond)
    wf.refine_kappa = float(np.sqrt(order[-FLAGGED] * order[-FLAGGED - 1]))
    wf._refine_cap = ROOM
    one, aux = wf.local_energy_full(p, r, static, debug=True)
    assert aux["refined"] == FLAGGED
    prob = O.Problem(mol.R, mol.Z, n_up)
    want, scale = np.zeros(WALKERS), np.zeros(WALKERS)
    for w in range(WALKERS):
        rw = r[w].double().cpu().numpy()
        _, g, lap = O.logpsi_fl(prob, p, rw)
        v = O.potential_energy(rw, mol.R, mol.Z)
        want[w], scale[w] = -0.5 * (lap + g @ g) + v, 0.5 * (abs(lap) + g @ g) + abs(v)  # the terms' magnitude
    return dict(wf=wf, p=p, r=r, static=static, one=one.double().cpu().numpy(), want=want, scale=scale,
                refined=aux["debug"]["refined"].cpu().numpy() > 0, mixed=request.param == "mixed")


def _check(c, e, refined, order=slice(None)):
    assert np.array_equal(refined, c["refined"][order])
    # the order of the per-center sums: FP32 rounding of the terms
    assert np.all(np.abs(e - c["one"][order]) <= 1e-5 * c["scale"][order])
    bound = np.where(c["refined"] | (not c["mixed"]), 1e-5, 1e-4)
    assert np.all((np.abs(e - c["want"][order]) <= (bound * c["scale"])[order]))


def test_passes(case):
    c, wf = case, case["wf"]
    try:
        wf.chunk_walkers = CHUNK
        for _ in range(3):
            wf._refine_cap = ROOM
            e, aux = wf.local_energy_full(c["p"], c["r"], c["static"], debug=True)
            _check(c, e.double().cpu().numpy(), aux["debug"]["refined"].cpu().numpy() > 0)
    finally:
        wf.chunk_walkers = 0


def test_passes_captured(case):
    """One graph, replayed on the walkers and on the walkers in reverse order (other walkers in every pass)."""
    c, wf = case, case["wf"]
    dev = wf._params(c["p"])
    prob = wf._problem(WALKERS, c["static"], refine=True)
    prob.chunk_walkers, prob.refine_cap = CHUNK, ROOM
    ws, status = wf._workspace(prob), torch.zeros(_lib.STATUS_WORDS, dtype=torch.int32, device="cuda")
    r, eloc = c["r"].clone(), torch.empty(WALKERS, dtype=wf.dtype, device="cuda")
    refined = torch.zeros(WALKERS, dtype=torch.int32, device="cuda")
    dbg = _lib.ElocDebug()
    dbg.refined = refined.data_ptr()

    def call():
        _lib.check(_lib.load().fire_local_energy(
            wf._stream(), C.byref(prob), C.c_void_p(wf.R_dev.data_ptr()), C.c_void_p(wf.Z_dev.data_ptr()),
            C.c_void_p(dev.prepared.data_ptr()), C.c_void_p(r.data_ptr()), None, None, C.c_void_p(eloc.data_ptr()), None,
            C.byref(dbg), C.c_void_p(ws.data_ptr()), C.c_size_t(ws.numel()), C.c_void_p(status.data_ptr())),
            "fire_local_energy")

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        call()
    for order in (slice(None), slice(None, None, -1)):
        r.copy_(c["r"].flip(0) if order.step else c["r"])
        status.zero_()
        eloc.fill_(float("nan"))
        refined.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert int(status[5]) == FLAGGED and int(status[0]) == 0
        _check(c, eloc.double().cpu().numpy(), refined.cpu().numpy() > 0, order)
