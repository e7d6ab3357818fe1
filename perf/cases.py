"""The work that users of this framework have it do, as measurable cases.

Every case is one pass through the public entry points on synthetic molecules: the hydrogen chains and all-trans
alkanes of the configurations, tests and benchmark of this repository.  ``kind`` selects the entry point:

* ``eloc``     local energy by the sparse forward Laplacian (``FireWaveFunction.local_energy_full``): E_loc,
               log|psi| and the sign of every walker;
* ``logpsi``   the value path alone (``FireWaveFunction.signed``);
* ``grad``     the per-walker parameter gradient (``FireWaveFunction.logpsi_grad``);
* ``mcmc``     one Metropolis block of a sampling loop (``make_mcmc``): all-electron moves evaluated in full, or
               single-electron sweeps from a state per walker (the default);
* ``ragged``   local energies of molecules of different sizes in one CUDA-graph launch (``RaggedBatch``).

Parameters are the random initialisation with an active Jastrow (a trained network's is not constant); the two
normalisation scales are the typical 1/std of the embedding, fixed here, so that the inputs follow from the seed
alone.  Walkers are drawn around the nuclei (sigma 1 bohr).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sparse_wf_gb300 import systems
from sparse_wf_gb300.params import PARAM_SLOT_NAMES, ModelDims, activate_jastrow, init_params, pack_params, unpack_params
from sparse_wf_gb300.ragged import RaggedBatch, ragged_alkanes
from sparse_wf_gb300.wavefunction import FireWaveFunction, make_mcmc

CUTOFF, CUTOFF_1EL = 5.0, 20.0
F, DETS, HEADS, HDIM = 256, 4, 16, 16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: log|psi| of a few walkers of a small molecule, where latency and launches count
        dict(name="logpsi_h10_fp32_w16", kind="logpsi", precision="fp32", mol="h", size=10, walkers=16),
        # the small configuration: H10, 512 walkers, in single precision ...
        dict(name="eloc_h10_fp32_w512", kind="eloc", precision="fp32", mol="h", size=10, walkers=512),
        # ... and in double precision (the validation build)
        dict(name="eloc_h10_fp64_w512", kind="eloc", precision="fp64", mol="h", size=10, walkers=512),
        # a small molecule with an odd number of walkers on the mixed path, as a request of a mixed load
        dict(name="eloc_c2h6_mixed_w77", kind="eloc", precision="mixed", mol="c", size=2, walkers=77),
        # the medium configuration, C10H22, on the mixed path (two passes, the second one ragged) ...
        dict(name="eloc_c10h22_mixed_w1021", kind="eloc", precision="mixed", mol="c", size=10, walkers=1021),
        # ... and in plain single precision
        dict(name="eloc_c10h22_fp32_w509", kind="eloc", precision="fp32", mol="c", size=10, walkers=509),
        # the large configuration, C40H82 (322 electrons), on the mixed path: the largest case
        dict(name="eloc_c40h82_mixed_w512", kind="eloc", precision="mixed", mol="c", size=40, walkers=512),
        # a Metropolis block of all-electron moves between two energy evaluations
        dict(name="mcmc_all_c10h22_mixed_w256", kind="mcmc", precision="mixed", mol="c", size=10, walkers=256,
             proposal="all-electron", steps=10),
        # the default sampler: one sweep of single-electron moves from a state per walker, small molecule
        dict(name="mcmc_single_h10_fp32_w256", kind="mcmc", precision="fp32", mol="h", size=10, walkers=256,
             proposal="single-electron", steps=10),
        # the same sampler on the large molecule (a part of a sweep)
        dict(name="mcmc_single_c40h82_mixed_w128", kind="mcmc", precision="mixed", mol="c", size=40, walkers=128,
             proposal="single-electron", steps=16),
        # rows of the optimizer's Jacobian: per-walker gradients with respect to every parameter
        dict(name="grad_c10h22_fp32_w64", kind="grad", precision="fp32", mol="c", size=10, walkers=64),
        # a ragged batch: molecules of different sizes and walker counts, one graph launch
        dict(name="ragged_c2_c12_mixed_m8", kind="ragged", precision="mixed", mol="c", size=12, walkers=128,
             molecules=8, smallest=2, fewest=32, draw_seed=4),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    limit = _cost(listed()[6])
    while True:
        kind = rng.choice(["eloc", "eloc", "eloc", "logpsi", "mcmc", "mcmc", "grad", "ragged"])
        mol = rng.choice(["h", "c", "c"])
        size = log_int(2, 30) if mol == "h" else log_int(1, 40)
        prec = rng.choice(["mixed", "mixed", "fp32", "fp32", "fp64"])
        c = dict(kind=kind, precision=prec, mol=mol, size=size, walkers=log_int(1, 1500))
        if kind == "mcmc":
            c["proposal"] = rng.choice(["all-electron", "single-electron"])
            c["steps"] = rng.randint(2, 12)
            c["walkers"] = log_int(1, 300)
        elif kind == "grad":
            c["precision"] = "fp32"
            c["walkers"] = log_int(1, 100)
        elif kind == "ragged":
            c.update(mol="c", size=rng.randint(4, 12), walkers=log_int(40, 200), precision=rng.choice(["mixed", "fp32"]),
                     molecules=rng.randint(2, 10), smallest=rng.randint(1, 3), fewest=rng.randint(8, 32),
                     draw_seed=rng.randint(0, 1000))
        if _cost(c) <= limit and (c["precision"] != "fp64" or c["size"] * (8 if mol == "c" else 1) <= 20):
            return c


def _cost(c):
    """Rough cost of a pass in the mixed path's floating-point operations (double precision runs at a small part of
    the rate, single precision at half)."""
    return work(c)["flops"] * {"mixed": 1.0, "fp32": 3.0, "fp64": 40.0}[c["precision"]]


# ------------------------------------------------------------------------------------------------ inputs
def _molecule(mol, size):
    return systems.hydrogen_chain(size, 1.8) if mol == "h" else systems.alkane(size)


def _params(mol, seed):
    n_up, _ = systems.spin_counts(mol)
    dims = ModelDims(mol.n_el, n_up, mol.n_nuc, CUTOFF, CUTOFF_1EL)
    p = activate_jastrow(init_params(dims, seed))
    p["scales"] = np.array([1.0 if np.any(mol.Z > 1) else 2.75, 3.0])
    blob, offs = pack_params(dims, p, np.float32)
    return unpack_params(dims, blob, offs)  # the values the device holds (float32)


def _walkers(mol, n, seed):
    return systems.init_electrons(mol, n, 1000 + seed)


def _ragged_sizes(case):
    return ragged_alkanes(case["molecules"], (case["smallest"], case["size"]), (case["fewest"], case["walkers"]),
                          case["draw_seed"])


def prepare(case, seed):
    if case["kind"] == "ragged":
        sizes, counts = _ragged_sizes(case)
        mols = [systems.alkane(n) for n in sizes]
        batch = RaggedBatch(mols, counts, precision=case["precision"], lanes=4, chunk=64)
        for i, (job, mol, b) in enumerate(zip(batch.jobs, mols, counts)):
            job.params = job.wf._params(_params(mol, seed + 17 * i))
            job.r.copy_(torch.from_numpy(_walkers(mol, b, seed + 17 * i)))
            job.static = job.wf.get_static_input(job.r).round_with_padding(1.1, mol.n_el, job.wf.n_up, mol.n_nuc)
        batch._alloc_workspaces()
        batch.run()  # captures the batch graph
        return dict(case=case, batch=batch)
    mol = _molecule(case["mol"], case["size"])
    wf = FireWaveFunction(mol, cutoff=CUTOFF, cutoff_1el=CUTOFF_1EL, precision=case["precision"])
    r = wf._electrons(_walkers(mol, case["walkers"], seed))
    static = wf.get_static_input(r).round_with_padding(1.1, mol.n_el, wf.n_up, mol.n_nuc)
    # walkers per pass: as the benchmark picks them, the Jacobian planes of a pass in at most 65535 row tiles of 64
    wf.chunk_walkers = max(1, min(case["walkers"], 65535 * 64 // (3 * (mol.n_el + static.n_pairs))))
    st = dict(case=case, wf=wf, p=wf._params(_params(mol, seed)), r=r, static=static)
    if case["kind"] == "mcmc":
        one = case["proposal"] == "single-electron"
        st["step"], st["width"] = make_mcmc(wf, steps=case["steps"], init_width=0.5 if one else 0.1,
                                            proposal=case["proposal"], sweeps=(case["steps"] + 0.5) / mol.n_el)
        st["key"] = seed
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "ragged":
        state["batch"].run()
        return [job.eloc for job in state["batch"].jobs]
    wf, p, r, static = state["wf"], state["p"], state["r"], state["static"]
    if case["kind"] == "eloc":
        eloc, aux = wf.local_energy_full(p, r, static)
        return dict(eloc=eloc, logpsi=aux["logpsi"], sign=aux["sign"])
    if case["kind"] == "logpsi":
        sign, logpsi = wf.signed(p, r, static)
        return dict(logpsi=logpsi, sign=sign)
    if case["kind"] == "grad":
        grad, sign, logpsi = wf.logpsi_grad(p, r, static)
        return dict(grad=grad, logpsi=logpsi, sign=sign)
    electrons, stats = state["step"](state["key"], p, r, static, state["width"])
    return dict(electrons=electrons, pmove=stats["pmove"])


# ------------------------------------------------------------------------------------------------ work
def _mean_pairs(mol):
    """Directed pairs within the cutoff of a typical walker."""
    ind = systems.assign_spins_to_atoms(mol.R, mol.Z)
    at = mol.R[ind].astype(np.float64)
    d = np.linalg.norm(at[:, None] - at[None], axis=-1)
    # electrons spread by sqrt(2) bohr per coordinate of a difference: a smooth step at the cutoff
    s = 1.0 / (1.0 + np.exp((np.sqrt(d**2 + 6.0) - CUTOFF) / 0.8))
    return float(s.sum() - np.trace(s))


def _value_flops(n, N, P):
    """Dense layers of one walker's value path (2 per multiply-add)."""
    f = n * 2 * F * (2 * F + F + 5 * F)  # ElecInit
    f += n * 2 * 2 * F * F  # update MLP
    f += n * 2 * (8 * N) * DETS * n + n * 2 * F * DETS * n  # envelopes, orbitals
    f += n * 2 * (3 * F * F + F * HEADS) + 2 * (2 * F * F + F * F)  # Jastrow
    f += P * 2 * 12 * F + n * N * 2 * 12 * F  # edges
    return f + DETS * 2.0 / 3.0 * n**3


def _eloc_flops(n, N, P):
    rows = 2 * n + 3 * (n + P)
    f = 5 * n * 2 * F * 8 * F + rows * 2 * 2 * F * F
    f += 5 * n * 2 * (8 * N) * DETS * n + rows * 2 * F * DETS * n
    f += rows * 2 * (3 * F * F + F * HEADS) + (3 * n + 2) * 2 * (2 * F * F + F * F)
    f += 5 * (P + n * N) * 2 * 12 * F
    c = 1.0 + P / n
    return f + DETS * 2.0 * n**3 + DETS * n * 2 * 3 * c * c * n


def _one_work(kind, mol, case, walkers):
    n, N = mol.n_el, mol.n_nuc
    P = _mean_pairs(mol)
    es = 8 if case["precision"] == "fp64" else 4
    slots = 2 * F * DETS * n + 2 * N * DETS * 8 * n + 2 * N * F + 1_200_000  # parameters
    if kind in ("eloc", "ragged"):
        return dict(flops=walkers * _eloc_flops(n, N, P), bytes=es * (slots + walkers * (3 * n + 3)))
    if kind == "logpsi":
        return dict(flops=walkers * _value_flops(n, N, P), bytes=es * (slots + walkers * (3 * n + 2)))
    if kind == "grad":
        return dict(flops=3 * walkers * _value_flops(n, N, P), bytes=es * (slots + walkers * (3 * n + 2 + slots)))
    full = _value_flops(n, N, P)
    k = 1.0 + 1.4 * P / n  # rows that a single move changes
    per_step = full if case["proposal"] == "all-electron" else full * min(1.0, k / n) + DETS * 4 * n * n * k * 0.5
    start = full if case["proposal"] == "all-electron" else 2 * full + DETS * 4.0 / 3.0 * n**3
    return dict(flops=walkers * (start + case["steps"] * per_step), bytes=es * (slots + walkers * 6 * n))


def work(case):
    if case["kind"] == "ragged":
        sizes, counts = _ragged_sizes(case)
        parts = [_one_work("ragged", systems.alkane(n), case, b) for n, b in zip(sizes, counts)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    return _one_work(case["kind"], _molecule(case["mol"], case["size"]), case, case["walkers"])


# ------------------------------------------------------------------------------------------------ exact values
# The wavefunction written densely in torch, in 64 bits: every electron pair and every electron-nucleus pair is
# evaluated, and the filters' cutoff functions make those beyond the cutoffs vanish.
def _cutoff_fn(x):
    y = 1 - 15 * x**4 + 24 * x**5 - 10 * x**6
    return torch.where(x < 1, y, torch.zeros_like(y))


def _silu(x):
    return x * torch.sigmoid(x)


def _features(diff):
    dist = diff.square().sum(-1, keepdim=True).sqrt()
    feat = torch.cat([dist, diff], -1)
    return dist, feat, feat / dist * torch.log1p(dist)


def _filter(dist, pre, dir_w, dir_b, scales, env_w, cutoff):
    env = torch.exp(-((dist / torch.nn.functional.softplus(scales)) ** 2)) * _cutoff_fn(dist / cutoff)
    return (_silu(pre) @ dir_w + dir_b) * (env @ env_w)


def _dense_logpsi(p, r, R, n_up):
    """(sign, log|psi|) of walkers r [B, n, 3]; p: dict of float64 tensors."""
    B, n, _ = r.shape
    dist, feat, scaled = _features(r[:, :, None] - R)
    pre = torch.einsum("bnek,ekf->bnef", feat, p["en_kernel"]) + p["en_bias"]
    gamma = _filter(dist, pre, p["ei_dir_W"], p["ei_dir_b"], p["en_scales"], p["ei_env_W"], CUTOFF_1EL) @ p["ei_gamma_W"]
    h = (gamma * (scaled @ p["ei_edge_W"] + p["en_nuc_emb"])).sum(2)
    mu = h.mean(-1, keepdim=True)
    var = (h - mu).square().mean(-1, keepdim=True)
    h = (h - mu) / (var + 1e-6).sqrt() * p["ei_ln_scale"] + p["ei_ln_bias"]
    g = h @ p["ei_glu_W"]
    h = _silu((g[..., :F] * _silu(g[..., F:])) @ p["ei_dense_W"] + p["ei_dense_b"])
    h, ct_s, ct_d, nb_s, nb_d = torch.split(h @ p["ei_out_W"] + p["ei_out_b"], F, -1)
    cutoff = CUTOFF * torch.sigmoid(p["cutoff_param"][0])
    eye = torch.eye(n, dtype=torch.bool, device=r.device)
    blocks = []
    for lo, hi in ((0, n_up), (n_up, n)):
        total = h[:, lo:hi]
        for nlo, nhi in ((0, n_up), (n_up, n)):
            same = nlo == lo
            tag, ct, nb = ("same", ct_s, nb_s) if same else ("diff", ct_d, nb_d)
            if hi == lo or nhi == nlo:
                continue
            own = eye[lo:hi, nlo:nhi, None]
            diff = torch.where(own, torch.full_like(r[:1, :1, :1], 100.0), r[:, lo:hi, None] - r[:, None, nlo:nhi])
            dist, feat, scaled = _features(diff)
            pre = feat @ p[f"ee{tag}_kernel"] + p[f"ee{tag}_bias"]
            beta = _filter(dist, pre, p[f"ee{tag}_dir_W"], p[f"ee{tag}_dir_b"], p[f"ee{tag}_scale"],
                           p[f"ee{tag}_env_W"], cutoff)
            edge = scaled @ p[f"ee{tag}_edge_W"] + p[f"ee{tag}_edge_b"]
            msg = _silu(edge + ct[:, lo:hi, None] + nb[:, None, nlo:nhi])
            total = total + ((beta @ p[f"ee{tag}_gamma_W"]) * msg).sum(2)
        blocks.append(total)
    h = torch.cat(blocks, 1)
    h = _silu((h * p["scales"][0]) @ p["upd1_W"] + p["upd1_b"])
    h = _silu(h @ p["upd2_W"] + p["upd2_b"]) * p["scales"][1]
    rows = []
    for tag, lo, hi in (("up", 0, n_up), ("dn", n_up, n)):
        d = (r[:, lo:hi, None] - R).square().sum(-1).sqrt()
        ex = torch.exp(-d[..., None, None] * torch.nn.functional.softplus(p[f"env_{tag}_sigma"]))
        N = R.shape[0]
        env = torch.einsum("bmdq,dqo->bmdo", ex.permute(0, 1, 3, 2, 4).reshape(B, hi - lo, DETS, -1),
                           p[f"env_{tag}_pi"].permute(1, 0, 2, 3).reshape(DETS, N * ex.shape[-1], n))
        rows.append((h[:, lo:hi] @ p[f"orb_{tag}_W"] + p[f"orb_{tag}_b"]) * env.reshape(B, hi - lo, -1))
    A = torch.cat(rows, 1).reshape(B, n, DETS, n).transpose(1, 2)
    sign, logdet = torch.linalg.slogdet(A)
    top = logdet.detach().max(-1, keepdim=True).values
    s = (sign * torch.exp(logdet - top)).sum(-1)
    log_det = top[..., 0] + s.abs().log()
    # Jastrow: cusps, attention readout, MLP
    ia, ib = torch.triu_indices(n, n, 1, device=r.device)
    d = (r[:, ia] - r[:, ib]).square().sum(-1).sqrt()
    same = (ia < n_up) == (ib < n_up)
    a_s, a_d, f_s, f_d = p["cusp"]
    cusp = torch.where(same, f_s * a_s**2 / (a_s + d), f_d * a_d**2 / (a_d + d)).sum(-1)
    q = (h @ p["att_Q_W"] + p["att_Q_b"]).reshape(B, n, HEADS, HDIM)
    v = (h @ p["att_V_W"] + p["att_V_b"]).reshape(B, n, HEADS, HDIM)
    att = torch.exp(-(q * p["att_keys"]).sum(-1) / math.sqrt(HDIM))
    x = torch.stack([(att[:, lo:hi, :, None] * v[:, lo:hi]).sum(1) / att[:, lo:hi].sum(1)[..., None]
                     for lo, hi in ((0, n_up), (n_up, n))], 1).reshape(B, -1)
    x = _silu(x @ p["att_out1_W"] + p["att_out1_b"])
    x = _silu(x @ p["att_out2_W"] + p["att_out2_b"])
    J = (x @ p["att_out3_W"] + p["att_out3_b"]) * p["att_scale"]
    m = _silu(h @ p["jmlp1_W"] + p["jmlp1_b"])
    m = _silu(m @ p["jmlp2_W"] + p["jmlp2_b"])
    m = _silu(m @ p["jmlp3_W"] + p["jmlp3_b"]) * p["mlp_scale"]
    J0 = J[:, 0] + m[..., 0].sum(1)
    J1 = J[:, 1] + p["att_bias"][0] + m[..., 1].sum(1) + n * p["log_bias"][0]
    return torch.sign(s.detach() * J1.detach()), log_det + cusp + J0 + J1.abs().log()


def _potential(r, R, Z):
    n = r.shape[1]
    ia, ib = torch.triu_indices(n, n, 1, device=r.device)
    e = (1.0 / (r[:, ia] - r[:, ib]).norm(dim=-1)).sum(-1)
    e = e - (Z / (r[:, :, None] - R).norm(dim=-1)).sum((1, 2))
    if len(R) > 1:
        ia, ib = torch.triu_indices(len(R), len(R), 1, device=r.device)
        e = e + (Z[ia] * Z[ib] / (R[ia] - R[ib]).norm(dim=-1)).sum()
    return e


def _exact_walkers(mol, p, walkers, energy):
    dev = "cuda"
    n, N = mol.n_el, mol.n_nuc
    n_up, _ = systems.spin_counts(mol)
    r_all = torch.from_numpy(walkers).to(dev, torch.float64)
    R = torch.from_numpy(mol.R).to(dev, torch.float64)
    Z = torch.from_numpy(mol.Z).to(dev, torch.float64)
    per = 8.0 * F * n * (n + N) * (60 if energy else 12)  # bytes of intermediates per walker
    step = max(1, int((20e9 if energy else 8e9) / per))
    sign, logpsi, eloc = [], [], []
    for k in range(0, len(r_all), step):
        r = r_all[k:k + step].clone()
        if not energy:
            with torch.no_grad():
                s, l = _dense_logpsi(p, r, R, n_up)
        else:
            r.requires_grad_(True)
            s, l = _dense_logpsi(p, r, R, n_up)
            (g,) = torch.autograd.grad(l.sum(), r, create_graph=True)
            lap = torch.zeros_like(l)
            for i in range(n):
                for c in range(3):
                    (h,) = torch.autograd.grad(g[:, i, c].sum(), r, retain_graph=True)
                    lap += h[:, i, c]
            with torch.no_grad():
                eloc.append(-0.5 * (lap + g.square().sum((1, 2))) + _potential(r, R, Z))
        sign.append(s.detach())
        logpsi.append(l.detach())
    return torch.cat(sign), torch.cat(logpsi), torch.cat(eloc) if energy else None


def _device_params(mol, seed):
    return {k: torch.from_numpy(v).to("cuda", torch.float64) for k, v in _params(mol, seed).items()}


def _energy_is_quick(mol, walkers):
    """3n second-derivative passes over dense pair tensors: minutes for the larger molecules."""
    return walkers * float(mol.n_el) * _dense_pairs(mol) < 2.0e7


def _dense_pairs(mol):
    return mol.n_el * (mol.n_el + mol.n_nuc)


def exact(case, seed):
    if case["kind"] == "mcmc":
        return None  # a chain's end follows from its accept/reject decisions, not from a formula
    if case["kind"] == "ragged":
        sizes, counts = _ragged_sizes(case)
        out = []
        for i, (size, b) in enumerate(zip(sizes, counts)):
            mol = systems.alkane(size)
            quick = _energy_is_quick(mol, b * 4)
            out.append(_exact_walkers(mol, _device_params(mol, seed + 17 * i), _walkers(mol, b, seed + 17 * i), True)[2]
                       if quick else None)
        return out if any(e is not None for e in out) else None
    mol = _molecule(case["mol"], case["size"])
    walkers = _walkers(mol, case["walkers"], seed)
    p = _device_params(mol, seed)
    dense = case["walkers"] * _dense_pairs(mol)
    if dense > (1.0e7 if case["kind"] == "grad" else 1.0e8):
        return None
    if case["kind"] == "eloc":
        sign, logpsi, eloc = _exact_walkers(mol, p, walkers, _energy_is_quick(mol, case["walkers"]))
        return dict(eloc=eloc, logpsi=logpsi, sign=sign)
    if case["kind"] == "logpsi":
        sign, logpsi, _ = _exact_walkers(mol, p, walkers, False)
        return dict(logpsi=logpsi, sign=sign)
    # gradient rows in the order of the parameter slots, each slot padded to a multiple of 64 elements
    names = list(PARAM_SLOT_NAMES)
    n_up, _ = systems.spin_counts(mol)
    R = torch.from_numpy(mol.R).to("cuda", torch.float64)
    for v in p.values():
        v.requires_grad_(True)
    rows, sign, logpsi = [], [], []
    for w in range(len(walkers)):
        s, l = _dense_logpsi(p, torch.from_numpy(walkers[w:w + 1]).to("cuda", torch.float64), R, n_up)
        g = torch.autograd.grad(l[0], [p[k] for k in names], allow_unused=True)
        parts = []
        for k, x in zip(names, g):
            x = torch.zeros_like(p[k]) if x is None else x
            parts.append(torch.nn.functional.pad(x.reshape(-1), (0, -x.numel() % 64)))
        rows.append(torch.cat(parts))
        sign.append(s.detach())
        logpsi.append(l.detach())
    return dict(grad=torch.stack(rows), logpsi=torch.cat(logpsi), sign=torch.cat(sign))
