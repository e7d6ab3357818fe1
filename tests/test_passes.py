"""Walkers per pass of the local energy (csrc/fire_passes.h): the rule, compiled for the host, and the passes that calls take."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from sparse_wf_gb300 import _lib, params as P, systems

CSRC = Path(__file__).resolve().parents[1] / "sparse_wf_gb300" / "csrc"


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("passes")
    src = d / "passes.cpp"
    src.write_text('#include "fire_passes.h"\n'
                   'extern "C" int walkers(long b, int c, int m, int p) { return fire::pass_walkers(b, c, m, p); }\n'
                   'extern "C" long rounds(long b, long c, int m, int p) { return fire::elimination_rounds(b, c, m, p); }\n')
    so = d / "passes.so"
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(src), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.walkers.argtypes = [C.c_long, C.c_int, C.c_int, C.c_int]
    lib.rounds.argtypes = [C.c_long, C.c_long, C.c_int, C.c_int]
    lib.rounds.restype = C.c_long
    return lib


def _rounds(b, c, places):
    return sum(-(-4 * min(c, b - w) // places) for w in range(0, b, c))


def test_rule_saves_rounds(rule):
    """Never more walkers than asked for, never more rounds, and a round less for every pass more; a whole batch stays whole."""
    rng = np.random.default_rng(0)
    for _ in range(3000):
        b, c, places = int(rng.integers(1, 3000)), int(rng.integers(1, 400)), int(rng.choice([0, 2, 152, 304, 608]))
        d = rule.walkers(b, c, 4, places)
        assert 1 <= d <= c
        if c >= b or places < 4:
            assert d == c
        if d < c:
            assert rule.rounds(b, c, 4, places) == _rounds(b, c, places) and rule.rounds(b, d, 4, places) == _rounds(b, d, places)
            assert _rounds(b, c, places) - _rounds(b, d, places) >= max(1, -(-b // d) - -(-b // c))


@pytest.mark.parametrize("b,c,want", [(77, 77, 77), (100, 100, 100), (100, 90, 76), (150, 150, 150), (153, 153, 153),
                                      (512, 153, 152), (512, 171, 152), (512, 146, 146), (2048, 152, 152), (2048, 227, 227)])
def test_rule_at_304_places(rule, b, c, want):
    assert rule.walkers(b, c, 4, 304) == want


@pytest.mark.gpu
@pytest.mark.parametrize("walkers", [77, 100])
def test_batch_that_fits_its_pass_is_one_pass(cuda_lib, walkers):
    """A fixed pass of the whole batch launches what a pass of the workspace's choosing does, for matrices of the large blocks."""
    import torch

    from sparse_wf_gb300.wavefunction import FireWaveFunction

    mol = systems.hydrogen_chain(226, 1.8)
    n_up, _ = systems.spin_counts(mol)
    dims = P.ModelDims(mol.n_el, n_up, mol.n_nuc)
    p = P.activate_jastrow(P.init_params(dims, 5))
    p["scales"] = np.array([2.0, 3.0])
    wf = FireWaveFunction(mol, precision="mixed")
    wf.refine = False
    dev = wf._params(p)
    r = wf._electrons(systems.init_electrons(mol, walkers, 3))
    static = wf.get_static_input(r).round_with_padding(1.1, mol.n_el, wf.n_up, mol.n_nuc)
    launches = []
    for chunk in (0, walkers):
        wf.chunk_walkers = chunk
        wf.local_energy_full(dev, r, static)
        _lib.profile_enable(True)
        try:
            wf.local_energy_full(dev, r, static)
            torch.cuda.synchronize()
            launches.append(_lib.profile_report()["kernels_launched"][0])
        finally:
            _lib.profile_enable(False)
    assert launches[0] == launches[1]
