"""What the prepared-parameter buffer and the workspace hold, through the C ABI (host arithmetic: no GPU)."""
import ctypes as C

import pytest

from sparse_wf_gb300 import _lib, systems

F, DETS = 256, 4


def _problem(mol, precision, walkers=1, pairs=1, chunk=0, refine=0):
    n_up, _ = systems.spin_counts(mol)
    return _lib.Problem(mol.n_el, n_up, mol.n_nuc, walkers, 5.0, 20.0, pairs, mol.n_nuc, _lib.PREC[precision], chunk, refine)


def _size(fn, *args):
    n = C.c_size_t()
    _lib.check(fn(*args, C.byref(n)), "size")
    return n.value


def _align(x):
    return (x + 255) // 256 * 256


def _slices(n_el, fp64):
    """Bytes of the sliced weights: per K x N weight, tiles of up to 64 (FP64) or 80 columns of 8 or 6 slices, 16 k deep, and
    one exponent per column; the attention readout's two weights are sliced in FP64 only."""
    shapes = [(F, 2 * F), (F, F), (F, 5 * F), (F, F), (F, F), (F, DETS * n_el), (F, DETS * n_el), (F, F), (F, F), (F, F)]
    if fp64:
        shapes += [(2 * F, F), (F, F)]
    width, count = (64, 8) if fp64 else (80, 6)
    return sum(_align(-(-n // width) * -(-k // 16) * count * 32 * width + _align(4 * n)) for k, n in shapes)


@pytest.mark.parametrize("mol", [systems.hydrogen_chain(10, 1.8), systems.alkane(2), systems.alkane(40)], ids=["h10", "c2h6", "c40h82"])
def test_fp64_copy_of_an_fp32_buffer_has_no_slices(mol):
    """The FP64 build's buffer is its slots and their slices; the FP32 build's is its slots, the value path's slices and the
    FP64 slots of the refinement pass, which slices nothing."""
    lib = _lib.load()
    size64 = _size(lib.fire_prepared_size, C.byref(_problem(mol, "fp64")))
    slots = (size64 - _slices(mol.n_el, True)) // 8
    assert _align(8 * slots) + _slices(mol.n_el, True) == size64
    size32 = _size(lib.fire_prepared_size, C.byref(_problem(mol, "fp32")))
    assert size32 == _align(4 * slots) + _slices(mol.n_el, False) + 8 * slots


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("walkers", [1, 2, 77])
def test_workspace_serves_value_and_energy_calls(precision, walkers):
    """fire_workspace_size covers the local energy and the value path of as many walkers: more room for refined walkers
    never shrinks it, and a call of one walker of two electrons has room for whole 128-row tiles of slices."""
    lib = _lib.load()
    mol = systems.hydrogen_chain(2, 1.8)
    size = [_size(lib.fire_workspace_size, C.byref(_problem(mol, precision, walkers, 2, 0, r)), walkers) for r in (0, 1, walkers)]
    assert size == sorted(size)
    tile = 128 * F * 2 * (8 if precision == "fp64" else 6)
    assert size[0] >= tile


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("mol,pairs,walkers,chunk", [(systems.alkane(40), 8000, 2048, 152), (systems.alkane(10), 1500, 2048, 610),
                                                     (systems.hydrogen_chain(10, 1.8), 80, 512, 16), (systems.alkane(2), 200, 512, 3)])
def test_room_for_refined_walkers_is_one_pass(mol, pairs, walkers, chunk, precision):
    """Before any count is known the refinement has room for a quarter of the batch, but for no more than one pass (the least
    room is two walkers), and a pass's workspace holds it."""
    from sparse_wf_gb300.wavefunction import FireWaveFunction, StaticArgs

    lib = _lib.load()
    wf = FireWaveFunction(mol, precision=precision, device="cpu", chunk_walkers=chunk)
    static = StaticArgs(pairs // 2, pairs - pairs // 2, 0, mol.n_nuc)
    prob = wf._problem(walkers, static, refine=True)
    assert 2 <= prob.refine_cap <= min(chunk, -(-walkers // 4))
    bare = wf._problem(walkers, static)
    room = _size(lib.fire_workspace_size, C.byref(prob), chunk) - _size(lib.fire_workspace_size, C.byref(bare), chunk)
    assert room <= _align((2 * prob.refine_cap + 1) * 4)  # the list of walkers
