"""TPQ samples in lockstep (hphi_tpq groups the NumAve samples of the reference's loop,
src/CalcByTPQ.c:76, into blocks that share one H*V per H application, hv_block_native):
every output file must equal the one-sample-at-a-time run (HPHI_B200_TPQ_BLOCK=0) digit for
digit, since per vector the block kernel does the general kernel's arithmetic in its order.
HPHI_B200_TPQ_BLOCK caps the block size (0: one sample at a time)."""
import os

import pytest

import hphi_b200
from hphi_b200 import expert

pytestmark = pytest.mark.gpu


def _models():
    out = {}
    # microcanonical TPQ, complex vectors (the reference's default), 10 samples: blocks of 8 and 2
    m = expert.heisenberg(12, expert.chain_bonds(12) + expert.chain_bonds(12, 2), J=[1.0] * 12 + [0.4] * 12,
                          calc_type="TPQ", lanczos_max=60, num_ave=10, large_value=3.0, expec_interval=20,
                          initial_vec_type=0)
    out["tpq_j1j2_chain12"] = m
    # canonical TPQ on a grand-canonical spin model, real vectors
    m = expert.kitaev_heisenberg(2, 2, 1.0, 0.3, calc_type="cTPQ", lanczos_max=30, num_ave=3, large_value=5.0)
    out["ctpq_kitaev2x2"] = m
    # a grand-canonical Hubbard sector with Green's functions every ExpecInterval steps
    m = expert.hubbard(5, expert.chain_bonds(5), 1.0, 4.0, 3, 2, calc_type="TPQ", lanczos_max=25, num_ave=4,
                       large_value=4.0, expec_interval=10)
    m.model, m.two_sz, m.ncond = "HubbardGC", None, None
    m.greenone = [(i, s, i, s) for i in range(5) for s in (0, 1)]
    out["tpq_hubbardgc5_green"] = m
    return out


MODELS = _models()


@pytest.mark.parametrize("name", sorted(MODELS))
def test_block_samples_equal_serial_samples(name, tmp_path, monkeypatch):
    d = tmp_path / "in"
    MODELS[name].write(str(d))
    outs = {}
    for mode in ("0", "8", "3"):  # one after another; blocks of up to 8; blocks of up to 3
        monkeypatch.setenv("HPHI_B200_TPQ_BLOCK", mode)
        o = tmp_path / f"out{mode}"
        with hphi_b200.Hamiltonian(str(d / "namelist.def")) as H:
            assert H.info["kernel"] == 0  # the general kernel: samples share block products
            H.calc_by_tpq(output_dir=str(o))
        outs[mode] = o
    files = sorted(os.listdir(outs["0"]))
    assert any(f.startswith("SS_rand") for f in files)
    for mode in ("8", "3"):
        assert files == sorted(os.listdir(outs[mode]))
        for f in files:
            assert (outs["0"] / f).read_text() == (outs[mode] / f).read_text(), (mode, f)


def _larger(kind):
    if kind == "chain14":
        m = expert.heisenberg(14, expert.chain_bonds(14), calc_type="TPQ", lanczos_max=12, large_value=3.0)
    else:   # a sector whose single H*v goes by tiles
        m = expert.kitaev_heisenberg(5, 2, 1.0, 0.3, calc_type="TPQ", lanczos_max=12, large_value=3.0)
    m.initial_vec_type = 1
    return m


@pytest.mark.parametrize("num_ave", [1, 3])
@pytest.mark.parametrize("kind", ["chain14", "kitaev5x2"])
def test_samples_of_planned_sectors(kind, num_ave, tmp_path, monkeypatch):
    """Sectors with a plan for single products: the same files whatever the block size, the contiguous
    start array (hphi_tpq) and one pointer per sample give the same numbers, and one sample alone and the
    general kernel agree (bound: 12 steps of order 10 multiply rounding by at most 2 each; 1e-11 of L)."""
    import ctypes

    import numpy as np
    m = _larger(kind)
    m.num_ave = num_ave
    path = m.write(str(tmp_path / "in"))
    rng = np.random.default_rng(2)
    runs = {}
    for mode in ("0", "8", "contiguous", "general"):
        monkeypatch.setenv("HPHI_B200_TPQ_BLOCK", mode if mode in "08" else "8")
        if mode == "general":
            monkeypatch.setenv("HPHI_B200_KERNEL", "general")
        o = str(tmp_path / f"out{mode}")
        with hphi_b200.Hamiltonian(path) as H:
            if not runs:
                starts = np.zeros((num_ave, H.dim + 1), dtype=np.complex128)
                starts[:, 1:] = rng.standard_normal((num_ave, H.dim))
            if mode == "contiguous":
                e = np.zeros(H.info["lanczos_max"])
                ptr = starts.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
                out = e.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
                assert hphi_b200.load_library().hphi_tpq(H.handle, ptr, os.fsencode(o), out, e.size) == 0
            else:
                e = H.calc_by_tpq(v_init=list(starts), output_dir=o)
        runs[mode] = (e, {f: open(os.path.join(o, f)).read() for f in sorted(os.listdir(o))})
    for mode in ("8", "contiguous"):
        assert np.array_equal(runs[mode][0], runs["0"][0]) and runs[mode][1] == runs["0"][1]
    assert np.max(np.abs(runs["general"][0] - runs["0"][0])) <= 1e-11 * 3.0 * m.nsite
