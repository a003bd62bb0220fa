"""Every H*v path against the general row kernel (HPHI_B200_KERNEL=general, itself pinned to the
reference by test_gpu_parity) at the sizes where a path can go wrong: the shapes of the row, block
and tile kernels and one below and above their limits, odd row lengths, one-row sectors,
coefficient groups up to and past what a plan holds.  Each case names the kernel it is there for,
which the engine has to report (hv_plan, the decision its launches take)."""
import os

import numpy as np
import pytest

import hphi_b200
from hphi_b200 import expert

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _open(path, general=False):
    saved = os.environ.get("HPHI_B200_KERNEL")
    os.environ.pop("HPHI_B200_KERNEL", None)
    if general:
        os.environ["HPHI_B200_KERNEL"] = "general"
    try:
        return hphi_b200.Hamiltonian(path)
    finally:
        os.environ.pop("HPHI_B200_KERNEL", None)
        if saved is not None:
            os.environ["HPHI_B200_KERNEL"] = saved


def _compare(m, tmp_path, vts=(hphi_b200.REAL64, hphi_b200.COMPLEX128), plan=None):
    """v0 = acc v0 + scale H v1 and <v1|H|v1>, both paths: mltply_device on vectors in HPhi's order and
    mltply_device_async between the changes of order, as the drivers' loops run (the product layout has
    kernels of its own for complex vectors there).  plan: the kernel expected for each vector type.
    Bound: a row sums at most
    ~200 products in another order, so |difference| <= 200 eps |H| |v| elementwise; 1e-13 of the
    largest element leaves a margin for the sums' size."""
    path = m.write(str(tmp_path))
    Ha, Hg = _open(path), _open(path, general=True)
    try:
        for vt in vts:
            if plan is not None:
                got = Ha.hv_plan(vt)
                want = plan if isinstance(plan, tuple) else (plan, None)
                assert got["kernel"] == want[0] and want[1] in (None, got["shape"]), got
            assert Hg.hv_plan(vt)["kernel"] == "general"
            dt = torch.float64 if vt == hphi_b200.REAL64 else torch.complex128
            g = torch.Generator(device="cuda").manual_seed(7)
            v1 = torch.randn(Ha.dim, dtype=dt, device="cuda", generator=g)
            w = torch.randn(Ha.dim, dtype=dt, device="cuda", generator=g)
            for acc, scale in ((0.0, 1.0), (0.5, -2.0)):
                out, pr = [], []
                for H in (Ha, Hg):
                    v0 = w.clone() if acc else torch.full_like(w, float("nan"))
                    torch.cuda.synchronize()
                    pr.append(H.mltply_device(v0.data_ptr(), v1.data_ptr(), vt, acc=acc, scale=scale))
                    out.append(v0)
                big = out[1].abs().max().item()
                assert (out[0] - out[1]).abs().max().item() <= 1e-13 * big
                n = torch.linalg.vector_norm(v1).item() * torch.linalg.vector_norm(out[1]).item()
                assert abs(pr[0] - pr[1]) <= 1e-13 * max(n, abs(pr[1]))
                a, b, o = (torch.zeros_like(v1) for _ in range(3))
                coef = torch.tensor([acc, scale], dtype=torch.float64, device="cuda")
                pa = torch.zeros(2, dtype=torch.float64, device="cuda")
                w0 = w if acc else torch.full_like(w, float("nan"))
                torch.cuda.synchronize()
                Ha.to_native(v1.data_ptr(), a.data_ptr(), vt)
                Ha.to_native(w0.data_ptr(), b.data_ptr(), vt)
                Ha.mltply_device_async(b.data_ptr(), a.data_ptr(), vt, coef.data_ptr(), pa.data_ptr())
                Ha.from_native(b.data_ptr(), o.data_ptr(), vt)
                assert (o - out[1]).abs().max().item() <= 1e-13 * big
                assert abs(complex(*pa.tolist()) - pr[1]) <= 1e-13 * max(n, abs(pr[1]))
        return Ha.info["kernel"]
    finally:
        Ha.close()
        Hg.close()


def _dm_chain(L, two_sz):
    """Complex exchange: InterAll J/2 (e^{ia} S+S- + h.c.) beside the Ising part."""
    m = expert.heisenberg(L, expert.chain_bonds(L), two_sz=two_sz)
    m.exchange = []
    for i, j in expert.chain_bonds(L):
        m.interall += [(i, 0, i, 1, j, 1, j, 0, 0.4, 0.3), (j, 0, j, 1, i, 1, i, 0, 0.4, -0.3)]
    return m


def _couplings(L, n):
    """A chain whose bonds within the lower half take n different couplings."""
    b = expert.chain_bonds(L) + expert.chain_bonds(L, 2)
    lower = [x for x in b if max(x) < L // 2]
    assert n <= len(lower)
    return expert.heisenberg(L, b, [1.0 + 0.1 * (lower.index(x) % n if x in lower else 0) for x in b], two_sz=L % 2)


def _nconserved(L, ne):
    m = expert.hubbard(L, expert.chain_bonds(L), 1.0, 3.0, 1, 1)
    m.ncond, m.two_sz = ne, None
    for i in range(L):
        m.trans += [(i, 0, (i + 1) % L, 1, 0.3, 0.0), ((i + 1) % L, 1, i, 0, 0.3, 0.0)]
    return m


BLOCK = {   # name: (shape of the planes, or the kernel instead of the block kernel; model)
    # longest blocks of 1, 3, 6, 70, 252, 924, 1716, 3432, 6435 and 12870 rows: every plane shape
    "chain2": (0, lambda: expert.heisenberg(2, [(0, 1)])),
    "chain3": (0, lambda: expert.heisenberg(3, expert.chain_bonds(3), two_sz=1)),
    "chain5": (0, lambda: expert.heisenberg(5, expert.chain_bonds(5), two_sz=-1)),
    "chain16": (0, lambda: expert.heisenberg(16, expert.chain_bonds(16))),
    "j1j2_19": (1, lambda: expert.heisenberg(19, expert.chain_bonds(19) + expert.chain_bonds(19, 2), two_sz=1)),
    "square4x6": (3, lambda: expert.heisenberg(24, expert.square_bonds(4, 6))),
    "chain26_few": (4, lambda: expert.heisenberg(26, expert.chain_bonds(26), two_sz=-12)),
    "chain28_few": (5, lambda: expert.heisenberg(28, expert.chain_bonds(28), two_sz=-14)),
    "chain30_few": (6, lambda: expert.heisenberg(30, expert.chain_bonds(30), two_sz=-16)),
    "chain32_few": (7, lambda: expert.heisenberg(32, expert.chain_bonds(32), two_sz=-16)),
    "groups8": (0, lambda: _couplings(12, 8)),
    "groups9": ("general", lambda: _couplings(12, 9)),     # more than a plan holds
    "kondo4": (0, lambda: expert.kondo_chain(4, 1.0, 1.5, U=2.0)),
    "kondo7_odd": (0, lambda: expert.kondo_chain(6, 1.0, 0.7, ncond=5, two_sz=1)),
    # few blocks, longer than one turn of a CTA's threads: shared out over several tasks
    "kondo8": (2, lambda: expert.kondo_chain(8, 1.0, 1.5)),
    "spin1_14": (3, lambda: expert.general_heisenberg([2] * 14, expert.chain_bonds(14), 1.0, two_sz=0)),
    "spin1": (0, lambda: expert.general_heisenberg([2] * 7, expert.chain_bonds(7), 1.0, D=0.3)),
    "mixed_spins": (0, lambda: expert.general_heisenberg([1, 2, 3, 1, 2, 3], expert.chain_bonds(6), 0.8, two_sz=2)),
    "nconserved": (0, lambda: _nconserved(6, 5)),
}


@pytest.mark.parametrize("name", list(BLOCK))
def test_block_kernel(name, tmp_path):
    want, make = BLOCK[name]
    assert _compare(make(), tmp_path, plan=want if isinstance(want, str) else ("block", want)) == 0


def test_block_kernel_complex_coefficients(tmp_path):
    _compare(_dm_chain(14, 0), tmp_path, vts=(hphi_b200.COMPLEX128,), plan="block")


def _spin_gc(n, field, seed=3):
    m = expert.kitaev_heisenberg(3, n // 6, -1.0, 0.3) if n % 6 == 0 else None
    if m is None:
        m = expert.heisenberg(n, expert.chain_bonds(n), 0.9)
        m.model, m.two_sz = "SpinGC", None
    rng = np.random.default_rng(seed)
    for i in range(n if field else 0):   # h.S with complex off-diagonal parts
        h = complex(rng.normal(), rng.normal()) if field == "complex" else complex(rng.normal(), 0.0)
        m.trans += [(i, 0, i, 1, h.real, h.imag), (i, 1, i, 0, h.real, -h.imag), (i, 0, i, 0, 0.1 * i, 0.0)]
    return m


def _hubbard_gc(L, complex_t=False, four_body=False):
    m = expert.hubbard(L, expert.chain_bonds(L), 1.0, 4.0, 1, 1)
    m.model, m.ncond, m.two_sz = "HubbardGC", None, None
    if complex_t:
        m.trans = []
        for i, j in expert.chain_bonds(L):
            for s in (0, 1):
                m.trans += [(i, s, j, s, 0.8, 0.3), (j, s, i, s, 0.8, -0.3)]
    m.trans += [(i, 0, i, 1, 0.2, 0.0) for i in range(L)] + [(i, 1, i, 0, 0.2, 0.0) for i in range(L)]
    if four_body:   # condition on four bits: not a tile group
        m.pairhop = [(0, 3, 0.5)]
    return m


GC = {   # name: (kernels of real and complex vectors, model)
    # below, at and above the sizes from which tiles are taken (2^19 rows complex, 2^20 real, 2^24 real with signs)
    "chain17": ("general", "general", lambda: _spin_gc(17, "real")),
    "kitaev18": ("general", "general", lambda: _spin_gc(18, None)),
    "kitaev18_field": ("general", "general", lambda: _spin_gc(18, "real")),
    "chain19": ("general", "tile", lambda: _spin_gc(19, "real")),
    "chain20": ("tile", "tile", lambda: _spin_gc(20, "real")),
    "kitaev20": ("tile", "tile", lambda: expert.kitaev_heisenberg(5, 2, -1.0, 0.3)),
    "hubbard9": ("general", "general", lambda: _hubbard_gc(9)),
    "hubbard10": ("general", "tile", lambda: _hubbard_gc(10)),   # signs over bits inside and outside a tile
    "hubbard12": ("tile", "tile", lambda: _hubbard_gc(12)),
    "hubbard9_four_body": ("general", "general", lambda: _hubbard_gc(9, four_body=True)),
    "hubbard10_four_body": ("general", "general", lambda: _hubbard_gc(10, four_body=True)),
}


@pytest.mark.parametrize("vt", [hphi_b200.REAL64, hphi_b200.COMPLEX128])
@pytest.mark.parametrize("name", list(GC))
def test_tile_kernel(name, vt, tmp_path):
    _compare(GC[name][2](), tmp_path, vts=(vt,), plan=GC[name][vt])


@pytest.mark.parametrize("m, plan", [(lambda: _spin_gc(18, "complex"), "general"), (lambda: _spin_gc(20, "complex"), "tile"),
                                     (lambda: _hubbard_gc(9, complex_t=True), "general"),
                                     (lambda: _hubbard_gc(10, complex_t=True), "tile")])
def test_tile_kernel_complex_coefficients(m, plan, tmp_path):
    _compare(m(), tmp_path, vts=(hphi_b200.COMPLEX128,), plan=plan)


def _hubbard(N, nup, ndown, phases=0, anisotropic=0):
    """Ring of N sites; `phases` hops carry their own phase, `anisotropic` their own amplitude."""
    m = expert.hubbard(N, [], 1.0, 4.0, nup, ndown)
    for k, (i, j) in enumerate(expert.chain_bonds(N)):
        t = (1.0 + 0.05 * k if k < anisotropic else 1.0) * np.exp(1j * (0.1 * (k + 1) if k < phases else 0.0))
        for s in (0, 1):
            m.trans += [(i, s, j, s, t.real, t.imag), (j, s, i, s, t.real, -t.imag)]
    return m


PROD = {   # name: (words of a row's plane, 0 for the one-pass kernel; model)
    # rows of 924, 1287 (odd), 1716, 3432, 5005 (odd) and 8008 elements: every row shape, both loads
    "n12": (960, lambda: _hubbard(12, 3, 6)),
    "n13": (1744, lambda: _hubbard(13, 2, 5)),
    "n13_6": (1744, lambda: _hubbard(13, 3, 6)),
    "n14": (3456, lambda: _hubbard(14, 2, 7)),
    "n15": (6560, lambda: _hubbard(15, 2, 6)),
    "n16": (12896, lambda: _hubbard(16, 2, 6)),
    "n7_odd": (960, lambda: _hubbard(7, 3, 3)),
    "one_row": (960, lambda: _hubbard(6, 6, 3)),
    "one_column": (960, lambda: _hubbard(6, 3, 6)),
    "two_amplitudes": (960, lambda: _hubbard(10, 5, 4, anisotropic=1)),
    "eight_amplitudes": (960, lambda: _hubbard(10, 5, 4, anisotropic=8)),
    "ten_amplitudes": (0, lambda: _hubbard(10, 5, 4, anisotropic=10)),   # past the groups: the one-pass kernel
}


@pytest.mark.parametrize("name", list(PROD))
def test_product_layout(name, tmp_path):
    words, make = PROD[name]
    assert _compare(make(), tmp_path, plan=("two_pass", words) if words else "one_pass") in (2, 3)


@pytest.mark.parametrize("phases", [1, 3, 10])
def test_product_layout_complex_coefficients(phases, tmp_path):
    _compare(_hubbard(10, 5, 4, phases=phases), tmp_path, vts=(hphi_b200.COMPLEX128,),
             plan="two_pass" if phases < 10 else "one_pass")


@pytest.mark.parametrize("N, nup, ndown", [(1, 1, 0), (5, 2, 3), (8, 4, 4), (11, 5, 6), (12, 6, 6)])
@pytest.mark.parametrize("vt", [hphi_b200.REAL64, hphi_b200.COMPLEX128])
def test_native_order_round_trip(N, nup, ndown, vt, tmp_path):
    """to_native then from_native is the identity, bit for bit (a permutation with signs)."""
    m = expert.hubbard(N, expert.chain_bonds(N) if N > 1 else [], 1.0, 4.0, nup, ndown)
    with _open(m.write(str(tmp_path))) as H:
        v = torch.randn(H.dim, dtype=torch.float64 if vt == hphi_b200.REAL64 else torch.complex128, device="cuda")
        a, b = torch.zeros_like(v), torch.zeros_like(v)
        torch.cuda.synchronize()
        H.to_native(v.data_ptr(), a.data_ptr(), vt)
        H.from_native(a.data_ptr(), b.data_ptr(), vt)
        assert torch.equal(v, b)


GREEN = {
    # longest blocks of 1, 36 (odd sector), 462 and, in pieces of 512 rows, 924
    "chain2": lambda: expert.heisenberg(2, [(0, 1)]),
    "hubbard9": lambda: expert.hubbard(9, expert.chain_bonds(9), 1.0, 3.0, 4, 5),
    "chain21": lambda: expert.heisenberg(21, expert.chain_bonds(21), two_sz=1),
    "chain24": lambda: expert.heisenberg(24, expert.chain_bonds(24)),
}


@pytest.mark.parametrize("vt", [hphi_b200.REAL64, hphi_b200.COMPLEX128])
@pytest.mark.parametrize("name", list(GREEN))
def test_green_blocks(name, vt, tmp_path):
    """<v|H|v> put together from Green's functions against the H*v's own, and adjoint rows as
    conjugates.  Bound: |v| = 1, so every function is at most 1 and sums products in another order;
    1e-13 of the sum of |coefficients| leaves a margin."""
    m = GREEN[name]()
    one, two = [], []   # (coefficient, row)
    for i, s1, j, s2, re, im in m.trans:
        one.append((-complex(re, im), (i, s1, j, s2)))
    for i, U in m.coulombintra:
        two.append((U, (i, 0, i, 0, i, 1, i, 1)))
    for i, j, J in m.ising:
        two += [(0.25 * J * (1 if a == b else -1), (i, a, i, a, j, b, j, b)) for a in (0, 1) for b in (0, 1)]
    for i, j, J in m.exchange:
        two += [(J, (i, 0, i, 1, j, 1, j, 0)), (J, (j, 0, j, 1, i, 1, i, 0))]
    with _open(m.write(str(tmp_path))) as H:
        v = torch.randn(H.dim, dtype=torch.float64 if vt == hphi_b200.REAL64 else torch.complex128, device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(5))
        v /= torch.linalg.vector_norm(v)
        w = torch.zeros_like(v)
        torch.cuda.synchronize()
        ref = H.mltply_device(w.data_ptr(), v.data_ptr(), vt, acc=0.0, scale=1.0)
        e, weight = 0.0, 0.0
        for body, rows in ((1, one), (2, two)):
            if not rows:
                continue
            g = H.expec_green_device(v.data_ptr(), vt, [r for _, r in rows], body)
            e += sum(c * x for (c, _), x in zip(rows, g))
            weight += sum(abs(c) for c, _ in rows)
            at = {r: x for (_, r), x in zip(rows, g)}
            for r, x in at.items():
                adj = r[2:4] + r[0:2] if body == 1 else r[6:8] + r[4:6] + r[2:4] + r[0:2]
                if adj in at:
                    assert abs(at[adj] - np.conj(x)) <= 1e-13
    assert abs(e - ref) <= 1e-13 * weight


@pytest.mark.parametrize("static, values", [(False, 1), (True, 1), (True, 5), (False, 12)])
def test_time_evolution_product_layout(static, values, tmp_path):
    """Energies, and files, of a run on the product layout against the general path (HPhi's order).
    static: the hops stay in H and the pulse adds to them; values: amplitudes of the pulse over the
    bonds (12 is past the coefficient groups, so that run stays on the general path).  Bound: 8
    steps of order 10 multiply rounding errors by e^(|H| dt) < 2 each; 1e-12 of the energies' scale."""
    N, steps = 8, 8
    m = _hubbard(N, 4, 3)
    m.calc_type, m.lanczos_max, m.input_eigenvec, m.expand_coef = "TimeEvolution", steps, 1, 10
    m.spectrum_vec, m.output_eigenvec, m.output_interval = "zvo_eigenvec_0", 1, steps - 1
    m.greenone = [(0, 0, 1, 0), (2, 1, 2, 1)]
    m.expec_interval = 3
    hops = list(m.trans)
    for k in range(steps):
        rows = []
        for b, (i, s1, j, s2, re, im) in enumerate(hops):
            a = 0.3 * np.sin(2.0 * k * 0.02) * (1.0 + 0.1 * ((b // 4) % values)) * (1 if (j - i) % N == 1 else -1)
            t = complex(re, im) * np.exp(1j * a) - (complex(re, im) if static else 0.0)
            rows.append((i, s1, j, s2, float(t.real), float(t.imag)))
        m.te_onebody.append((0.02 * k, rows))
    if not static:
        m.trans = []
    path = m.write(str(tmp_path))
    out = []
    for general in (False, True):
        with _open(path, general=general) as H:
            rng = np.random.default_rng(4)
            v = np.zeros(H.dim + 1, dtype=np.complex128)
            v[1:] = rng.standard_normal(H.dim) + 1j * rng.standard_normal(H.dim)
            v /= np.linalg.norm(v)
            d = str(tmp_path / f"out{general}")
            e = [H.calc_by_tem(v_init=v, output_dir=d) for _ in range(2)]
            assert np.array_equal(e[0], e[1])
            with open(os.path.join(d, "zvo_eigenvec_0_rank_0.dat"), "rb") as f:
                state = np.frombuffer(f.read()[12:], dtype=np.complex128)
            files = [np.loadtxt(os.path.join(d, n)) for n in ("Flct.dat", "SS.dat", "zvo_cisajs_step3.dat")]
            out.append((e[0], state[1:], files))
    (ea, sa, fa), (eg, sg, fg) = out
    assert np.max(np.abs(ea - eg)) <= 1e-12 * np.max(np.abs(eg))
    assert np.max(np.abs(sa - sg)) <= 1e-12 * np.max(np.abs(sg))
    for x, y in zip(fa, fg):
        np.testing.assert_allclose(x, y, rtol=0, atol=2e-10)


def _odd_copy(x):
    """x in memory that starts 8 bytes past a multiple of 16, as complex128 allows; (data pointer, view
    of the doubles, the buffer)."""
    buf = torch.zeros(2 * x.numel() + 2, dtype=torch.float64, device="cuda")
    at = 1 if buf.data_ptr() % 16 == 0 else 0
    view = buf[at:at + 2 * x.numel()]
    view.copy_(torch.view_as_real(x).reshape(-1))
    return view.data_ptr(), view, buf


ODD = {
    "block": (lambda: expert.heisenberg(16, expert.chain_bonds(16)), None),
    "row_block": (lambda: expert.heisenberg(16, expert.chain_bonds(16)), "rowblock"),
    "tiles": (lambda: _spin_gc(20, "real"), None),
    "product": (lambda: _hubbard(10, 5, 4), None),
    "product_no_up_hops": (lambda: _hubbard(6, 6, 3), None),
    "product_short_blocks": (lambda: _hubbard(9, 2, 2), None),
}


@pytest.mark.parametrize("name", list(ODD))
def test_complex_vectors_at_8_byte_boundaries(name, tmp_path, monkeypatch):
    """Every call that takes device vectors, with complex vectors at 8 mod 16 bytes (the type's own
    alignment): the results of the same call on vectors at 16 (bound of _compare; copies bit for bit)."""
    make, kernel = ODD[name]
    if kernel:
        monkeypatch.setenv("HPHI_B200_KERNEL", kernel)
    C = hphi_b200.COMPLEX128
    with hphi_b200.Hamiltonian(make().write(str(tmp_path))) as H:
        assert H.hv_plan(C)["kernel"] == {"block": "block", "row_block": "rowblock", "tiles": "tile"}.get(name, "two_pass")
        g = torch.Generator(device="cuda").manual_seed(3)
        v1, w = (torch.randn(H.dim, dtype=torch.complex128, device="cuda", generator=g) for _ in range(2))
        p1, _, keep = _odd_copy(v1)
        coef = torch.tensor([0.5, -2.0], dtype=torch.float64, device="cuda")
        pr = torch.zeros(2, 2, dtype=torch.float64, device="cuda")

        def close(view, ref, pa, pb):
            big = ref.abs().max().item()
            assert (torch.view_as_complex(view.clone().reshape(-1, 2)) - ref).abs().max().item() <= 1e-13 * big
            n = torch.linalg.vector_norm(v1).item() * torch.linalg.vector_norm(ref).item()
            assert abs(pa - pb) <= 1e-13 * n

        ref = w.clone()
        p0, o0, keep0 = _odd_copy(w)
        torch.cuda.synchronize()
        a = H.mltply_device(ref.data_ptr(), v1.data_ptr(), C, acc=0.5, scale=-2.0)
        b = H.mltply_device(p0, p1, C, acc=0.5, scale=-2.0)
        close(o0, ref, a, b)
        for native in (H.to_native, H.from_native):
            x = torch.zeros_like(v1)
            px, ox, keepx = _odd_copy(x)
            torch.cuda.synchronize()
            native(v1.data_ptr(), x.data_ptr(), C)
            native(p1, px, C)
            assert torch.equal(torch.view_as_real(x).reshape(-1), ox)
        # vectors in native order
        ref = w.clone()
        p0, o0, keep0 = _odd_copy(w)
        pn, on, keepn = _odd_copy(w)
        torch.cuda.synchronize()
        H.mltply_device_async(ref.data_ptr(), v1.data_ptr(), C, coef.data_ptr(), pr[0].data_ptr())
        if name.startswith("product") and name != "product_no_up_hops":   # refused, not read past the alignment
            for call in (lambda: H.mltply_device_async(p0, p1, C, coef.data_ptr(), pr[1].data_ptr()),
                         lambda: H.mltply_device_noalloc(pn, p1, C, acc=0.5, scale=-2.0)):
                with pytest.raises(hphi_b200.HPhiError, match="multiple of 16"):
                    call()
        else:
            H.mltply_device_async(p0, p1, C, coef.data_ptr(), pr[1].data_ptr())
            H.synchronize()
            close(o0, ref, complex(*pr[0].tolist()), complex(*pr[1].tolist()))
            close(on, ref, complex(*pr[0].tolist()), H.mltply_device_noalloc(pn, p1, C, acc=0.5, scale=-2.0))
        rows = [(0, 0, 0, 0), (0, 0, 1, 0), (1, 0, 0, 0)] if H.info["calc_model"] in (0, 3) else [(0, 0, 0, 0), (1, 1, 1, 1)]
        a = H.expec_green_device(v1.data_ptr(), C, rows, 1)
        b = H.expec_green_device(p1, C, rows, 1)
        assert np.max(np.abs(a - b)) <= 1e-13 * np.sum(np.abs(v1.cpu().numpy()) ** 2)


NONFINITE = {
    "tiles": lambda: _spin_gc(20, "real"),
    "tiles_kitaev": lambda: expert.kitaev_heisenberg(5, 2, -1.0, 0.3),
    "tiles_signs": lambda: _hubbard_gc(10),
    "block": lambda: expert.heisenberg(16, expert.chain_bonds(16)),
    "block_complex": lambda: _dm_chain(14, 0),
    "product": lambda: _hubbard(10, 5, 4),
    "product_complex": lambda: _hubbard(10, 5, 4, phases=3),
}


@pytest.mark.parametrize("vt", [hphi_b200.REAL64, hphi_b200.COMPLEX128])
@pytest.mark.parametrize("name", list(NONFINITE))
def test_non_finite_elements_reach_their_neighbours_only(name, vt, tmp_path):
    """An infinity in v1 changes the rows that H couples to it and no other: elsewhere H v1 is that of
    the vector with a zero in its place, exactly (the terms of those rows are the same)."""
    if vt == hphi_b200.REAL64 and name.endswith("complex"):
        pytest.skip("complex H")
    dt = torch.float64 if vt == hphi_b200.REAL64 else torch.complex128
    path = NONFINITE[name]().write(str(tmp_path))
    with _open(path) as H, _open(path, general=True) as Hg:
        v = torch.randn(H.dim, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(11))
        at = H.dim // 3
        probe = torch.zeros_like(v)
        probe[at] = 1.0
        out = {}
        for key, vec, h in (("near", probe, Hg), ("zero", v.clone(), H), ("inf", v.clone(), H)):
            if key != "near":
                vec[at] = 0.0 if key == "zero" else float("inf")
            out[key] = torch.zeros_like(v)
            torch.cuda.synchronize()
            coef = torch.tensor([0.0, 1.0], dtype=torch.float64, device="cuda")
            pr = torch.zeros(2, dtype=torch.float64, device="cuda")
            a, b = torch.zeros_like(v), torch.zeros_like(v)
            torch.cuda.synchronize()
            h.to_native(vec.data_ptr(), a.data_ptr(), vt)
            h.mltply_device_async(b.data_ptr(), a.data_ptr(), vt, coef.data_ptr(), pr.data_ptr())
            h.from_native(b.data_ptr(), out[key].data_ptr(), vt)
        far = out["near"] == 0
        far[at] = False
        assert 0 < int((~far).sum()) < H.dim
        assert torch.equal(out["inf"][far], out["zero"][far])
        assert not torch.isfinite(torch.view_as_real(out["inf"]) if dt == torch.complex128 else out["inf"]).all()
