"""The device memory that a handle keeps between the drivers' calls: bounded over all handles, given back,
and without influence on results; and the H*v launches, chained ones among them, in a CUDA graph."""
import numpy as np
import pytest

import hphi_b200
from hphi_b200 import expert

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kept_memory_is_bounded_over_handles(tmp_path):
    """Twelve handles whose Lanczos runs take 43 MB each: together they keep 256 MB at most (16 MB for
    what the allocator rounds), and closing them gives all of it back."""
    path = expert.heisenberg(24, expert.chain_bonds(24)).write(str(tmp_path))
    with hphi_b200.Hamiltonian(path) as H:   # modules, first allocations of the process
        H.lanczos_steps(2)
    start = _free()
    hs = [hphi_b200.Hamiltonian(path) for _ in range(12)]
    opened = _free()
    e = [H.lanczos_steps(6, seed=5)[0] for H in hs]
    assert opened - _free() <= (256 + 16) << 20
    assert len(set(e)) == 1   # kept or not, the same numbers
    for H in hs:
        H.close()
    assert start - _free() <= 16 << 20


def test_calls_of_different_sizes_share_a_handle(tmp_path):
    """A small call, a larger one, the small one again: each as on a handle of its own."""
    m = expert.heisenberg(14, expert.chain_bonds(14), calc_type="TPQ", lanczos_max=8, num_ave=5, large_value=3.0)
    path = m.write(str(tmp_path / "in"))
    rng = np.random.default_rng(1)
    with hphi_b200.Hamiltonian(path) as H:
        starts = np.zeros((5, H.dim + 1), dtype=np.complex128)
        starts[:, 1:] = rng.standard_normal((5, H.dim))
        calls = [lambda H: H.lanczos_steps(8, seed=3), lambda H: H.calc_by_tpq(v_init=list(starts), output_dir=str(tmp_path / "o")),
                 lambda H: H.lanczos_steps(8, seed=3)]
        shared = [c(H) for c in calls]
    for c, r in zip(calls, shared):
        with hphi_b200.Hamiltonian(path) as H:
            assert np.array_equal(c(H), r)


MODELS = {
    "block": (lambda: expert.heisenberg(16, expert.chain_bonds(16)), hphi_b200.REAL64),
    "tiles": (lambda: expert.kitaev_heisenberg(5, 2, -1.0, 0.3), hphi_b200.COMPLEX128),
    "product": (lambda: expert.hubbard(8, expert.square_bonds(2, 4), 1.0, 4.0, 4, 4), hphi_b200.REAL64),
}


@pytest.mark.parametrize("name", list(MODELS))
def test_products_in_a_graph(name, tmp_path):
    make, vt = MODELS[name]
    with hphi_b200.Hamiltonian(make().write(str(tmp_path))) as H:
        dt = torch.float64 if vt == hphi_b200.REAL64 else torch.complex128
        v = torch.randn(H.dim, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
        v /= torch.linalg.vector_norm(v)
        a, b = v.clone(), torch.zeros_like(v)
        coef = torch.tensor([-0.5, 0.25], dtype=torch.float64, device="cuda")
        mu = torch.zeros(6, 2, dtype=torch.float64, device="cuda")

        def steps():
            x, y = a, b
            for k in range(6):
                H.mltply_device_async(y.data_ptr(), x.data_ptr(), vt, coef.data_ptr(), mu[k].data_ptr())
                x, y = y, x

        def reset():
            a.copy_(v)
            b.zero_()
            mu.zero_()
            torch.cuda.synchronize()

        reset()
        steps()
        H.synchronize()
        want = [t.clone() for t in (a, b, mu)]
        reset()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(H.stream)):
            steps()
        for _ in range(2):
            reset()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(x, y) for x, y in zip((a, b, mu), want))
        del graph
