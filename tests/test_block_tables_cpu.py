"""The block kernel's host tables against the terms they come from, on the CPU: every index the kernel
would form stays inside its room, and H*v put together from them is the terms' (host/block_tables_check.cpp).
The models are small, but their lists and graphs are of every kind the plan takes: regular lattices, graphs
whose blocks have many upper-half terms beside few crossing ones, random ones, signs and complex couplings."""
import os
import subprocess

import numpy as np
import pytest

import hphi_b200
from conftest import ROOT
from hphi_b200 import expert


@pytest.fixture(scope="session")
def tables_check(tmp_path_factory):
    lib = hphi_b200.library_path()
    exe = str(tmp_path_factory.mktemp("host") / "block_tables_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "hphi_b200", "csrc"),
                    "-I" + os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "host", "block_tables_check.cpp"),
                    "-o", exe, lib, "-Wl,-rpath," + os.path.dirname(lib), "-L" + os.path.join(cuda, "lib64"), "-lcudart"],
                   check=True)
    return exe


def _uneven_ring():
    """24 sites, one spin up: site 23 is joined to the lower half and to three upper sites, site 22 to
    nine upper ones, so neighbouring blocks have (upper-half, crossing) terms (4, 11) and (11, 0)."""
    b = expert.chain_bonds(24)
    b += [(23, k) for k in range(1, 11)] + [(23, k) for k in (13, 15, 17)] + [(22, k) for k in range(12, 21)]
    return expert.heisenberg(24, b, two_sz=-22)


def _random_graph(n, nbonds, seed, two_sz, values=1):
    rng = np.random.default_rng(seed)
    every = [(i, j) for i in range(n) for j in range(i)]
    pick = rng.choice(len(every), size=nbonds, replace=False)
    return expert.heisenberg(n, [every[k] for k in pick], [1.0 + 0.1 * (k % values) for k in range(nbonds)], two_sz=two_sz)


def _star(n, two_sz):
    return expert.heisenberg(n, [(n - 1, k) for k in range(n - 1)] + [(n - 2, k) for k in range(n // 2, n - 2)], two_sz=two_sz)


def _dm(n):
    m = expert.heisenberg(n, expert.chain_bonds(n))
    m.exchange = []
    for i, j in expert.chain_bonds(n) + expert.chain_bonds(n, 3):
        m.interall += [(i, 0, i, 1, j, 1, j, 0, 0.4, 0.3), (j, 0, j, 1, i, 1, i, 0, 0.4, -0.3)]
    return m


def _nconserved(L, ne):
    m = expert.hubbard(L, expert.chain_bonds(L), 1.0, 3.0, 1, 1)
    m.ncond, m.two_sz = ne, None
    for i in range(L):
        m.trans += [(i, 0, (i + 1) % L, 1, 0.3, 0.1), ((i + 1) % L, 1, i, 0, 0.3, -0.1)]
    return m


MODELS = {
    "uneven_ring": _uneven_ring,
    "star12": lambda: _star(12, 0),
    "star17_few": lambda: _star(17, -11),
    "chain16": lambda: expert.heisenberg(16, expert.chain_bonds(16)),
    "square4x4": lambda: expert.heisenberg(16, expert.square_bonds(4, 4)),
    "dm14": lambda: _dm(14),
    "nconserved6": lambda: _nconserved(6, 5),
    "hubbard6": lambda: expert.hubbard(6, expert.square_bonds(2, 3), 1.0, 4.0, 3, 2),
    "all_to_all15": lambda: _random_graph(15, 105, 0, 1),
}
for _k in range(24):
    _n = 9 + _k % 8
    MODELS[f"random{_k}"] = (lambda n=_n, k=_k: _random_graph(n, 8 + 3 * (k % 11), k, n % 2 if k % 3 else 4 + n % 2 - n,
                                                              values=1 + k % 4))


@pytest.mark.parametrize("name", list(MODELS))
def test_block_tables(name, tables_check, tmp_path):
    r = subprocess.run([tables_check, MODELS[name]().write(str(tmp_path))], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    if not name.startswith("random"):
        assert "shape" in r.stdout  # the plan applies


def test_many_crossing_terms(tables_check, tmp_path):
    """100 bonds between the halves, each acting on every block: too many for whole products, not for the
    row-block plan's row pass."""
    m = expert.heisenberg(20, [(i, j) for i in range(10) for j in range(10, 20)], two_sz=-14)
    r = subprocess.run([tables_check, m.write(str(tmp_path))], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("no plan shape"), r.stdout + r.stderr


def test_crowded_bank(tables_check):
    """More entries on one bank pair than a packed slot count holds: the plan must not lose any."""
    r = subprocess.run([tables_check, "crowded"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("gc", [False, True])
def test_plans_without_device_memory(gc, tables_check, tmp_path):
    """The plans are optional: where the device gives no memory for one, opening the sector goes on."""
    m = expert.kitaev_heisenberg(5, 2, -1.0, 0.3) if gc else expert.heisenberg(12, expert.chain_bonds(12))
    r = subprocess.run([tables_check, m.write(str(tmp_path)), "no_memory"], capture_output=True, text=True,
                       env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
    assert r.returncode == 0, r.stdout + r.stderr
