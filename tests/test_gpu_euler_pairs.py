"""The pair form of PeriPy's CPU integrator on the GPU against its kernels
per Cython function (``Euler(fused=False)``).

Bit-identical on every output array, the whole neighbour list included, for
rows that ascend and rows that do not, equal and differing volumes, breaking
in tension and in compression with force boundaries, neighbours listed
twice, rows wider than a warp and a length beyond the integer route's range.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.cython_setup import breaking_lattice, run_gpu_euler
from tests.gpu_helpers import pull_bcs

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def _lattice(nx, ny, nz, horizon, jitter=0.0):
    from probabilistic_peridynamics_gb300.model import (build_family,
                                                        neighbour_pairs)
    rng = np.random.default_rng(2)
    ii, jj, kk = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz),
                             indexing="ij")
    coords = np.stack([ii.ravel(), jj.ravel(), kk.ravel()], 1).astype(float)
    coords += rng.uniform(-jitter, jitter, coords.shape)
    n = coords.shape[0]
    family, nlist, _ = build_family(n, neighbour_pairs(coords, horizon),
                                    pow2=False)
    bc_types, bc_values = pull_bcs(coords, 0, width=0.1)
    return dict(coords=coords, volume=np.ones(n), family=family, nlist=nlist,
                n_neigh=family.copy(), bc_types=bc_types, bc_values=bc_values,
                force_bc_types=np.zeros((n, 3), dtype=np.intc),
                force_bc_values=np.zeros((n, 3)))


def _setup(form):
    if form == "shuffled":
        return breaking_lattice()
    if form == "twice":
        s = _lattice(7, 6, 4, 2.2)
        n = s["nlist"].shape[0]
        extra = np.zeros((n, 2), dtype=np.intc)
        nl = np.concatenate([s["nlist"], extra], axis=1)
        for i in range(0, n - 1, 2):  # the bond (i, i + 1) once more
            for a, b in ((i, i + 1), (i + 1, i)):
                if b in nl[a, :s["family"][a]]:
                    nl[a, s["n_neigh"][a]] = b
                    s["n_neigh"][a] += 1
        s["nlist"], s["family"] = nl, s["n_neigh"].copy()
        return s
    if form == "wide":
        return _lattice(8, 7, 6, 4.015, jitter=0.05)
    s = _lattice(9, 8, 5, 2.2)
    if form == "scaled":
        s["coords"] = s["coords"] * 2.0 ** 205
    return s


@pytest.mark.parametrize("form", ["ascending", "shuffled", "twice", "wide",
                                  "scaled"])
def test_same_bits(form):
    setup = _setup(form)
    steps = 50
    scale = 2.0 ** 205 if form == "scaled" else 1.0
    mags = 4e-3 * scale * np.arange(1, steps + 1)
    fmags = 0.05 * np.arange(1, steps + 1)
    args = (setup, steps, mags, 0.5, 0.05 * scale, 0.01)
    two = run_gpu_euler(*args, fmags=fmags, fused=False)
    one = run_gpu_euler(*args, fmags=fmags, fused=True)
    for a, b in zip(one, two):
        assert np.array_equal(a, b, equal_nan=True)
    assert int(setup["n_neigh"].sum() - two[4].sum()) > 50  # bonds broke


@pytest.mark.parametrize("form", ["ascending", "shuffled", "one_sided",
                                  "twice", "twice_one_sided", "own", "range"])
def test_symmetry_count(form):
    """Entries whose row does not hold them back as often, against a count on
    the host."""
    import torch
    from probabilistic_peridynamics_gb300._lib import check, lib
    s = _lattice(7, 6, 4, 3.1)
    rng = np.random.default_rng(1)
    nl, n_neigh = s["nlist"].copy(), s["family"].copy()
    n = nl.shape[0]
    nl = np.concatenate([nl, np.zeros((n, 3), nl.dtype)], axis=1)

    def add(i, j):
        nl[i, n_neigh[i]] = j
        n_neigh[i] += 1
    if form == "shuffled":
        for i in range(n):
            rng.shuffle(nl[i, :n_neigh[i]])
    elif form == "one_sided":
        n_neigh[::5] -= 1
    elif form.startswith("twice"):
        for i in range(0, n, 7):
            j = nl[i, 2]
            add(i, j)
            if form == "twice":
                add(j, i)
    elif form == "own":
        for i in range(0, n, 3):
            add(i, i)
    elif form == "range":
        nl[3, 1], nl[8, 0] = n, -2
    rows = [nl[i, :n_neigh[i]].tolist() for i in range(n)]
    want = sum(j < 0 or j >= n or rows[i].count(j) != rows[j].count(i)
               for i in range(n) for j in rows[i])
    dev = [torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda()
           for x in (nl, n_neigh)]
    bad = torch.empty(1, dtype=torch.int32, device="cuda")
    check(lib().pp_cy_check_symmetric(
        dev[0].data_ptr(), dev[1].data_ptr(), n, nl.shape[1], bad.data_ptr(),
        torch.cuda.current_stream().cuda_stream), "pp_cy_check_symmetric")
    assert int(bad.item()) == want
    assert (want == 0) == (form in ("ascending", "shuffled", "twice", "own"))
