"""The mixed form's V_xc contraction where its tiles end: the symmetric part (tiles of 128 AOs, mirrored below the
diagonal) and functionals that have none.

Bound, element by element: both operands are represented to 2^-33 of their row's largest value among 32 points, the
products left out and the truncated sums of the corrections are of the same size, a handful in all: 2^-30 of the
product of those values for each point, and what FP32 cannot hold at all (below 10^-38 for each point)."""
import numpy as np
import pytest
import torch

import oracle as O
from graddft_gb300 import synthetic
from test_gpu_fx import E, _tables  # noqa: F401

pytestmark = pytest.mark.gpu


def _chunk_max(x, N):
    return np.abs(np.pad(x, ((0, -N % 32), (0, 0)))).reshape(-1, 32, x.shape[1]).max(1)


@pytest.mark.parametrize("n,N", [(1, 40), (127, 130), (128, 31), (129, 300), (256, 1001), (257, 640), (390, 513)])
def test_vxc(E, n, N):  # noqa: F811
    ao, g1, g2, _, pot = _tables(n, N, 10 * n + N)
    r = E.Resident.from_tables(ao, g1, g2, np.ones(N), "tf32x3", "cuda:0")
    got = r.vxc_from_potentials(pot).cpu().numpy()
    assert r.status() == 0
    for s in range(2):
        c = pot[s][..., None]
        Q = c[0] * ao + sum(c[1 + j] * g1[..., j] for j in range(3)) + c[4] * g2.sum(-1)
        aQ = np.abs(c[0] * ao) + sum(np.abs(c[1 + j] * g1[..., j]) for j in range(3)) + np.abs(c[4] * g2.sum(-1))
        ref, bound = ao.T @ Q, 32 * _chunk_max(ao, N).T @ _chunk_max(aQ, N)
        for j in range(3):
            x = g1[..., j]
            ref += x.T @ (c[5] * x)
            bound += 32 * _chunk_max(x, N).T @ _chunk_max(c[5] * x, N)
        bound = 2.0 ** -30 * np.maximum(bound, bound.T) + N * 1e-36
        assert np.all(np.abs(got[s] - ref) <= bound), np.max(np.abs(got[s] - ref) / bound)


@pytest.mark.parametrize("n_ao,n_grid", [(20, 200), (140, 700)])
def test_no_kinetic_part(E, n_ao, n_grid):  # noqa: F811
    """LSDA (only the phi plane is contracted) against the oracle, at the tolerance of the mixed form's other tests."""
    from graddft_gb300 import _lib
    from test_gpu_mixed import TOL_E, TOL_V, _rel

    wl = synthetic.make_workload(n_grid, n_ao, max(1, n_ao // 8), seed=3, box_angstrom=8.0, centre_box_angstrom=5.0)
    ao, g1, g2 = O.eval_ao_planes(wl.basis, wl.coords)
    r = E.Resident.from_tables(ao, g1, g2, wl.weights, "tf32x3")
    exc, vxc = r.xc_energy_and_grads(wl.rdm1, E.make_functional([_lib.COL_LSDA], [1.0]))
    e_ref, v_ref = O.xc_energy_and_grads("LSDA", wl.rdm1, ao, g1, g2, wl.weights)
    assert r.status() == 0 and abs(float(exc) - e_ref) <= TOL_E * abs(e_ref) and _rel(vxc, v_ref) <= TOL_V
