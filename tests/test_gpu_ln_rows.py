"""LayerNorm + ELU passes of the FP64 network against the oracle, where their exponential changes its form."""
import numpy as np
import pytest
import torch

import oracle as O
from graddft_gb300 import synthetic
from test_gpu_scf import _case, _molecule, _rel, _t, G  # noqa: F401

pytestmark = pytest.mark.gpu

# LayerNorm biases: positive and negative arguments of the ELU, near zero, past
# the table's range (-700) and where exp is denormal or zero.
BIASES = np.array([0.0, 1e-3, -1e-3, 0.5, -0.7, -3.0, -40.0, -697.0, -703.0, -720.0, -800.0, 3.0])


@pytest.mark.parametrize("width,n_grid", [(32, 131), (64, 258), (128, 515), (256, 1030)])
def test_first_and_second_order(G, width, n_grid):  # noqa: F811
    """E, V_xc, dE/dtheta and the second-order pass.  Values are sums of some 10^5 terms rounded at 2^-53, with the
    layers' scales of order one to ten: 1e-10 of each array's largest value."""
    wl, ao, g1, g2, ehf = _case(n_grid=n_grid, n_ao=13, n_occ=3, seed=width)
    params = synthetic.glorot_params(layer_widths=(width,) * 3, seed=width)
    g = np.random.default_rng(width)
    for i in range(3):
        params["params"][f"LayerNorm_{i}"]["bias"] = g.choice(BIASES, width)
    tangent = g.standard_normal(wl.rdm1.shape)
    hf = lambda atoms, *_, **__: atoms.ehf  # noqa: E731
    f = G.DM21(layer_widths=(width,) * 3, densitygrads=None, coefficient_input_grads=None, nograd_densities=hf,
               nograd_coefficient_inputs=hf)
    net, mol = f.network(), _molecule(G, ao, g1, g2, wl.weights, wl.rdm1, ehf)
    r = mol.resident()
    tp = {"params": {k: {kk: torch.as_tensor(v) for kk, v in d.items()} for k, d in params["params"].items()}}
    flat = net.flatten(tp, r.device)
    e_ref, v_ref, dp_ref = O.xc_energy_and_grads("DM21", wl.rdm1, ao, g1, g2, wl.weights, params=params, ehf=ehf,
                                                 want_param_grads=True)
    L_ref, hD_ref, hp_ref = O.xc_hvp("DM21", wl.rdm1, ao, g1, g2, wl.weights, tangent, params=params, ehf=ehf)
    e, v, dp = r.neural_xc_energy_and_grads(mol._rdm1(), net, flat, mol.ehf, want_dparams=True)
    L, hD, hp = r.neural_xc_hvp(mol._rdm1(), net, flat, mol.ehf, _t(tangent), want_value=True)
    assert r.status() == 0
    assert abs(float(e) - e_ref) <= 1e-10 * abs(e_ref) and abs(float(L) - L_ref) <= 1e-10 * abs(L_ref)
    assert _rel(v, v_ref) <= 1e-10 and _rel(hD, hD_ref) <= 1e-10
    for got, ref in ((net.unflatten(dp), dp_ref), (net.unflatten(hp), hp_ref)):
        for mod, d in ref["params"].items():
            for leaf, x in d.items():
                assert _rel(got["params"][mod][leaf], x) <= 1e-10, (mod, leaf)


def test_non_finite_row(G):  # noqa: F811
    """A NaN and an infinite input leave their own rows not finite and the others as they were (the GEMMs
    then take their plain form, which rounds differently: 1e-13 as in the network's other tests)."""
    f = G.DM21(layer_widths=(64,) * 3)
    p = synthetic.glorot_params(layer_widths=(64,) * 3, seed=4)
    x = torch.as_tensor(np.random.default_rng(4).standard_normal((37, 11)), device="cuda")
    clean = f.apply(p, x)
    x[5, 2], x[18, 0] = float("nan"), float("inf")
    got = f.apply(p, x)
    assert not torch.isfinite(got[5]).any()
    keep = [i for i in range(37) if i not in (5, 18)]
    assert torch.max(torch.abs(got[keep] - clean[keep])) <= 1e-13
