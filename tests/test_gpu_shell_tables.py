"""The table-driven parts of the shell kernels where their form changes: the radial exponential near the smallest
FP64 numbers and the Boys function at its table's ends."""
import numpy as np
import pytest
import torch
from scipy.special import erf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G(built_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import graddft_gb300 as G

    return G


def _s_shell(G, exps, coefs):
    from graddft_gb300.basis import Shell

    return G.ShellBasis([Shell(np.zeros(3), 0, np.array(exps), np.array([coefs]), np.ones((1, 1)))])


def test_radial_exponential(G):
    """exp(-a r^2) for r^2 from 0 to past the last denormal.  Below exp(-708) the argument is moved by 64 ln 2, an
    error of 2^-44 of a result that is 2^-1021 at most; elsewhere a few roundings."""
    x = np.concatenate([np.linspace(0.0, 26.7, 500), np.sqrt(np.linspace(690.0, 760.0, 700))])
    coords = torch.as_tensor(np.stack([x, 0 * x, 0 * x], 1), device="cuda")
    got = G.eval_ao(_s_shell(G, [1.0], [1.0]), coords, 0)
    got = (got[0] if isinstance(got, (tuple, list)) else got).cpu().numpy()[:, 0]
    ref = np.exp(-x * x)
    assert np.all(np.abs(got - ref) <= 4 * 2.0 ** -53 * ref + 2.0 ** -43 * 2.0 ** -1021 + 5e-324)
    assert np.all(got[x * x > 746.0] == 0.0)


def test_boys_function_ends(G):
    """int phi phi / |r - C| = pi F_0(2 R^2) for phi = exp(-r^2), at T = 2 R^2 on and between the table's points, around
    60 and far beyond.  F_0 is off by some 8 roundings below 60 (the table and its series)."""
    T = np.concatenate([[0.0, 1e-12, 1 / 32 - 1e-9, 1 / 32 + 1e-9, 15.99, 16.0, 16.01, 59.97, 59.999999, 60.0, 60.01, 1e4, 1e12],
                        np.random.default_rng(0).uniform(0, 61, 300)])
    coords = torch.as_tensor(np.stack([np.sqrt(T / 2), 0 * T, 0 * T], 1), device="cuda")
    nu = G.chi.nu_integrals(_s_shell(G, [1.0], [1.0]), coords, 0.0).cpu().numpy().reshape(-1)
    t = np.maximum(T, 1e-300)
    ref = np.pi * np.where(T < 1e-9, 1.0 - T / 3, np.sqrt(np.pi / t) / 2 * erf(np.sqrt(t)))
    assert np.all(np.abs(nu - ref) <= 24 * 2.0 ** -53 * ref), np.max(np.abs(nu - ref) / ref)
