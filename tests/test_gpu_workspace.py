"""No result depends on what a workspace held before the call: bytes of NaN patterns (all 0xFF) in place of zeros, and
another molecule's NaN left in a shared workspace.  The sums are the same ones, so results are equal bit for bit."""
import ctypes

import pytest
import torch

import oracle as O
from graddft_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E(built_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from graddft_gb300 import engine

    return engine


def _workload(n_ao, n_grid, seed=1):
    wl = synthetic.make_workload(n_grid, n_ao, max(1, n_ao // 8), seed=seed, box_angstrom=7.0, centre_box_angstrom=4.0)
    return wl, O.eval_ao_planes(wl.basis, wl.coords)


@pytest.mark.parametrize("precision", ["fp64", "tf32x3"])
@pytest.mark.parametrize("n_ao,n_grid", [(1, 130), (24, 300), (33, 257), (43, 1000), (187, 640), (192, 129)])
def test_contents_do_not_matter(E, precision, n_ao, n_grid):
    from graddft_gb300 import _lib

    L = _lib.load()
    wl, (ao, g1, g2) = _workload(n_ao, n_grid)
    r = E.Resident.from_tables(ao, g1, g2, wl.weights, precision)
    fn = E.make_functional([_lib.COL_LSDA, _lib.COL_B88, _lib.COL_LYP], [1.0])
    lsda = E.make_functional([_lib.COL_LSDA], [1.0])
    d = torch.as_tensor(wl.rdm1, device="cuda")
    nbytes = ctypes.c_size_t()
    _lib.check(L.gdft_workspace_bytes(ctypes.byref(r.desc), ctypes.byref(nbytes)))
    mol, st = ctypes.byref(r.desc), E._stream(r.device)

    def calls(value):
        out = [torch.empty(s, dtype=torch.float64, device="cuda")
               for s in ((n_grid, 2), (n_grid, 2, 3), (n_grid, 2), (n_grid, 2), (n_grid, 2), (), (2, n_ao, n_ao), (),
                         (2, n_ao, n_ao))]
        p = [E._ptr(t) for t in out]

        def ws():  # fresh for each call
            t = torch.full((nbytes.value,), value, dtype=torch.uint8, device="cuda")
            return t, E._ptr(t), t.numel()

        keep = [ws() for _ in range(4)]
        _lib.check(L.gdft_density(mol, E._ptr(d), *p[:4], *keep[0][1:], st))
        _lib.check(L.gdft_density(mol, E._ptr(d), p[4], None, None, None, *keep[1][1:], st))
        _lib.check(L.gdft_xc_energy_and_grads(mol, E._ptr(d), ctypes.byref(fn), None, 0, p[5], p[6], *keep[2][1:], st))
        _lib.check(L.gdft_xc_energy_and_grads(mol, E._ptr(d), ctypes.byref(lsda), None, 0, p[7], p[8], *keep[3][1:],
                                              st))
        torch.cuda.synchronize()
        return out

    for a, b in zip(calls(0), calls(0xFF)):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("net_form", ["fp64", "tf32x3"])
def test_network_contents_do_not_matter(E, net_form):
    from graddft_gb300 import _lib

    L = _lib.load()
    n_ao, n_grid = 43, 700
    wl, (ao, g1, g2) = _workload(n_ao, n_grid)
    r = E.Resident.from_tables(ao, g1, g2, wl.weights, "fp64")
    net = E.Network(n_layers=2, width=128, precision=net_form)
    p = synthetic.glorot_params(layer_widths=(128,) * 2, seed=6)["params"]
    flat = net.flatten({k: {kk: torch.as_tensor(v) for kk, v in q.items()} for k, q in p.items()}, r.device)
    ehf = torch.as_tensor(synthetic.make_ehf(n_grid, 3, None, 2), device="cuda")
    d = torch.as_tensor(wl.rdm1, device="cuda")
    mol, dn, st = ctypes.byref(r.desc), ctypes.byref(net.desc), E._stream(r.device)
    nb, hb = ctypes.c_size_t(), ctypes.c_size_t()
    _lib.check(L.gdft_neural_workspace_bytes(mol, dn, ctypes.byref(nb)))
    _lib.check(L.gdft_neural_hvp_workspace_bytes(mol, dn, ctypes.byref(hb)))

    def calls(value):
        new = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")  # noqa: E731
        a, b, c = (torch.full((x.value,), value, dtype=torch.uint8, device="cuda") for x in (nb, hb, nb))
        out = [new(), new(2, n_ao, n_ao), new(net.n_params), new(), new(2, n_ao, n_ao), new(net.n_params), new(),
               new(2, n_ao, n_ao), new(2, 2, n_grid), new(2, 2, n_grid)]
        q = [E._ptr(t) for t in out]
        _lib.check(L.gdft_neural_xc_energy_and_grads(mol, E._ptr(d), dn, E._ptr(flat), E._ptr(ehf), *q[:3], E._ptr(a),
                                                     a.numel(), st))
        _lib.check(L.gdft_neural_xc_hvp(mol, E._ptr(d), dn, E._ptr(flat), E._ptr(ehf), E._ptr(d), *q[3:6], E._ptr(b),
                                        b.numel(), st))
        _lib.check(L.gdft_neural_xc_hf_grads(mol, E._ptr(d), dn, E._ptr(flat), E._ptr(ehf), *q[6:], E._ptr(c),
                                             c.numel(), st))
        torch.cuda.synchronize()
        return out

    for x, y in zip(calls(0), calls(0xFF)):
        assert torch.isfinite(x).all() and torch.equal(x, y)


def test_another_molecules_nan_stays_its_own(E):
    """Molecules of different sizes one after another in one workspace pool, the first with a NaN density matrix."""
    from graddft_gb300 import _lib

    fn = E.make_functional([_lib.COL_LSDA, _lib.COL_B88, _lib.COL_LYP], [1.0])
    made = []
    for n_ao, n_grid in ((187, 900), (43, 700), (33, 900)):
        wl, _ = _workload(n_ao, n_grid)
        made.append((wl, torch.as_tensor(wl.rdm1, device="cuda")))
    chunked = lambda wl, pool: E.ChunkedResident(wl.basis.packed(), wl.coords, wl.weights, "fp64", 512,  # noqa: E731
                                                 workspace_pool=pool)
    alone = [chunked(wl, {}).xc_energy_and_grads(d, fn) for wl, d in made]
    pool = {}
    e, v = chunked(made[0][0], pool).xc_energy_and_grads(torch.full_like(made[0][1], float("nan")), fn)
    assert not torch.isfinite(v).any()
    for (wl, d), (e0, v0) in list(zip(made, alone))[1:]:
        e, v = chunked(wl, pool).xc_energy_and_grads(d, fn)
        assert torch.equal(e, e0) and torch.equal(v, v0)


@pytest.mark.parametrize("kind", ["resident", "chunked", "network"])
def test_molecules_hold_no_workspace(E, kind):
    """After its calls an FP64 molecule holds its tables (chunked: its grid), not a workspace of its own."""
    from graddft_gb300 import _lib

    fn = E.make_functional([_lib.COL_LSDA, _lib.COL_B88, _lib.COL_LYP], [1.0])
    n_ao, n_grid = 24, 3600
    wl, (ao, g1, g2) = _workload(n_ao, n_grid)
    d = torch.as_tensor(wl.rdm1, device="cuda")
    net = E.Network(n_layers=2, width=64)
    flat = torch.zeros(net.n_params, dtype=torch.float64, device="cuda")
    ehf = torch.as_tensor(synthetic.make_ehf(n_grid, 3, None, 2), device="cuda")
    torch.cuda.synchronize()
    before, made, held = torch.cuda.memory_allocated(), [], 0
    for _ in range(4):
        if kind == "chunked":
            r = E.ChunkedResident(wl.basis.packed(), wl.coords, wl.weights, "fp64", 2048)
            held += r.coords.numel() * 8 + r.weights.numel() * 8 + n_ao * 64
        else:
            r = E.Resident.from_tables(ao, g1, g2, wl.weights)
            held += r.buffer.numel()
            r.density(d)
        r.xc_energy_and_grads(d, fn)
        if kind == "network":
            r.neural_xc_energy_and_grads(d, net, flat, ehf, want_dparams=True)
            r.neural_xc_hvp(d, net, flat, ehf, d)
        assert r.status() == 0
        made.append(r)
    assert torch.cuda.memory_allocated() - before <= held + len(made) * 4096
    assert kind == "chunked" or sum(r.nbytes for r in made) == held


def test_captured_calls_own_their_workspace(E):
    """Calls captured in a CUDA graph, replayed with new density matrices between other molecules' calls."""
    from graddft_gb300 import _lib

    fn = E.make_functional([_lib.COL_LSDA, _lib.COL_B88, _lib.COL_LYP], [1.0])
    made = []
    for n_ao, n_grid in ((43, 700), (130, 900), (24, 300)):
        wl, (ao, g1, g2) = _workload(n_ao, n_grid)
        made.append((E.Resident.from_tables(ao, g1, g2, wl.weights), torch.as_tensor(wl.rdm1, device="cuda")))
    ref = [r.xc_energy_and_grads(d * 0.5, fn) for r, d in made]
    graphs = []
    for r, d in made:
        d = d.clone()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = r.xc_energy_and_grads(d, fn)
        graphs.append((g, d, out))
    for g, d, _ in graphs:
        d.mul_(0.5)
    for i, (g, _, (e, v)) in enumerate(graphs):
        other, d = made[(i + 1) % len(made)]
        other.density(d)
        g.replay()
        other.density(torch.full_like(d, float("nan")))
        assert torch.equal(e, ref[i][0]) and torch.equal(v, ref[i][1])
    assert all(r.status() == 0 for r, _ in made)
