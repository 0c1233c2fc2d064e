"""GPU coloured FD Jacobian (all colours in one launch) vs the reference's FDJacobian values."""
import numpy as np
import pytest

from cases import build, golden

pytestmark = pytest.mark.gpu


def test_fd_jacobian_matches_reference():
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    d = golden("jacobian_3x4x6.npz")
    m, _ = build(TVSAModel, {"grid.Nr": 3, "grid.Ntheta": 4, "grid.Nz": 6}, 0, d["P0"])
    jac = FDJacobian(m)
    J = jac(float(d["t"]), d["y"])
    assert np.array_equal(J.indptr, d["indptr"]) and np.array_equal(J.indices, d["indices"])
    ref = d["data"]
    # compare column by column relative to the column's largest entry: the forward difference
    # amplifies ulp-level residual differences by 1/h (h = 1.5e-8 max(|y|, typ)).
    col = np.repeat(np.arange(J.shape[1]), np.diff(J.indptr))
    colmax = np.zeros(J.shape[1])
    np.maximum.at(colmax, col, np.abs(ref))
    err = np.abs(J.data - ref) / np.maximum(colmax[col], 1e-300)
    assert err.max() <= 1e-6, err.max()


def test_jacobian_matches_dense_fd_and_colouring_is_valid():
    """Reference test (tests/test_physics_and_numerics.py:118-138) on the GPU: 12 random columns of the
    coloured Jacobian vs one-column-at-a-time differences of the GPU residual, 1e-3 relative."""
    from dac_vtsa_b200 import host
    from dac_vtsa_b200.config import load_config
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    cfg = load_config(override_dict={"grid.Nr": 3, "grid.Ntheta": 4, "grid.Nz": 6})
    g = host.Grid.from_config(cfg)
    props = host.get_backend(cfg)
    st = host.initial_state(cfg, g, props)
    st.T = st.T + np.random.default_rng(0).random(st.T.shape)
    m = TVSAModel(cfg, g, props, cfg.cycle[0], st)
    y = m.pack(st)
    jac = FDJacobian(m)
    J = jac(5.0, y).toarray()
    f0, _ = m.rhs(5.0, y, want_acc=False)
    for j in np.random.default_rng(2).choice(len(y), 12, replace=False):
        h = 1e-7 * max(abs(y[j]), 1e-3)
        yp = y.copy()
        yp[j] += h
        col_fd = (m.rhs(5.0, yp, want_acc=False)[0] - f0) / h
        scale = max(np.abs(col_fd).max(), 1e-12)
        assert np.abs(col_fd - J[:, j]).max() / scale < 1e-3
    Pr = jac.P.tocsr()
    for r in range(Pr.shape[0]):
        cc = jac.color[Pr.indices[Pr.indptr[r]:Pr.indptr[r + 1]]]
        assert len(np.unique(cc)) == len(cc)


@pytest.mark.parametrize("grid", [(1, 1, 1), (1, 1, 9), (1, 4, 2), (2, 3, 3), (3, 5, 5), (4, 1, 34)])
@pytest.mark.parametrize("step", [0, 2])
def test_jacobian_entries_are_the_quotients_of_the_residual(grid, step):
    """Every entry equals the difference quotient of the whole residual with that one column perturbed,
    to the bit (the same expressions on the same operands): columns, rings and sectors at the edges of
    the grid, beds shorter than a slope's stencil, tiles with a remainder, feed / vent and vacuum ends."""
    import torch
    from dac_vtsa_b200 import host
    from dac_vtsa_b200.config import load_config
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    cfg = load_config(override_dict={"grid.Nr": grid[0], "grid.Ntheta": grid[1], "grid.Nz": grid[2],
                                     "wall.enabled": grid != (4, 1, 34)})
    g = host.Grid.from_config(cfg)
    props = host.get_backend(cfg)
    st = host.seeded_state(cfg, g, props, seed=5, amplitude=0.02, P=101325.0 if step == 0 else 2.2e4)
    st.q = st.q + np.random.default_rng(6).random(st.q.shape)
    m = TVSAModel(cfg, g, props, cfg.cycle[step], st)
    y = torch.from_numpy(m.pack(st)).to(m.device)
    J = FDJacobian(m)(3.0, y).toarray()
    f0, _ = m.rhs(3.0, y, want_acc=False)
    typ = np.concatenate([np.full(g.ncell, a) for a in m.params.typ[:6]] + [np.full(m.n_w, m.params.typ[6])])
    ref = np.zeros_like(J)
    for col in range(m.n_core):
        yv = float(y[col])
        h = (yv + 1.5e-8 * max(abs(yv), typ[col])) - yv
        yp = y.clone()
        yp[col] = yv + h
        # (divided by numpy: torch multiplies a CUDA tensor by a scalar's rounded reciprocal)
        ref[:, col] = (m.rhs(3.0, yp, want_acc=False)[0] - f0).cpu().numpy() / h
    assert np.array_equal(J, ref)


@pytest.mark.parametrize("grid", [(1, 1, 9), (3, 5, 7), (8, 8, 12)])
def test_jacobian_without_scratch_and_in_a_captured_graph(grid, monkeypatch):
    """A model without the Jacobian's scratch, and a captured call, give the same bits; replays of the captured
    call run beside direct calls at another state on another stream (no order between them, no shared scratch)."""
    import ctypes as C
    import torch
    from dac_vtsa_b200 import host
    from dac_vtsa_b200.config import load_config
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    cfg = load_config(override_dict={"grid.Nr": grid[0], "grid.Ntheta": grid[1], "grid.Nz": grid[2]})
    g = host.Grid.from_config(cfg)
    props = host.get_backend(cfg)
    st = host.seeded_state(cfg, g, props, seed=5, amplitude=0.02)
    m = TVSAModel(cfg, g, props, cfg.cycle[0], st)
    y1 = torch.from_numpy(m.pack(st)).to(m.device)
    y2 = y1 * 1.001
    f1, f2 = m.rhs(3.0, y1, want_acc=False)[0], m.rhs(3.0, y2, want_acc=False)[0]
    J1, J2 = FDJacobian(m).block(3.0, y1, f1), FDJacobian(m).block(3.0, y2, f2)
    monkeypatch.setenv("DVTSA_JAC_SCRATCH", "0")
    bare = TVSAModel(cfg, g, props, cfg.cycle[0], st)
    assert torch.equal(FDJacobian(bare).block(3.0, y1, f1), J1)

    def call(y, f, J, stream):
        assert m.lib.dv_fd_jacobian(m.handle, 3.0, y.data_ptr(), f.data_ptr(), J.data_ptr(),
                                    C.c_void_p(stream.cuda_stream)) == 0, m.lib.dv_last_error()

    out1 = torch.full_like(J1, np.nan)
    out2 = [torch.full_like(J2, np.nan) for _ in range(20)]
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        call(y1, f1, out1, torch.cuda.current_stream())
    for o in out2:
        graph.replay()
        call(y2, f2, o, side)
    torch.cuda.synchronize()
    assert torch.equal(out1, J1)
    assert all(torch.equal(o, J2) for o in out2)
