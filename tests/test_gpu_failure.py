"""Failure detection on the GPU without a fault: the library's bounded device waits run against
events that never happen, give up, record the error word and return; the context stays usable."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bounded_waits_time_out_and_report():
    from dac_vtsa_b200 import _lib
    lib = _lib.load()
    bits = C.c_int32(-1)
    rc = lib.dv_selftest_wait_timeout(1000, C.byref(bits))
    assert rc == 0, lib.dv_last_error()
    assert bits.value == 5, bits.value          # 1: the sweep's copy wait, 4: the grid barrier


def test_context_usable_after_timeouts():
    from cases import build, golden
    from dac_vtsa_b200 import _lib
    from dac_vtsa_b200.model import TVSAModel
    lib = _lib.load()
    bits = C.c_int32(0)
    assert lib.dv_selftest_wait_timeout(200, C.byref(bits)) == 0
    d = golden("jacobian_3x4x6.npz")
    m, _ = build(TVSAModel, {"grid.Nr": 3, "grid.Ntheta": 4, "grid.Nz": 6}, 0, d["P0"])
    f, _ = m.rhs(5.0, d["y"], want_acc=False)
    assert np.all(np.isfinite(f))


def test_model_recovers_after_a_reported_timeout():
    """A wait that gave up (injected on the host into the model's error word) is reported once as a
    CUDA-class error naming the wait; the next integration on the same model runs normally."""
    import ctypes as C
    from cases import build, golden
    from dac_vtsa_b200 import _lib
    from dac_vtsa_b200._lib import LibraryError
    from dac_vtsa_b200.model import TVSAModel
    from dac_vtsa_b200.solver import TRBDF2
    d = golden("jacobian_3x4x6.npz")
    m, cfg = build(TVSAModel, {"grid.Nr": 3, "grid.Ntheta": 4, "grid.Nz": 6}, 0, d["P0"], duration=2.0)
    lib = _lib.load()
    assert lib.dv_model_flag_wait_timeout(m.handle, 4) == 0
    with pytest.raises(LibraryError, match="grid barrier"):
        TRBDF2(m, cfg, h_max=0.5).integrate(d["y"], 2.0, [2.0])
    res = TRBDF2(m, cfg, h_max=0.5).integrate(d["y"], 2.0, [2.0])
    assert res.t == pytest.approx(2.0) and np.all(np.isfinite(res.y))


@pytest.mark.parametrize("polls", [1, 1000])
def test_gram_schmidt_exchange_gives_up_and_reports(polls):
    """The exchange every Arnoldi step waits in: with a block that never publishes its sums it gives up after
    `polls` polls and sets the bit that a solve reports; with both blocks it delivers their sums."""
    from dac_vtsa_b200 import _lib
    lib = _lib.load()
    total, bits = C.c_double(-1.0), C.c_int32(-1)
    assert lib.dv_selftest_exchange_timeout(polls, 0, C.byref(total), C.byref(bits)) == 0, lib.dv_last_error()
    assert (bits.value, total.value) == (4, 0.0)
    assert lib.dv_selftest_exchange_timeout(1 << 22, 1, C.byref(total), C.byref(bits)) == 0, lib.dv_last_error()
    assert (bits.value, total.value) == (0, 768.0)


@pytest.mark.parametrize("grid", [(8, 8, 12), (12, 12, 48)])
def test_solve_whose_exchange_gave_up_reports_it_and_the_model_recovers(grid, monkeypatch):
    """A GMRES graph captured with a limit of one poll: the exchange gives up inside a stage solve (other blocks'
    sums take a trip through L2), the solve ends with the wait's error, and the same model, its graph captured
    again with the usual limit, then gives the bits of a model that never failed."""
    import torch
    from dac_vtsa_b200 import autotune, host
    from dac_vtsa_b200._lib import LibraryError
    from dac_vtsa_b200.config import load_config
    from dac_vtsa_b200.jacobian import FDJacobian
    from dac_vtsa_b200.model import TVSAModel
    cfg = load_config(override_dict={"grid.Nr": grid[0], "grid.Ntheta": grid[1], "grid.Nz": grid[2]})
    g = host.Grid.from_config(cfg)
    props = host.get_backend(cfg)
    st = host.seeded_state(cfg, g, props, seed=2)

    def model():
        m = TVSAModel(cfg, g, props, cfg.cycle[0], st)
        y = torch.from_numpy(m.pack(st)).to(m.device)
        m.precond_factor(FDJacobian(m).block(1.0, y), 0.5)
        return m, y

    m, y = model()
    ref = m.newton_stage(1.5, y, y, 0.5)
    m, y = model()
    monkeypatch.setenv("DVTSA_CG_POLLS", "-1")          # gives up after its first poll
    with pytest.raises(LibraryError, match="exchange"):
        m.newton_stage(1.5, y, y, 0.5)
    monkeypatch.delenv("DVTSA_CG_POLLS")
    autotune.apply(m, {"gmres_prefix": 2})              # (the graph is captured again)
    z = m.newton_stage(1.5, y, y, 0.5)
    assert torch.equal(z[0], ref[0]) and z[1] == ref[1] and z[2] == ref[2]
