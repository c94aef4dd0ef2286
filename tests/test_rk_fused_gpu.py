"""The fused RK kernels where tiles and chunks end: grids narrower than a tile, tiles that
reach past the domain in x and in y, a single interior plane pair, one chunk and several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("u_crf", [0.0, 0.3])
@pytest.mark.parametrize("nx,ny,nz", [(6, 4, 2), (32, 16, 4), (36, 18, 10), (54, 24, 6), (24, 48, 66), (96, 36, 150)])
def test_fp64_step_matches_oracle(gpu, oracle_mod, nx, ny, nz, u_crf):
    """1e-12 as on the other grids: 50 times what rounding leaves after two steps."""
    plb, O = gpu, oracle_mod
    ch = plb.Channel(plb.ChannelConfig(nx=nx, ny=ny, nz=nz, stretch_ratio=1.5, re_tau=180.0, u_crf=u_crf))
    ch.init_flow(3, 0.1)
    ch.step(2)
    g = O.Grid(nx, ny, nz, stretch=1.5, re_tau=180.0, u_crf=u_crf)
    u, v, w, p = g.init_flow(3, 0.1)
    u1, v1, w1 = g.zeros(), g.zeros(), g.zeros()
    ppe = O.PPE(nx, ny, nz, g.g.dx, g.g.dy, g.dzf_global)
    for _ in range(2):
        g.step(ppe, u, v, w, u1, v1, w1, p)
    got = ch.get_fields()
    errs = [rel(a, b) for a, b in zip(got, (u, v, w))]
    print(f"{nx}x{ny}x{nz} u_crf {u_crf}: max rel err u v w", errs)
    assert max(errs) < 1e-12
    ch.close()


@pytest.mark.parametrize("u_crf", [0.0, 0.3])
@pytest.mark.parametrize("nx,ny,nz", [(6, 4, 2), (32, 16, 4), (36, 18, 10), (54, 24, 6), (24, 48, 66), (96, 36, 150)])
def test_mixed_step_matches_oracle(gpu, oracle_mod, nx, ny, nz, u_crf):
    """Four steps (the last two subtract the pressure prediction's gradient) at 1e-5, the mixed
    path's bar: the first projection of a noisy field leaves up to 2e-6 of max |v|."""
    plb, O = gpu, oracle_mod
    ch = plb.Channel(plb.ChannelConfig(nx=nx, ny=ny, nz=nz, stretch_ratio=1.5, re_tau=180.0, u_crf=u_crf,
                                       precision=plb.PL_MIXED))
    ch.init_flow(3, 0.1)
    ch.step(4)
    g = O.Grid(nx, ny, nz, stretch=1.5, re_tau=180.0, u_crf=u_crf)
    u, v, w, p = g.init_flow(3, 0.1)
    u1, v1, w1 = g.zeros(), g.zeros(), g.zeros()
    ppe = O.PPE(nx, ny, nz, g.g.dx, g.g.dy, g.dzf_global)
    for _ in range(4):
        g.step(ppe, u, v, w, u1, v1, w1, p)
    errs = [rel(a, b) for a, b in zip(ch.get_fields(), (u, v, w))]
    print(f"mixed {nx}x{ny}x{nz} u_crf {u_crf}: max rel err u v w", errs)
    assert max(errs) < 1e-5
    assert ch.diagnostics()["div_max"] < 1e-10
    ch.close()


def _dzf(nz, stretch, lz=2.0):
    zf = 0.5 * (1.0 + np.tanh((np.arange(nz + 1) / nz - 0.5) * stretch) / np.tanh(stretch / 2.0))
    d = lz * np.diff(zf)
    return np.concatenate([d[:1], d, d[-1:]])


@pytest.mark.parametrize("u_crf", [0.0, 0.3])
@pytest.mark.parametrize("nx,ny,nz", [(36, 18, 10), (54, 24, 6), (96, 36, 150), (324, 162, 30)])
def test_mixed_ragged_rk_is_as_exact_as_the_stage_kernels(gpu, nx, ny, nz, u_crf):
    """Grids that the tiles do not divide: the stage-1 field and the update are formed in FP64, as the
    two stage kernels form them.  u_hat against FP64 from one state, with the full pressure ahead (after
    one step) and with a prediction (after three).  The flux form rounds less often than the
    stage kernels' expressions, so the RMS error is smaller than theirs (at most 0.92 of it; with the
    sums in FP32 up to 1.11)."""
    plb = gpu
    kw = dict(nx=nx, ny=ny, nz=nz, stretch_ratio=1.5, re_tau=180.0, u_crf=u_crf, dt=1e-3)
    for steps in (1, 3):
        stage, fused = (plb.Channel(plb.ChannelConfig(precision=plb.PL_MIXED, **kw)) for _ in range(2))
        for ch in (stage, fused):
            ch.init_flow(3, 0.1)
            ch.step(steps - 1)
            before = ch.get_field(3).astype(np.float32)
            ch.step(1)
        u, v, w, p = fused.get_fields()
        ref = plb.Channel(plb.ChannelConfig(**kw))
        ref.set_fields(u, v, w)
        for ch, phases in ((stage, ("rk1", "rk2")), (fused, ("rk",)), (ref, ("rk",))):
            for ph in phases:
                ch.phase(ph)
        exact = [f[1:-1, 1:-1, 1:-1].copy() for f in ref.get_fields()[:3]]
        if steps == 3:  # less dt G (2 p_n - p_{n-1}), the prediction in FP32
            q = np.float32(2.0) * p.astype(np.float32) - before
            q = q.astype(np.float64)
            dzf = _dzf(nz, 1.5)
            dzc = 0.5 * (dzf[:-1] + dzf[1:])
            c = q[1:-1, 1:-1, 1:-1]
            exact[0] -= 1e-3 * (q[1:-1, 1:-1, 2:] - c) * (nx / (2 * np.pi))
            exact[1] -= 1e-3 * (q[1:-1, 2:, 1:-1] - c) * (ny / np.pi)
            exact[2][:-1] -= (1e-3 * (q[2:, 1:-1, 1:-1] - c) / dzc[1:, None, None])[:-1]
        for f in range(3):
            a, b = (ch.get_field(f)[1:-1, 1:-1, 1:-1] for ch in (stage, fused))
            ea, eb = (np.sqrt(((x - exact[f]) ** 2).mean()) for x in (a, b))
            print(f"{nx}x{ny}x{nz} u_crf {u_crf} after {steps}, field {f}: stage {ea:.3e} fused {eb:.3e} ratio {eb / ea:.3f}")
            assert eb <= ea
        for ch in (stage, fused, ref):
            ch.close()
