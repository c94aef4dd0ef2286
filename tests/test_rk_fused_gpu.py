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
