"""Models with an active q field but no liquid (one q field, or none with passive_q off): every kernel
form takes the dry Richardson number.  The point, tiled and contracted kernels against each other on
a grid that the tiles divide and one that they do not."""
import numpy as np
import pytest

from monc_b200 import api, config as cf, init as ini

pytestmark = pytest.mark.gpu

GRIDS = [(32, 16, 12), (36, 20, 9)]


def config(grid, nq, reproducible, precision=cf.FP64):
    c = cf.dry_cbl_config(*grid, 50.0, 40.0, 0.5, ug=3.0, fcoriol=1e-4, precision=precision)
    c.passive_q, c.number_q_fields, c.reproducible = 0, nq, reproducible
    return c


def state(grid, nq):
    nx, ny, nz = grid
    st = ini.random_flow_state(nx, ny, nz, seed=5, amp_uv=1.0, amp_w=0.4, ug=2.0)
    for n in range(nq):
        st[f"q{n}"] = 1.2e-2 * (1.0 + 0.5 * ini.uniform_noise((nz, ny, nx), 6, 30 + n, 1.0))
        st[f"zq{n}"] = st[f"q{n}"] * (1.0 + 0.1 * ini.uniform_noise((nz, ny, nx), 6, 40 + n, 1.0))
    return st


@pytest.mark.parametrize("timestep", [1, 2], ids=["forward", "centred"])
@pytest.mark.parametrize("nq", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_subgrid_is_that_of_the_dry_model(gpu_lib, grid, nq, timestep):
    """The component and a step, in the separately rounded form, bit for bit against a model whose q is
    passive (the dry Richardson number by definition); nothing else in the subgrid model reads q."""
    out = []
    for passive in (1, 0):
        c = config(grid, nq, 1)
        c.passive_q = passive
        for fused in (False, True):
            with api.Model(c) as m:
                m.set_state(state(grid, nq))
                m.set_timestep(timestep)
                if fused:
                    m.step(1)
                else:
                    m.component("smagorinsky")
                # (the lowest level is lower_bc's, whose buoyancy flux reads the vapour's)
                out.append({f: m.download(f)[1:] for f in ("vis", "diff")})
    for a, b in ((out[0], out[2]), (out[1], out[3])):
        for f in a:
            np.testing.assert_array_equal(b[f], a[f], err_msg=f)


@pytest.mark.parametrize("precision", [cf.FP64, cf.FP32_MIXED], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nq", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_steps_of_both_builds_agree(gpu_lib, grid, nq, precision):
    """Within the bound of the other comparisons of the two builds (1e-12, FP32 2e-4 after 3 steps)."""
    out = []
    for reproducible in (1, 0):
        with api.Model(config(grid, nq, reproducible, precision)) as m:
            m.set_state(state(grid, nq))
            m.step(4)  # the forward step and three centred ones
            out.append({f: m.download(f) for f in api.STATE_FIELDS + [p + str(n) for n in range(nq) for p in ("q", "zq")]})
    tol = 1e-12 if precision == cf.FP64 else 2e-4
    for f in out[0]:
        assert np.abs(out[0][f] - out[1][f]).max() <= tol * np.abs(out[0][f]).max(), f
