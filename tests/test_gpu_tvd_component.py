"""tvd_advection as a component, theta and u, v, w by tiles that march up some levels, against the
oracle on grids for each number of levels a march takes (8, 4, 2 and 1: many to few tiles), with ragged
tiles and last marches cut short.  FP64 in the separately rounded form the components have: the
scalars bit for bit, the flow to 1e-12 as in the other comparisons of it."""
import numpy as np
import pytest

from monc_b200 import api, config as cf, init as ini
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

# tiles x marches: 1000 rows are 125 tiles, 250 rows with the flow's four fields 128
SCALAR_GRIDS = [(6, 1000, 162), (6, 1000, 32), (6, 1000, 18), (6, 1000, 7), (36, 10, 5)]
FLOW_GRIDS = [(6, 250, 160), (6, 250, 31), (6, 250, 19), (6, 250, 6), (36, 10, 4)]


def run(grid, flow, timestep, nq=0):
    nx, ny, nz = grid
    c = cf.dry_cbl_config(nx, ny, nz, 50.0, 25.0, 0.5, ug=5.0, fcoriol=1e-4)
    c.advection_flow_fields = flow
    st = ini.random_flow_state(nx, ny, nz, seed=3, ug=3.0)
    sources = ["sth"] + (["su", "sv", "sw"] if flow == cf.ADVECT_TVD else [])
    for n in range(nq):
        st[f"q{n}"] = 1.0 + ini.uniform_noise((nz, ny, nx), 6, 30 + n, 0.5)
        st[f"zq{n}"] = st[f"q{n}"] * (1.0 + 0.1 * ini.uniform_noise((nz, ny, nx), 6, 40 + n, 1.0))
    if nq:
        c.passive_q, c.number_q_fields = 0, nq
        sources += [f"sq{n}" for n in range(nq)]
    for n, name in enumerate(sources):
        st[name] = ini.uniform_noise((nz, ny, nx), 4, 20 + n, 1e-2)
    o, m = po.Oracle(c), api.Model(c)
    for name, arr in st.items():
        o.set(api.field_id(name), arr)
        m.upload(name, arr)
    o.set_timestep(timestep)
    m.set_timestep(timestep)
    o.component(api.COMPONENTS["tvd_advection"])
    m.component("tvd_advection")
    out = {s: (m.download(s), o.get(api.field_id(s))) for s in sources}
    m.close()
    o.close()
    return out


@pytest.mark.parametrize("timestep", [1, 2], ids=["forward", "centred"])
@pytest.mark.parametrize("grid", SCALAR_GRIDS, ids=str)
def test_scalars(gpu_lib, grid, timestep):
    for name, (a, b) in run(grid, cf.ADVECT_PW, timestep, nq=2 if grid[2] < 40 else 0).items():
        np.testing.assert_array_equal(a, b, err_msg=name)


@pytest.mark.parametrize("timestep", [1, 2], ids=["forward", "centred"])
@pytest.mark.parametrize("grid", FLOW_GRIDS, ids=str)
def test_flow_and_scalars(gpu_lib, grid, timestep):
    for name, (a, b) in run(grid, cf.ADVECT_TVD, timestep, nq=1).items():
        if name[1] in "uvw":
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), name
        else:
            np.testing.assert_array_equal(a, b, err_msg=name)
