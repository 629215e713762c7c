"""Component kernels on grids no thread block divides, FP64, bit for bit against the CPU oracle."""
import numpy as np
import pytest

from monc_b200 import api, config as cf, init as ini
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

OUTPUTS = {"diverr": ["p"], "pstep": ["u", "zu", "v", "zv", "zw"],
           "swap_smooth": ["u", "v", "w", "th", "zu", "zv", "zw", "zth"], "tvd_advection": ["sth"]}


@pytest.mark.parametrize("timestep", [1, 2], ids=["forward", "centred"])
@pytest.mark.parametrize("grid", [(30, 12, 4), (36, 20, 9), (64, 10, 5), (32, 8, 18)], ids=str)
@pytest.mark.parametrize("comp", sorted(OUTPUTS))
def test_component_on_ragged_grid(gpu_lib, comp, grid, timestep):
    nx, ny, nz = grid
    c = cf.dry_cbl_config(nx, ny, nz, 50.0, 25.0, 0.5, ug=5.0, fcoriol=1e-4)
    o, m = po.Oracle(c), api.Model(c)
    st = ini.random_flow_state(nx, ny, nz, seed=3, ug=3.0)
    for n, name in enumerate(["p", "savu", "savv", "savw", "sth"]):
        st[name] = ini.uniform_noise((nz, ny, nx), 4, 20 + n, 1e-2)
    for name, arr in st.items():
        o.set(api.FIELDS[name], arr)
        m.upload(name, arr)
    o.set_timestep(timestep)
    m.set_timestep(timestep)
    o.component(api.COMPONENTS[comp])
    m.component(comp)
    for f in OUTPUTS[comp]:
        np.testing.assert_array_equal(m.download(f), o.get(api.FIELDS[f]), err_msg=f)
    if comp == "diverr":
        assert m.reductions().global_divmax == np.abs(m.download("p")).max()
    m.close()
    o.close()
