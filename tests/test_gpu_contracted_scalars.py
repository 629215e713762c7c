"""The contracted build's tiled TVD kernels (theta, groups of q fields, saturation adjustment, flow
components) against the separately rounded build on the same state.

Both evaluate the same formulas; the values differ by rounding and by the order of operations.  A
step makes some 10^3 roundings per value of relative size 1.1e-16 (6e-8 in FP32) and mixes them with
weights below 1, so after 3 steps the difference stays below 1e-12 (2e-4) of the field's maximum.
"""
import numpy as np
import pytest

from monc_b200 import api, config as cf, init as ini

pytestmark = pytest.mark.gpu


def config(nx, ny, nz, nq, cloud, precision, flow):
    c = cf.dry_cbl_config(nx, ny, nz, 50.0, 40.0, 0.5, ug=3.0, fcoriol=1e-4, precision=precision)
    c.advection_flow_fields = flow
    if nq:
        c.passive_q, c.number_q_fields, c.simplecloud_enabled = 0, nq, int(cloud)
        c.surface_latent_heat_flux = 100.0
    return c


def state(nx, ny, nz, nq):
    st = ini.random_flow_state(nx, ny, nz, seed=5, amp_uv=1.0, amp_w=0.4, ug=2.0)
    for n in range(nq):
        base = (1.2e-2, 2e-4, 1.0, 0.5, 0.1)[n]
        st[f"q{n}"] = base * (1.0 + 0.5 * ini.uniform_noise((nz, ny, nx), 6, 30 + n, 1.0))
        st[f"zq{n}"] = st[f"q{n}"] * (1.0 + 0.1 * ini.uniform_noise((nz, ny, nx), 6, 40 + n, 1.0))
    return st


def compare(grid, nq, cloud, precision, flow=cf.ADVECT_PW, chunks=0, monkeypatch=None):
    nx, ny, nz = grid
    out = []
    for rep in (1, 0):
        if monkeypatch is not None:
            monkeypatch.setenv("MGPU_LEVEL_CHUNKS", str(chunks))
        c = config(nx, ny, nz, nq, cloud, precision, flow)
        c.reproducible = rep
        m = api.Model(c)
        m.set_state(state(nx, ny, nz, nq))
        m.set_timestep(2)  # centred steps
        m.step(3)
        names = api.STATE_FIELDS + [p + str(n) for n in range(nq) for p in ("q", "zq")]
        out.append({f: m.download(f) for f in names})
        m.close()
    tol = 1e-12 if precision == cf.FP64 else 2e-4
    for f in out[0]:
        scale = np.abs(out[0][f]).max()
        assert np.abs(out[0][f] - out[1][f]).max() <= tol * scale, f


@pytest.mark.parametrize("precision", [cf.FP64, cf.FP32_MIXED], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nq,cloud", [(0, False), (1, False), (2, True), (3, False), (5, True)])
def test_scalar_groups(gpu_lib, nq, cloud, precision):
    compare((64, 16, 20), nq, cloud, precision)


@pytest.mark.parametrize("precision", [cf.FP64, cf.FP32_MIXED], ids=["fp64", "fp32"])
@pytest.mark.parametrize("chunks", [1, 2, 5, 16])
@pytest.mark.parametrize("flow", [cf.ADVECT_PW, cf.ADVECT_TVD], ids=["pw", "tvd"])
def test_level_chunks(gpu_lib, monkeypatch, flow, chunks, precision):
    """Any split of the levels, down to chunks of one level at the top and the bottom."""
    compare((32, 8, 17), 0, False, precision, flow, chunks, monkeypatch)


@pytest.mark.parametrize("precision", [cf.FP64, cf.FP32_MIXED], ids=["fp64", "fp32"])
@pytest.mark.parametrize("grid", [(4, 4, 5), (30, 10, 9), (36, 20, 12), (50, 8, 7), (100, 60, 11)], ids=str)
@pytest.mark.parametrize("nq,flow", [(2, cf.ADVECT_PW), (0, cf.ADVECT_TVD)], ids=["moist", "tvd"])
def test_grids_no_tile_divides(gpu_lib, nq, flow, grid, precision):
    """Tiles reaching past the domain; in FP32 nx = 30, 50 also rows that are not whole 16-byte chunks."""
    compare(grid, nq, nq > 0, precision, flow)


@pytest.mark.parametrize("flow", [cf.ADVECT_PW, cf.ADVECT_TVD], ids=["pw", "tvd"])
def test_smallest_columns(gpu_lib, flow):
    compare((32, 8, 4), 0, False, cf.FP64, flow)
