"""The contracted build's tiled kernels with the options its default steps leave out -- stretched
levels, damping, subsidence, the Galilean frame, mean baroclinicity, no viscosity, a passive theta,
another reference density -- against the separately rounded build on the same state, which the
oracle tests hold to MONC.

The bound is the one of the other comparisons of the two builds: some 10^3 roundings per value and step
of relative size 1.1e-16 (6e-8 in FP32), mixed with weights below 1, stay below 1e-12 (2e-4) of the field's
maximum after 3 steps.
"""
import numpy as np
import pytest

from monc_b200 import api, config as cf, init as ini

pytestmark = pytest.mark.gpu

GRID = (36, 20, 12)  # a tile and a ragged one in each direction


def levels(c):
    cf.set_explicit_levels(c, cf.stretched_levels(c.nz, 20.0, 60.0, ztop=440.0))


def subsidence(local):
    return lambda c: cf.enable_subsidence(c, [0.0, 150.0, 300.0, 440.0], [0.0, -0.02, -0.03, -0.01], theta=True,
                                          q=c.number_q_fields > 0, local_theta=local, local_q=local)


def damping(c):
    cf.enable_damping(c, 0.02, 100.0, 150.0)


def galilean(c):
    cf.enable_galilean(c, 2.5, -1.5)


def flags(**kw):
    def f(c):
        for k, v in kw.items():
            setattr(c, k, v)
    return f


OPTIONS = {
    "stretched": [levels],
    "damping": [levels, damping],
    "subsidence-mean": [levels, subsidence(False)],
    "subsidence-local": [levels, subsidence(True)],
    "all-forcing-galilean": [levels, damping, subsidence(False), galilean],
    "local-forcing-galilean": [damping, subsidence(True), galilean],
    "inviscid": [flags(use_viscosity_and_diffusion=0)],
    "inviscid-forced": [levels, flags(use_viscosity_and_diffusion=0), damping, subsidence(True), galilean],
    "density": [levels, flags(rhobous=1.17)],
    "passive-theta": [flags(passive_th=1), damping],
    "at-rest": [flags(coriolis_enabled=0, use_surface_boundary_conditions=0)],
    "baroclinic": [levels, lambda c: cf.enable_baroclinicity(c, 2e-3, -1e-3), galilean],
}


def final_fields(options, nq, flow, precision, reproducible, grid=GRID):
    nx, ny, nz = grid
    c = cf.dry_cbl_config(nx, ny, nz, 50.0, 40.0, 0.5, ug=3.0, fcoriol=1e-4, precision=precision)
    c.advection_flow_fields = flow
    if nq:
        c.passive_q, c.number_q_fields, c.simplecloud_enabled = 0, nq, 1
        c.surface_latent_heat_flux = 100.0
    for f in OPTIONS[options]:
        f(c)
    c.reproducible = reproducible
    st = ini.random_flow_state(nx, ny, nz, seed=5, amp_uv=1.0, amp_w=0.4, ug=2.0)
    zn = api.reference_profile(c, "zn")
    for f in ("th", "zth"):
        st[f] = st[f] + 0.004 * zn[:, None, None]
    for n in range(nq):
        base = (1.2e-2, 2e-4, 1.0)[n]
        st[f"q{n}"] = base * (1.0 + 0.5 * ini.uniform_noise((nz, ny, nx), 6, 30 + n, 1.0))
        st[f"zq{n}"] = st[f"q{n}"] * (1.0 + 0.1 * ini.uniform_noise((nz, ny, nx), 6, 40 + n, 1.0))
    with api.Model(c) as m:
        m.set_state(st)
        m.set_timestep(3)  # centred, with damping and forcing acting
        m.step(3)
        return {f: m.download(f) for f in api.STATE_FIELDS + [p + str(n) for n in range(nq) for p in ("q", "zq")]}


def compare(options, nq, flow, precision, grid=GRID):
    ref = final_fields(options, nq, flow, precision, 1, grid)
    got = final_fields(options, nq, flow, precision, 0, grid)
    tol = 1e-12 if precision == cf.FP64 else 2e-4
    for f in ref:
        assert np.abs(ref[f] - got[f]).max() <= tol * np.abs(ref[f]).max(), f


@pytest.mark.parametrize("options", sorted(OPTIONS))
@pytest.mark.parametrize("nq,flow", [(0, cf.ADVECT_PW), (3, cf.ADVECT_PW), (2, cf.ADVECT_TVD)],
                         ids=["dry", "moist-tracer", "moist-tvd"])
def test_options(gpu_lib, nq, flow, options):
    compare(options, nq, flow, cf.FP64)


@pytest.mark.parametrize("options", ["all-forcing-galilean", "inviscid-forced"])
@pytest.mark.parametrize("nq,flow", [(0, cf.ADVECT_TVD), (3, cf.ADVECT_PW)], ids=["dry-tvd", "moist-tracer"])
def test_options_fp32(gpu_lib, nq, flow, options):
    compare(options, nq, flow, cf.FP32_MIXED)


@pytest.mark.parametrize("chunks", [1, 11])
@pytest.mark.parametrize("options", ["all-forcing-galilean", "inviscid-forced", "stretched"])
def test_options_in_level_chunks(gpu_lib, monkeypatch, options, chunks):
    """The whole column in one chunk, and chunks of one level."""
    monkeypatch.setenv("MGPU_LEVEL_CHUNKS", str(chunks))
    compare(options, 2, cf.ADVECT_TVD, cf.FP64)


# on both sides of the line below which a thread takes a point: 16 blocks of 32 x 8 points, 64 with TVD flow
@pytest.mark.parametrize("flow,grid", [(cf.ADVECT_PW, (32, 8, 16)), (cf.ADVECT_PW, (32, 8, 17)),
                                       (cf.ADVECT_PW, (36, 10, 4)), (cf.ADVECT_PW, (36, 10, 5)),
                                       (cf.ADVECT_TVD, (4, 4, 64)), (cf.ADVECT_TVD, (4, 4, 65)),
                                       (cf.ADVECT_TVD, (36, 10, 16)), (cf.ADVECT_TVD, (36, 10, 17))], ids=str)
@pytest.mark.parametrize("nq", [0, 2])
def test_grids_of_few_points(gpu_lib, nq, flow, grid):
    compare("inviscid", nq, flow, cf.FP64, grid)


@pytest.mark.parametrize("nq,flow", [(0, cf.ADVECT_PW), (2, cf.ADVECT_TVD)], ids=["dry", "moist-tvd"])
def test_shortest_columns_on_tiles(gpu_lib, monkeypatch, nq, flow):
    """Four levels on the tiles, which a fixed number of level chunks asks for."""
    monkeypatch.setenv("MGPU_LEVEL_CHUNKS", "1")
    compare("at-rest", nq, flow, cf.FP64, (36, 10, 4))
