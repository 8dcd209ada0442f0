"""The stage kernels' dispatch at the sizes where it changes or can go wrong, against the CPU
oracle: the row-tile kernel of small meshes (edges of tiles, one-cell sides), the strip heights
of the size rule with either form of the reduction, states whose values leave the range of the
short arithmetic, stored stage derivatives beside every per-cell field, and batches of more
members than one launch takes. FP64 is compared bit for bit. FP32 has no rounding of its own per
kernel, so its kernels are compared with one another bit for bit."""
import numpy as np
import pytest

from mfcm_b200 import (SaintVenantSolver, SvError, synth, RK_METHODS, EDGE_XMAX, EDGE_XMIN, EDGE_YMIN, EDGE_YMAX, RAIN_FIELDS,
                       HEAD_FIELDS)
from mfcm_b200.batch import SaintVenantBatch
from oracle.sv_oracle_py import OracleSolver
from tests.scenarios import wet_dry_state, setup, forcing, same, first_diff

pytestmark = pytest.mark.gpu


def assert_same(g, o, what):
    d = first_diff(g, o)
    assert d is None, f"{what}: first mismatch at {d[0]}: {d[1]!r} against {d[2]!r} ({d[3]} cells differ)"


def one_timestep(b, t=0.5, dt=0.02):
    """(control number, ...) and U_[N] of one timestep"""
    r = b.do_timestep(t, dt)
    return r, [b.get_field(100 + 3 * b.nstages + f) for f in range(3)]


@pytest.mark.parametrize("dx", [2.0, 3.0])
@pytest.mark.parametrize("shape", [(1, 1), (1, 30), (30, 1), (28, 8), (29, 9), (27, 7), (57, 17), (84, 25)])
@pytest.mark.parametrize("nan_cells", [0, 3])
def test_row_tiles(shape, dx, nan_cells):
    nx, ny = shape
    if nan_cells and nx * ny < 100:
        pytest.skip("too small for coded-out cells")
    z, h, u, v = wet_dry_state(nx, ny, dx, seed=nx + 7 * ny, nan_cells=nan_cells)
    out = []
    for cls in (SaintVenantSolver, OracleSolver):
        b = cls(nx, ny, dx, rain_mode="physical")
        setup(b, z, h, u, v, n=(0.03, 0.06, 0.1, 0.3))
        b.set_forcing(forcing((2e-5, 1e-5), head=(0.01, 0.0), edges=EDGE_XMIN | EDGE_YMAX))
        out.append(one_timestep(b))
    for f in range(3):
        assert_same(out[0][1][f], out[1][1][f], f"U_[N] field {f}")
    if not nan_cells:
        assert out[0][0] == out[1][0]


# heights of the size rule in FP64: 4 just above the row tiles' sizes, then 9, 9 and 18; all strips
# resident at once (one form of the sweep) and several waves of them (two forms); up to 2048 strips
# reduced by one block, more by a cluster
@pytest.mark.parametrize("shape", [(300, 280), (800, 701), (1100, 1001), (1500, 1450)])
def test_strip_heights_of_the_size_rule(shape):
    nx, ny = shape
    z, h, u, v = wet_dry_state(nx, ny, 2.0, seed=nx)
    out = []
    for cls in (SaintVenantSolver, OracleSolver):
        b = cls(nx, ny, 2.0, cn_target=0.5, step_duration=0.02, initial_dt=0.02, rain_mode="physical")
        setup(b, z, h, u, v)
        b.set_forcing(forcing((2e-5, 1e-5), head=(0.01, 0.0), edges=EDGE_XMAX | EDGE_YMIN))
        b.advance()
        out.append(([b.get_field(f) for f in ("H", "U", "V")], b.stats(), b.get_dt()))
    (gf, gs, gdt), (of, os_, odt) = out
    for f in range(3):
        assert_same(gf[f], of[f], f"field {f}")
    assert gdt == odt and gs["accepted"] == os_["accepted"] and gs["repeated"] == os_["repeated"]
    # FP64 sums over the cells in another order: n eps of the terms' magnitude (the signed tallies'
    # terms are thousandths of the volume)
    for k in ("volume", "rain_in", "outflow", "wall_in"):
        assert abs(gs[k] - os_[k]) <= nx * ny * 2.3e-16 * max(abs(os_[k]), 1e-3 * os_["volume"]), k


@pytest.mark.parametrize("variant", [5, 8])
@pytest.mark.parametrize("field", ["H", "U", "V"])
def test_values_out_of_the_short_arithmetics_range(variant, field):
    """Values below 2^-200 and above 2^200, infinities and NaN, in rows near a strip's start, in
    its middle and in its last rows: from the first such row on the general form runs."""
    nx, ny = 90, 70
    z, h, u, v = wet_dry_state(nx, ny, 2.0, seed=5)
    a = {"H": h, "U": u, "V": v}[field]
    for y, x, val in ((3, 40, 1e-80), (17, 10, 1e-310), (29, 44, 1e70), (33, 70, np.inf), (50, 20, np.nan), (69, 89, 1e-100)):
        a[y, x] = val
    out = []
    for cls in (SaintVenantSolver, OracleSolver):
        b = cls(nx, ny, 2.0, rain_mode="physical")
        if cls is SaintVenantSolver:
            b.set_kernel_variant(variant)
        setup(b, z, h, u, v)
        b.set_forcing(forcing((2e-5, 1e-5), head=(0.01, 0.0), edges=EDGE_XMIN))
        out.append(one_timestep(b)[1])
    for f in range(3):
        assert_same(out[0][f], out[1][f], f"U_[N] field {f}")


@pytest.mark.parametrize("rk", RK_METHODS)
@pytest.mark.parametrize("dx", [2.0, 3.0])
def test_stored_stages_beside_every_field(rk, dx):
    nx, ny = 87, 45
    z, h, u, v = wet_dry_state(nx, ny, dx, seed=9)
    rng = np.random.default_rng(4)
    shape = (ny, nx)
    fields = {"N_SHALLOW": rng.uniform(0.02, 0.05, shape), "N_DEEP": rng.uniform(0.05, 0.1, shape),
              "D_SHALLOW": rng.uniform(0.05, 0.1, shape), "D_DEEP": rng.uniform(0.2, 0.4, shape),
              "QBDY0": rng.uniform(0, 3e-5, shape), "QBDY1": rng.uniform(0, 3e-5, shape),
              "INFIL_RATE": rng.uniform(0, 2e-5, shape), "INFIL_CAP": rng.uniform(0, 2e-4, shape),
              "ELOSS_FX": rng.uniform(0, 0.5, shape), "ELOSS_FY": rng.uniform(0, 0.5, shape),
              "EDDY_MU": rng.uniform(0, 2.0, shape)}
    h0 = np.where(rng.uniform(size=shape) < 0.05, 0.02, np.nan)
    fields["HBDY0"], fields["HBDY1"] = h0, h0 * 2.0
    out = []
    for cls in (SaintVenantSolver, OracleSolver):
        b = cls(nx, ny, dx, rk_method=rk, rain_mode="physical")
        setup(b, z, h, u, v)
        for name, a in fields.items():
            b.set_field(name, a)
        b.set_eddy_viscosity("constant")
        f = forcing((0.0, 0.0), rain_kind=RAIN_FIELDS)
        f.head_kind = HEAD_FIELDS
        b.set_forcing(f)
        for name in ("QBDY0", "QBDY1"):  # the oracle's set_forcing clears the rain fields
            b.set_field(name, fields[name])
        r, un = one_timestep(b)
        out.append((r, un + [b.get_field("INFIL_CAP")]))
    assert out[0][0] == out[1][0]
    for f in range(4):
        assert_same(out[0][1][f], out[1][1][f], f"field {f}")


@pytest.mark.parametrize("precision", ["f32", "f32_datum64"])
@pytest.mark.parametrize("dx", [2.0, 3.0])
@pytest.mark.parametrize("shape", [(29, 9), (231, 170)])
def test_fp32_kernels_round_alike(precision, dx, shape):
    """The row tiles (variant 5 at these sizes) and the sweeps of every strip height give the
    same bits."""
    nx, ny = shape
    z, h, u, v = wet_dry_state(nx, ny, dx, seed=3)
    out = []
    for variant in (5, 4, 6, 8):
        b = SaintVenantSolver(nx, ny, dx, precision=precision, rain_mode="physical")
        b.set_kernel_variant(variant)
        setup(b, z, h, u, v, n=(0.03, 0.06, 0.1, 0.3))
        b.set_forcing(forcing((2e-5, 1e-5), head=(0.01, 0.0), edges=EDGE_XMIN | EDGE_YMAX))
        out.append(one_timestep(b)[1])
    for o in out[1:]:
        for f in range(3):
            assert_same(o[f], out[0][f], f"U_[N] field {f}")


@pytest.mark.parametrize("dx", [2.0, 3.0])
@pytest.mark.parametrize("shape", [(29, 9), (1500, 1100), (2100, 1800)])
def test_fp32_sweeps_with_every_term_round_alike(dx, shape):
    """Variant 5's height (all strips resident, then more than one wave: edge form only, then two
    forms) against strips of 32 rows and of 64, which stay resident."""
    nx, ny = shape
    z, h, u, v = wet_dry_state(nx, ny, dx, seed=3)
    rng = np.random.default_rng(2)
    extra = {"ELOSS_FX": rng.uniform(0, 0.5, (ny, nx)), "ELOSS_FY": rng.uniform(0, 0.5, (ny, nx)),
             "INFIL_RATE": rng.uniform(0, 2e-5, (ny, nx)), "INFIL_CAP": rng.uniform(0, 2e-4, (ny, nx))}
    out = []
    for variant in (5, 8, 6):
        b = SaintVenantSolver(nx, ny, dx, precision="f32", rain_mode="physical")
        b.set_kernel_variant(variant)
        setup(b, z, h, u, v, n=(0.03, 0.06, 0.1, 0.3))
        for name, a in extra.items():
            b.set_field(name, a)
        b.set_eddy_viscosity("smagorinsky")
        b.set_forcing(forcing((2e-5, 1e-5), head=(0.01, 0.0), edges=EDGE_XMIN | EDGE_YMAX))
        out.append(one_timestep(b)[1] + [b.get_field("INFIL_CAP")])
        b.close()
    for o in out[1:]:
        for f in range(4):
            assert_same(o[f], out[0][f], f"field {f}")


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("precision", ["f64", "f32", "f32_datum64"])
@pytest.mark.parametrize("count", [3, 35])
def test_batches_of_mixed_members(precision, count, persistent):
    """Members with cell sizes that are powers of two beside others that are not, one of them with
    infiltration; 35 of them need two launches. Every member keeps its solo run's bits."""
    L = 4.0
    sizes = [(40, 33, 2.0), (29, 61, 3.0), (17, 9, 1.0), (64, 40, 5.0)]

    def fill(b, i):
        nx, ny, dx = sizes[i % 4]
        z = synth.plane_with_gaussians(nx, ny, dx, slope=0.01, seed=i)
        setup(b, z, np.full((ny, nx), 2e-3 * (1 + i % 3)), np.zeros((ny, nx)), np.zeros((ny, nx)))
        if i == 1:
            b.set_field("INFIL_RATE", np.full((ny, nx), 5e-6))
            b.set_field("INFIL_CAP", np.full((ny, nx), 1e-3))
        b.set_forcing(forcing((3e-5, 3e-5), head=(0.0, 0.0), edges=EDGE_XMAX | EDGE_YMIN))

    kw = dict(cn_target=0.5, step_duration=L, rain_mode="physical")
    batch = SaintVenantBatch(precision)
    if persistent:
        batch.set_persistent(True)
    members = [batch.add(*sizes[i % 4], **kw) for i in range(count)]
    for i, m in enumerate(members):
        fill(m, i)
    variant = batch.kernel_variant()
    batch.advance()
    for i, m in enumerate(members):
        s = SaintVenantSolver(*sizes[i % 4], precision=precision, **kw)
        s.set_kernel_variant(variant)
        fill(s, i)
        s.advance()
        for f in ("H", "U", "V"):
            assert same(m.get_field(f), s.get_field(f)), f"member {i}: {f} differs from its solo run"
    batch.close()


@pytest.mark.parametrize("variant", [16, 17])
def test_internal_kernels_are_no_variants(variant):
    s = SaintVenantSolver(8, 8, 1.0)
    with pytest.raises(SvError):
        s.set_kernel_variant(variant)
