"""The O(N) per-halo properties of the main script's property loop (pyHALMA.py:930-1016) against the
reference's own functions (golden fixture; the Fortran routines through the reference's
wrappers on the C restatement of the Fortran) and the oracle.

Tolerances: FP64 quantities whose reference sums run in an unspecified order (numba
fastmath) at 1e-10 relative; the FP32 Fortran quantities (shape, projections) and the
half-mass radii, which the GPU computes in the reference's own order, exactly.
"""
import numpy as np
import pytest

import oracle.properties as op
from oracle.reductions import CM_velocity, half_mass_radius, sigma_effective

COLS = ["cx", "cy", "cz", "mass", "rmax", "r05", "r05x", "r05y", "r05z", "vx", "vy", "vz", "jx", "jy", "jz", "j",
        "v_tf", "k_co", "a", "b", "c", "sig_3d", "sig_1d_x", "sig_1d_y", "sig_1d_z", "v_sigma", "lambda"]
EXACT = {"r05", "r05x", "r05y", "r05z", "a", "b", "c", "sig_1d_x", "sig_1d_y", "sig_1d_z", "v_sigma", "lambda"}
RTOL = 1e-10


def _load(d):
    arrays = tuple(d[k] for k in ("x", "y", "z", "vx", "vy", "vz", "m"))
    return arrays, d["off"], d["mem"], d["rows"], float(d["ll"])


def test_oracle_matches_reference_functions(golden):
    (x, y, z, vx, vy, vz, m), off, mem, rows, LL = _load(golden("properties.npz"))
    assert len(rows) >= 5
    for h, row in enumerate(rows):
        pl = mem[off[h]:off[h + 1]]
        cx, cy, cz, M, rmax = row[:5]
        r05 = half_mass_radius(cx, cy, cz, M, pl, x, y, z, m)
        r05x, r05y, r05z = op.half_mass_radius_proj(cx, cy, cz, M, pl, x, y, z, m)
        ux, uy, uz = CM_velocity(M, pl, vx, vy, vz, m)
        jx, jy, jz = op.angular_momentum(M, pl, x, y, z, vx, vy, vz, m, cx, cy, cz, ux, uy, uz)
        j = (jx ** 2 + jy ** 2 + jz ** 2) ** 0.5
        vtf = op.tully_fisher_velocity(pl, cx, cy, cz, x, y, z, ux, uy, uz, jx, jy, jz, vx, vy, vz, m, r05)
        kco = op.kinematic_morphology(pl, x, y, z, vx, vy, vz, m, cx, cy, cz, ux, uy, uz, jx, jy, jz)
        sa, sb, sc = op.halo_shape_fortran(pl, x, y, z, m, cx, cy, cz, r05)
        s3 = sigma_effective(pl, r05, x, y, z, vx, vy, vz, cx, cy, cz, ux, uy, uz)
        grid = np.arange(-(rmax + LL), rmax + LL, 2 * LL)
        sp = op.sigma_projections_fortran(grid, len(grid), pl, x, y, z, vx, vy, vz, ux, uy, uz, m, cx, cy, cz,
                                          r05x, r05y, r05z, LL)
        got = [cx, cy, cz, M, rmax, r05, r05x, r05y, r05z, ux, uy, uz, jx, jy, jz, j, vtf, kco, sa, sb, sc, s3, *sp]
        for k, (g, r) in enumerate(zip(got, row)):
            if COLS[k] in EXACT:
                assert g == r, (h, COLS[k])
            else:
                assert abs(g - r) <= RTOL * abs(r) + 1e-300, (h, COLS[k], g, r)


def test_shape_known_answer():
    # an ellipsoidal shell with semi-axes 3, 2, 1: <x^2> = a^2 / 3, so sqrt(eigenvalues) = a/sqrt(3)
    rng = np.random.default_rng(1)
    u = rng.normal(size=(100_000, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    p = u * np.array([3.0, 2.0, 1.0])
    a, b, c = op.halo_shape_fortran(np.arange(len(p)), p[:, 0], p[:, 1], p[:, 2], np.ones(len(p)), 0, 0, 0, 1.0)
    assert np.allclose([a, b, c], np.array([3.0, 2.0, 1.0]) / np.sqrt(3.0), rtol=5e-3)


@pytest.mark.gpu
def test_gpu_matches_reference_functions(golden, cuda):
    from pyhalma_gb300 import _lib, halo_properties
    (x, y, z, vx, vy, vz, m), off, mem, rows, LL = _load(golden("properties.npz"))
    t = halo_properties.halo_property_table(off, mem, x, y, z, vx, vy, vz, m, rows[:, :5], LL)
    for f in _lib.PROP_FIELDS:
        got, ref = t[:, _lib.PROP_FIELDS.index(f)], rows[:, COLS.index(f)]
        if f in EXACT:
            assert np.array_equal(got, ref.astype(np.float32).astype(np.float64) if f not in
                                  ("r05", "r05x", "r05y", "r05z") else ref), f
        else:
            np.testing.assert_allclose(got, ref, rtol=RTOL, atol=0, err_msg=f)


@pytest.mark.gpu
def test_gpu_property_loop_on_cleaned_groups(cuda):
    """FoF -> phase-space cleaning -> property loop on a 200k-particle snapshot, against the
    oracle group by group."""
    import oracle.phase_space as ops
    from pyhalma_gb300 import fof, halo_properties, phase_space, synth
    s = synth.plummer_snapshot(200_000, 60, seed=43, box_mpc=2.0, contaminant_frac=0.1)
    arrays = (s.x, s.y, s.z, s.vx, s.vy, s.vz, s.mass)
    groups = [g for g in fof.friends_of_friends_serial(s.x, s.y, s.z, 0.0015) if len(g) >= 50]
    cl = phase_space.phase_space_cleaning(groups, *arrays, 0.0015, 1.0, 3.0, True, 50)
    res = halo_properties.property_loop(cl["new_groups"], *arrays, cl["center_x"], cl["center_y"], cl["center_z"],
                                        cl["masses"], cl["rmax"], 0.0015)
    for h, pl in enumerate(cl["new_groups"]):
        cx, cy, cz, M, rmax = (cl[k][h] for k in ("center_x", "center_y", "center_z", "masses", "rmax"))
        r05 = half_mass_radius(cx, cy, cz, M, pl, s.x, s.y, s.z, s.mass)
        assert res["rad05"][h] == r05
        rp = op.half_mass_radius_proj(cx, cy, cz, M, pl, s.x, s.y, s.z, s.mass)
        assert (res["rad05_x"][h], res["rad05_y"][h], res["rad05_z"][h]) == rp
        ux, uy, uz = CM_velocity(M, pl, s.vx, s.vy, s.vz, s.mass)
        jx, jy, jz = op.angular_momentum(M, pl, *arrays[:6], s.mass, cx, cy, cz, ux, uy, uz)
        np.testing.assert_allclose([res["specific_angular_momentum_x"][h], res["specific_angular_momentum_y"][h],
                                    res["specific_angular_momentum_z"][h]], [jx, jy, jz], rtol=1e-9)
        kco = op.kinematic_morphology(pl, *arrays[:6], s.mass, cx, cy, cz, ux, uy, uz, jx, jy, jz)
        np.testing.assert_allclose(res["kinematic_morphologies"][h], kco, rtol=1e-9)
        sa, sb, sc = op.halo_shape_fortran(pl, s.x, s.y, s.z, s.mass, cx, cy, cz, r05)
        assert (res["s_axis_major"][h], res["s_axis_intermediate"][h], res["s_axis_minor"][h]) == (sa, sb, sc)
        grid = np.arange(-(rmax + 0.0015), rmax + 0.0015, 2 * 0.0015)
        sp = op.sigma_projections_fortran(grid, len(grid), pl, *arrays[:6], ux, uy, uz, s.mass, cx, cy, cz, *rp,
                                          0.0015)
        assert tuple(res[k][h] for k in ("sig_1D_x", "sig_1D_y", "sig_1D_z", "vsigma", "lambda_ensellem")) == sp


def _same(a, b):
    """Equal value for value (float32 widened exactly), NaN equal to NaN."""
    return np.array_equal(np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64), equal_nan=True)


@pytest.mark.gpu
def test_tiny_groups(cuda):
    """One- and two-member groups: the projections of a single cell, an empty Tully-Fisher
    shell (NaN here, ZeroDivisionError in the reference), shape of a degenerate tensor."""
    from pyhalma_gb300 import halo_properties
    x = np.array([0.10, 0.1004, 0.3, 0.3002, 0.3001])
    y = np.array([0.20, 0.2003, 0.1, 0.1001, 0.1003])
    z = np.array([0.00, 0.0001, 0.5, 0.5004, 0.4999])
    vx, vy, vz = np.array([[10.0, -20.0, 5.0, 7.0, -3.0], [1.0, 2.0, 3.0, 4.0, 5.0], [0.0, 1.0, -1.0, 2.0, -2.0]])
    m = np.array([1.0, 2.0, 1.0, 1.0, 3.0])
    groups = [np.array([0]), np.array([0, 1]), np.array([2, 3, 4])]
    cen = []
    for g in groups:
        M = m[g].sum()
        c = [(m[g] * a[g]).sum() / M for a in (x, y, z)]
        r = np.sqrt((c[0] - x[g]) ** 2 + (c[1] - y[g]) ** 2 + (c[2] - z[g]) ** 2).max()
        cen.append(c + [M, r])
    off = np.array([0, 1, 3, 6])
    t = halo_properties.halo_property_table(off, np.concatenate(groups), x, y, z, vx, vy, vz, m, np.array(cen), 0.0015)
    from pyhalma_gb300 import _lib
    F = {k: i for i, k in enumerate(_lib.PROP_FIELDS)}
    for h, g in enumerate(groups):
        cx, cy, cz, M, rmax = cen[h]
        r05 = half_mass_radius(cx, cy, cz, M, g, x, y, z, m)
        assert t[h, F["r05"]] == r05
        sa, sb, sc = op.halo_shape_fortran(g, x, y, z, m, cx, cy, cz, r05)
        assert _same((t[h, F["a"]], t[h, F["b"]], t[h, F["c"]]), (sa, sb, sc))
        ux, uy, uz = CM_velocity(M, g, vx, vy, vz, m)
        rp = op.half_mass_radius_proj(cx, cy, cz, M, g, x, y, z, m)
        grid = np.arange(-(rmax + 0.0015), rmax + 0.0015, 2 * 0.0015)
        sp = op.sigma_projections_fortran(grid, len(grid), g, x, y, z, vx, vy, vz, ux, uy, uz, m, cx, cy, cz, *rp,
                                          0.0015)
        assert _same(tuple(t[h, F[k]] for k in ("sig_1d_x", "sig_1d_y", "sig_1d_z", "v_sigma", "lambda")), sp)
    assert np.isnan(t[0, F["v_tf"]])


@pytest.mark.gpu
@pytest.mark.parametrize("ll", [0.0004, 0.02])
def test_projections_at_cell_and_tile_edges(cuda, ll):
    """The projections' sums with cells of one member up to all of them (small cells are a lane's, others a warp's) and
    groups at the edges of the 1,024-entry tiles: exactly the oracle's."""
    from pyhalma_gb300 import _lib, halo_properties
    rng = np.random.default_rng(7)
    sizes = [8, 9, 32, 33, 1023, 1024, 1025, 2049]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    mem = rng.permutation(n).astype(np.int32)
    x, y, z = rng.normal(0.0, 0.01, (3, n))
    vx, vy, vz = rng.normal(0.0, 100.0, (3, n))
    m = rng.uniform(0.5, 2.0, n)
    cen = []
    for h in range(len(sizes)):
        g = mem[off[h]:off[h + 1]]
        M = m[g].sum()
        c = [(m[g] * a[g]).sum() / M for a in (x, y, z)]
        cen.append(c + [M, np.sqrt((c[0] - x[g]) ** 2 + (c[1] - y[g]) ** 2 + (c[2] - z[g]) ** 2).max()])
    t = halo_properties.halo_property_table(off, mem, x, y, z, vx, vy, vz, m, np.array(cen), ll)
    F = {k: i for i, k in enumerate(_lib.PROP_FIELDS)}
    for h in range(len(sizes)):
        g = mem[off[h]:off[h + 1]]
        cx, cy, cz, M, rmax = cen[h]
        rp = tuple(t[h, F[k]] for k in ("r05x", "r05y", "r05z"))
        ux, uy, uz = (t[h, F[k]] for k in ("vx", "vy", "vz"))
        grid = np.arange(-(rmax + ll), rmax + ll, 2 * ll)
        sp = op.sigma_projections_fortran(grid, len(grid), g, x, y, z, vx, vy, vz, ux, uy, uz, m, cx, cy, cz, *rp, ll)
        assert _same(tuple(t[h, F[k]] for k in ("sig_1d_x", "sig_1d_y", "sig_1d_z", "v_sigma", "lambda")), sp), sizes[h]


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [-1, 40, 2 ** 31 - 1])
def test_member_index_out_of_range(cuda, bad):
    from pyhalma_gb300 import halo_properties
    rng = np.random.default_rng(3)
    cols = rng.uniform(0.1, 1.0, (7, 40))
    mem = np.arange(20, dtype=np.int32)
    cen = np.array([[0.5, 0.5, 0.5, cols[6, :20].sum(), 1.0]])
    off = np.array([0, 20])
    good = halo_properties.halo_property_table(off, mem, *cols, cen, 0.1)
    wrong = mem.copy()
    wrong[7] = bad
    with pytest.raises(ValueError, match="outside"):
        halo_properties.halo_property_table(off, wrong, *cols, cen, 0.1)
    assert _same(halo_properties.halo_property_table(off, mem, *cols, cen, 0.1), good)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["velocity", "mass"])
def test_non_finite_bulk_velocity(cuda, what):
    """A member outside the half-mass radius whose velocity is NaN: the bulk velocity is, and so is the dispersion about
    it.  With a NaN mass the masses have no sum, and the dispersion is that about a velocity of 0."""
    from pyhalma_gb300 import _lib, halo_properties
    rng = np.random.default_rng(12)
    n = 60
    x, y, z = rng.normal(0.0, 0.01, (3, n))
    vx, vy, vz = rng.normal(50.0, 100.0, (3, n))
    m = rng.uniform(0.5, 2.0, n)
    x[29] = 5.0
    cen = np.array([[0.0, 0.0, 0.0, m[:30].sum(), 5.0], [0.0, 0.0, 0.0, m[30:].sum(), 1.0]])
    args = lambda: (np.array([0, 30, 60]), np.arange(n, dtype=np.int32), x, y, z, vx, vy, vz, m, cen, 0.05)
    F = {k: i for i, k in enumerate(_lib.PROP_FIELDS)}
    good = halo_properties.halo_property_table(*args())
    (vx if what == "velocity" else m)[29] = np.nan
    t = halo_properties.halo_property_table(*args())
    assert _same(t[1], good[1])
    assert np.isnan(t[0, F["vx"]])
    if what == "velocity":
        assert np.isnan(t[0, F["sig_3d"]])
    else:
        d = np.sqrt(x[:30] ** 2 + y[:30] ** 2 + z[:30] ** 2)
        inside = d < t[0, F["r05"]]
        v2 = (vx[:30][inside] ** 2 + vy[:30][inside] ** 2 + vz[:30][inside] ** 2).sum()
        np.testing.assert_allclose(t[0, F["sig_3d"]], np.sqrt(v2 / 3.0 / inside.sum()), rtol=RTOL)


@pytest.mark.gpu
def test_device_table_is_not_touched_by_a_refused_call(cuda):
    import torch
    from pyhalma_gb300 import _lib
    rng = np.random.default_rng(3)
    cols = rng.uniform(0.1, 1.0, (7, 40))
    cen = np.array([[0.5, 0.5, 0.5, cols[6, :20].sum(), 1.0]])
    off, mem = np.array([0, 20]), np.arange(20, dtype=np.int32)
    D = lambda a: torch.tensor(a, device=cuda)
    arrs, dmem, doff, dcen = [D(c) for c in cols], D(mem), D(off), D(cen)
    out = torch.full((1, len(_lib.PROP_FIELDS)), 77.0, dtype=torch.float64, device=cuda)

    def call():
        return _lib.lib().halma_halo_properties(40, *[_lib.ptr(a) for a in arrs], 1, _lib.ptr(doff), _lib.ptr(dmem),
                                                _lib.ptr(dcen), 0.1, _lib.ptr(out), _lib.stream_of(out))
    dmem[7] = 40
    assert call() == _lib.ERR_INVALID
    assert bool((out == 77.0).all())
    dmem[7] = 7
    assert call() == 0
    from pyhalma_gb300 import halo_properties
    assert _same(out.cpu().numpy(), halo_properties.halo_property_table(off, mem, *cols, cen, 0.1))
