"""GPU potential parity.

* reference mode: bit-identical to the float32 restatement of particle_subroutines.f90:466-514
  (sequential sum, coordinate mask, each operation rounded);
* fast mode: float32 rsqrt pair terms + compensated sums, relative error <= 1e-6 against the
  FP64 oracle (tolerance stated here: RTOL_FAST);
* FP64 comparator path: <= 1e-12 against the FP64 oracle;
* the drop-in wrappers, RPS and most_bound_particle: equal to the reference's outputs.
"""
import numpy as np
import pytest

import oracle
from pyhalma_gb300 import _lib, halo_gas, synth

pytestmark = pytest.mark.gpu
RTOL_FAST = 1e-6


def _cloud(rng, n, scale=0.01, centre=(12.3, -4.5, 7.7)):
    p = rng.normal(0, scale, (n, 3)) + np.asarray(centre)
    m = np.exp(rng.normal(np.log(1e6), 1.0, n))
    return p, m


def test_reference_mode_bit_exact(cuda):
    rng = np.random.default_rng(0)
    for ns, nt in ((1, 1), (31, 33), (1000, 257), (5003, 1999)):
        p, m = _cloud(rng, ns)
        t, _ = _cloud(rng, nt)
        got = halo_gas.bf_potential(m, p[:, 0], p[:, 1], p[:, 2], t[:, 0], t[:, 1], t[:, 2], mode="reference")
        ref = oracle.bf_potential_f32(m, p[:, 0], p[:, 1], p[:, 2], t[:, 0], t[:, 1], t[:, 2])
        assert got.dtype == np.float32
        assert np.array_equal(got, ref), (ns, nt)


def test_reference_mode_mask_and_duplicates_bit_exact(cuda):
    # AMR-like lattice: many sources share one or two coordinates with a target, duplicates too
    g = (np.arange(12) * 0.25 + 3.0).astype(np.float32)
    X, Y, Z = np.meshgrid(g, g, g, indexing="ij")
    src = np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1)
    src = np.concatenate([src, src[:50]])
    m = np.linspace(1.0, 2.0, len(src)).astype(np.float32)
    tgt = src[::7]
    got = halo_gas.bf_potential(m, *src.T, *tgt.T, mode="reference")
    ref = oracle.bf_potential_f32(m, *src.T, *tgt.T)
    assert np.array_equal(got, ref)
    fast = halo_gas.bf_potential(m, *src.T, *tgt.T, mode="fast")
    r64 = oracle.potential_f64(m, *src.T.astype(np.float64), *tgt.T.astype(np.float64), mask=oracle.MASK_COORD)
    assert np.max(np.abs(fast / r64 - 1)) < RTOL_FAST


def test_fast_mode_relative_error_vs_fp64(cuda):
    rng = np.random.default_rng(1)
    for ns, nt, eps in ((20_000, 3_000, 0.0), (100_000, 512, 1e-4), (64, 100_000, 1e-4)):
        p, m = _cloud(rng, ns)
        t, _ = _cloud(rng, nt)
        p32, t32, m32 = p.astype(np.float32), t.astype(np.float32), m.astype(np.float32)
        got = _lib.lib()  # noqa: F841 (library loads)
        phi = halo_gas.bf_potential(m32, *p32.T, *t32.T, mode="fast", eps2=eps * eps)
        ref = oracle.potential_f64(m32, *p32.T.astype(np.float64), *t32.T.astype(np.float64), eps2=eps * eps,
                                   mask=oracle.MASK_COORD)
        rel = np.abs(phi.astype(np.float64) / ref - 1.0)
        assert rel.max() < RTOL_FAST, (ns, nt, rel.max())


def test_wrapper_semantics(cuda):
    e = halo_gas.brute_force_binding_energy_fortran([1.0], [0.0], [0.0], [0.0], [], [], [])
    assert e.size == 0 and e.dtype == np.float64            # np.array([]) as in halo_gas.py:169-170
    out = halo_gas.brute_force_binding_energy_fortran([1.0, 2.0], [0.0, 1.0], [0.0, 1.0], [0.0, 1.0],
                                                      [3.0], [4.0], [5.0])
    assert out.dtype == np.float32
    # no sources: zero potential
    z = halo_gas.bf_potential([], [], [], [], [1.0, 2.0], [1.0, 2.0], [1.0, 2.0])
    assert np.array_equal(z, np.zeros(2, np.float32))


def test_fp64_path_vs_oracle(cuda):
    rng = np.random.default_rng(2)
    p, m = _cloud(rng, 3000)
    phi = np.empty(3000)
    for mask in (oracle.MASK_COORD, oracle.MASK_SELF, oracle.MASK_NONE):
        eps2 = 0.0 if mask != oracle.MASK_NONE else 1e-8
        st = _lib.lib().halma_potential_f64(3000, _lib.ptr(m), *[_lib.ptr(np.ascontiguousarray(p[:, k])) for k in range(3)],
                                            3000, *[_lib.ptr(np.ascontiguousarray(p[:, k])) for k in range(3)],
                                            eps2, mask, 0, _lib.ptr(phi), None)
        _lib.check(st, "halma_potential_f64")
        ref = oracle.potential_f64(m, *p.T, *p.T, eps2=eps2, mask=mask)
        assert np.max(np.abs(phi / ref - 1)) < 1e-12


def test_rps_and_most_bound_match_reference(golden, cuda):
    d = golden("rps.npz")
    for k in range(int(d["ncase"])):
        g = lambda n: d[f"c{k}_{n}"]
        lim, mass_dm_part = g("params")
        gas = [g(n) for n in ("gx", "gy", "gz", "gvx", "gvy", "gvz", "gm", "gt")]
        for nspec in (1, 2):
            np.random.seed(1234 + k)
            out = halo_gas.RPS(*gas, g("dx"), g("dy"), g("dz"), g("dm"), g("sx"), g("sy"), g("sz"), g("sm"),
                               *g("bulk"), int(lim), mass_dm_part, nspec)
            assert np.array_equal(np.array(out, dtype=np.float64), g(f"rps{nspec}")), (k, nspec)
        np.random.seed(999 + k)
        mb = halo_gas.most_bound_particle(gas[0], gas[1], gas[2], gas[6], g("dx"), g("dy"), g("dz"), g("dm"),
                                          g("sx"), g("sy"), g("sz"), g("sm"), g("oripa"), int(lim), mass_dm_part)
        assert np.array_equal(np.array(mb, dtype=np.float64), g("mb")), k


def test_device_tensor_path(cuda):
    import torch
    rng = np.random.default_rng(4)
    p, m = _cloud(rng, 4000)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(cuda)
    phi = halo_gas.bf_potential(t(m), t(p[:, 0]), t(p[:, 1]), t(p[:, 2]), t(p[:, 0]), t(p[:, 1]), t(p[:, 2]),
                                mode="reference")
    assert phi.is_cuda
    ref = oracle.bf_potential_f32(m, p[:, 0], p[:, 1], p[:, 2], p[:, 0], p[:, 1], p[:, 2])
    assert np.array_equal(phi.cpu().numpy(), ref)


@pytest.mark.parametrize("nt,ns,self_mask", [(20_001, 20_001, False), (20_001, 26_000, False),
                                             (9_000, 300_000, False), (12_345, 15_000, True)])
def test_self_set_potential_symmetric_route(cuda, nt, ns, self_mask):
    """Targets that are the first sources (the same device arrays): the set's pairs go through
    the symmetric block kernel, once for both particles; the other sources through the tile
    kernel.  Against the FP64 oracle at RTOL_FAST and against the tile kernel alone (the same
    targets as separate arrays) at RTOL_FAST."""
    import torch
    from pyhalma_gb300.autograd import potential_f32
    rng = np.random.default_rng(nt + ns)
    p, m = _cloud(rng, ns, scale=0.005, centre=(0.3, -0.2, 0.1))
    f = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device=cuda)
    sx, sy, sz, sm = f(p[:, 0]), f(p[:, 1]), f(p[:, 2]), f(m)
    eps = 1e-4
    so = 0 if self_mask else None
    phi = potential_f32(sx, sy, sz, sm, sx[:nt], sy[:nt], sz[:nt], eps, self_offset=so).cpu().numpy()
    tile = potential_f32(sx, sy, sz, sm, sx[:nt].clone(), sy[:nt].clone(), sz[:nt].clone(), eps,
                         self_offset=so).cpu().numpy()
    q = p.astype(np.float32).astype(np.float64)
    ref = oracle.potential_f64(m.astype(np.float32).astype(np.float64), *q.T, *q[:nt].T, eps2=eps * eps,
                               mask=oracle.MASK_SELF if self_mask else oracle.MASK_NONE)
    assert np.max(np.abs(phi / ref - 1.0)) <= RTOL_FAST
    assert np.max(np.abs(phi.astype(np.float64) / tile - 1.0)) <= RTOL_FAST


def _reference_inputs(kind, ns, nt, seed):
    """float32 sources and targets; half of the targets are sources (coincident points)."""
    rng = np.random.default_rng(seed)
    scale = {"tiny": 1e-30, "huge": 1e18}.get(kind, 0.05)
    s = (rng.normal(0.0, scale, (ns, 3)) + (3.0 if kind == "offset" else 0.0)).astype(np.float32)
    t = (rng.normal(0.0, scale, (nt, 3)) + (3.0 if kind == "offset" else 0.0)).astype(np.float32)
    k = min(ns, nt // 2)
    t[:k] = s[rng.permutation(ns)[:k]]
    m = np.exp(rng.normal(np.log(1e5), 1.0, ns)).astype(np.float32)
    if kind == "signs":
        m *= rng.choice([-1.0, 0.0, 1.0], ns).astype(np.float32)
    if kind == "ones":   # square roots whose mantissa is all ones, masses a power of two
        t[: nt // 2 + 1] = 0.0
        s[rng.random(ns) < 0.5] = np.float32([2.0 - 2.0 ** -23, 1e-7, 1e-7])
        m = (2.0 ** rng.integers(-2, 3, ns)).astype(np.float32)
    if kind == "masses":
        m = (10.0 ** rng.uniform(-37, 37, ns)).astype(np.float32)
    if kind == "nonfinite":
        s[rng.integers(0, ns), 0] = np.inf
        t[0, 1] = np.nan
        m[rng.integers(0, ns)] = np.inf
    return s, t, m


@pytest.mark.parametrize("kind,ns,nt", [
    ("offset", 1, 1), ("offset", 255, 7), ("offset", 256, 8), ("offset", 257, 9), ("centred", 1023, 33),
    ("centred", 511, 3648), ("centred", 300, 3649), ("offset", 2049, 4863), ("tiny", 700, 65), ("huge", 700, 65),
    ("signs", 513, 3700), ("ones", 600, 50), ("ones", 300, 4000), ("masses", 600, 129), ("nonfinite", 400, 40)])
def test_reference_mode_split_over_sources(cuda, kind, ns, nt):
    """Terms computed by several warps and added in order: bit for bit the sequential loop."""
    s, t, m = _reference_inputs(kind, ns, nt, 7)
    got = halo_gas.bf_potential(m, *s.T, *t.T, mode="reference")
    with np.errstate(all="ignore"):
        ref = oracle.bf_potential_f32(m, *s.T, *t.T)
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 33, 2049, 70_001])
def test_host_arrays_at_any_address(cuda, n):
    """Host inputs are copied to the device whole, in the widest words their addresses allow: the same potentials for
    arrays that start 0, 4, 8 and 12 bytes past a 16-byte boundary."""
    rng = np.random.default_rng(n)
    cols = [rng.normal(0, 1, n).astype(np.float32) for _ in range(3)] + [rng.uniform(1, 2, n).astype(np.float32)]
    tgt = [rng.normal(0, 1, 19).astype(np.float32) for _ in range(3)]

    def moved(a, k):
        raw = np.zeros(len(a) + 8, dtype=np.float32)
        first = (-raw.ctypes.data // 4) % 4 + k
        out = raw[first:first + len(a)]
        out[:] = a
        assert out.ctypes.data % 16 == 4 * k
        return out
    want = halo_gas.bf_potential(cols[3], *cols[:3], *tgt, mode="reference")
    for k in range(4):
        c, t = [moved(a, (k + q) % 4) for q, a in enumerate(cols)], [moved(a, k) for a in tgt]
        assert np.array_equal(halo_gas.bf_potential(c[3], *c[:3], *t, mode="reference"), want), k


@pytest.mark.parametrize("n", [40, 300, 5000])
def test_skipped_pair_of_an_infinite_mass(cuda, n):
    """Mask SELF leaves the self pair out whatever its mass: a particle of infinite mass has the potential of the others."""
    rng = np.random.default_rng(21)
    p, m = _cloud(rng, n)
    x, y, z, m = (np.ascontiguousarray(a, dtype=np.float32) for a in (*p.T, m))
    at = n // 3
    m[at] = np.inf
    phi = np.zeros(n, dtype=np.float32)
    P = _lib.ptr
    _lib.check(_lib.lib().halma_potential_f32(n, P(m), P(x), P(y), P(z), n, P(x), P(y), P(z), 1e-8, _lib.MASK_SELF, 0, P(phi),
                                              None), "halma_potential_f32")
    others = np.arange(n) != at
    assert np.all(np.isnan(phi[others]) | np.isinf(phi[others]))
    d = lambda a: a.astype(np.float64)
    m[at] = 0.0
    ref = oracle.potential_f64(d(m), d(x), d(y), d(z), d(x[at:at + 1]), d(y[at:at + 1]), d(z[at:at + 1]), eps2=1e-8,
                               mask=oracle.MASK_NONE)
    assert abs(phi[at] / ref[0] - 1.0) < RTOL_FAST


@pytest.mark.parametrize("ns", [2 ** 22 - 1, 2 ** 22, 2 ** 22 + 1, 2 ** 23 + 77])
def test_reference_mode_in_pieces_of_the_sources(cuda, ns):
    """More sources than are packed at a time, in one block of targets and with the plain operations in one piece alone (a
    mass outside the fast terms' range)."""
    rng = np.random.default_rng(22)
    p, m = _cloud(rng, ns)
    m[5] = 1e-20
    m[ns - 1] = 2.0 ** 20
    t, _ = _cloud(rng, 9)
    t[3] = p[ns - 1]
    got = halo_gas.bf_potential(m, *p.T, *t.T, mode="reference")
    assert np.array_equal(got, oracle.bf_potential_f32(m, *p.T, *t.T))


def test_host_pages_that_nobody_touched(cuda):
    """Inputs fresh from the allocator (zeros whose pages are not there yet) take no longer than a CPU needs to map them."""
    import time
    n = 1 << 24
    t = np.ones(1, dtype=np.float32)

    def ms(fresh):
        best = np.inf
        for _ in range(3):
            cols = [np.zeros(n, dtype=np.float32) for _ in range(4)]
            if not fresh:
                for c in cols:
                    c += 0.0
            t0 = time.perf_counter()
            assert halo_gas.bf_potential(*cols, t, t, t, mode="fast", eps2=1.0)[0] == 0.0
            best = min(best, 1e3 * (time.perf_counter() - t0))
        return best
    ms(False)
    touched, fresh = ms(False), ms(True)
    assert fresh < 2.0 * touched + 8.0, (fresh, touched)


@pytest.mark.parametrize("ns", [1, 63, 64, 65, 257, 320, 321, 600])
@pytest.mark.parametrize("nt", [1, 255, 257, 99_999, 100_000])
@pytest.mark.parametrize("plain", [False, True])
def test_reference_mode_of_few_sources_and_many_targets(cuda, ns, nt, plain):
    """Both sides of the 64 sources up to which a thread takes a target, of the 320 for 100,000 targets and more, and of that
    number, from which it does when the plain operations are needed (a mass outside the others' range)."""
    rng = np.random.default_rng(ns + nt)
    p, m = _cloud(rng, ns)
    t, _ = _cloud(rng, nt)
    t[::5] = p[rng.integers(0, ns, len(t[::5]))]
    if plain:
        m[ns // 2] = 1e-30
    got = halo_gas.bf_potential(m, *p.T, *t.T, mode="reference")
    assert np.array_equal(got, oracle.bf_potential_f32(m, *p.T, *t.T))


def test_reference_mode_has_no_stages_for_few_sources(cuda):
    """One launch with 64 sources or fewer; many targets take about as long with the plain operations as with the others."""
    import torch
    T = lambda n: torch.rand(n, device=cuda)
    x, y, z, m = T(400), T(400), T(400), T(400) + 1.0
    t = [T(300_000) for _ in range(3)]
    count = _lib.lib().halma_kernel_launch_count
    before = count()
    halo_gas.bf_potential(m[:64].clone(), x[:64].clone(), y[:64].clone(), z[:64].clone(), *t, mode="reference")
    assert count() - before == 1

    def ms():
        halo_gas.bf_potential(m, x, y, z, *t, mode="reference")
        best = np.inf
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            halo_gas.bf_potential(m, x, y, z, *t, mode="reference")
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best
    usual = ms()
    m[7] = 1e-30
    assert ms() < 1.5 * usual
