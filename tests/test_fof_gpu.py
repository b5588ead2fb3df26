"""GPU FoF parity: bit-exact partition and labels against the reference (golden fixtures)
and against the exact C oracle at the single-GPU workload size."""
import hashlib

import numpy as np
import pytest

import oracle
from pyhalma_gb300 import fof, synth

pytestmark = pytest.mark.gpu


def _cases(d):
    return sorted(set(k.split("__")[0] for k in d.files))


def test_reference_cases_bit_exact(golden, cuda):
    d = golden("fof_cases.npz")
    for name in _cases(d):
        xyz = d[name + "__xyz"]
        ll = float(d[name + "__ll"])
        lab = fof.fof_labels(xyz[:, 0].copy(), xyz[:, 1].copy(), xyz[:, 2].copy(), ll)
        assert np.array_equal(lab, d[name + "__labels"]), name
        groups = fof.friends_of_friends(xyz, ll)
        assert groups == oracle.labels_to_groups(d[name + "__labels"]), name


def test_reference_config1_bit_exact(golden, cuda):
    c = golden("fof_config1.npz")
    x, y, z = c["x"], c["y"], c["z"]          # the exact positions the reference saw
    groups = fof.friends_of_friends_serial(x, y, z, float(c["ll"]))
    assert len(groups) == int(c["ngroups"])
    assert np.array_equal(oracle.groups_to_labels(groups, len(x)), c["labels"])


def test_two_million_particles_match_oracle(cuda):
    s = synth.plummer_snapshot(2_000_000, 500, seed=1, box_mpc=10.0, contaminant_frac=0.15)
    lab = fof.fof_labels(s.x, s.y, s.z, 0.0015)
    ref = oracle.fof_labels(s.x, s.y, s.z, 0.0015)
    assert np.array_equal(lab, ref)
    # CSR groups: reference order, strict minp filter of the "parallel" variant
    off, mem = fof.fof_groups(lab, 50)
    ref_groups = [g for g in oracle.labels_to_groups(ref) if len(g) >= 50]
    assert len(off) - 1 == len(ref_groups)
    for g in (0, len(ref_groups) // 2, len(ref_groups) - 1):
        assert mem[off[g]:off[g + 1]].tolist() == ref_groups[g]


def test_device_tensors_in_place(cuda):
    import torch
    s = synth.plummer_snapshot(50_000, 20, seed=9, box_mpc=2.0)
    x, y, z = (torch.from_numpy(a).to(cuda) for a in (s.x, s.y, s.z))
    lab = fof.fof_labels(x, y, z, 0.0015)
    assert lab.is_cuda and lab.dtype == torch.int32
    assert np.array_equal(lab.cpu().numpy(), oracle.fof_labels(s.x, s.y, s.z, 0.0015))


def test_edge_cases(cuda):
    e = np.zeros(0)
    assert fof.friends_of_friends_serial(e, e, e, 0.0015) == []
    assert fof.friends_of_friends_serial(np.array([1.0]), np.array([2.0]), np.array([3.0]), 0.0015) == []
    # zero linking length links coincident points only
    p = np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 0.0], [1e-12, 0.0, 0.0], [5.0, 5.0, 5.0], [5.0, 5.0, 5.0]])
    assert fof.friends_of_friends(p, 0.0) == [[0, 1], [3, 4]]
    # a linking length larger than the box puts everything in one group
    rng = np.random.default_rng(3)
    q = rng.uniform(0, 1, (1000, 3))
    assert fof.friends_of_friends(q, 10.0) == [list(range(1000))]
    with pytest.raises(ValueError):
        fof.friends_of_friends(np.array([[0.0, np.nan, 0.0], [0.0, 0.0, 0.0]]), 1.0)
    with pytest.raises(ValueError):
        fof.friends_of_friends(q, -1.0)


def test_parallel_variants_filter_strictly(cuda):
    s = synth.plummer_snapshot(30_000, 12, seed=2, box_mpc=1.0)
    groups = fof.friends_of_friends_parallel(s.x, s.y, s.z, 0.0015, 1.0, 50, s.mass)
    ref = [g for g in oracle.labels_to_groups(oracle.fof_labels(s.x, s.y, s.z, 0.0015)) if len(g) > 50]
    assert [g.tolist() for g in groups] == ref
    assert [g.tolist() for g in fof.pyfof_friends_of_friends_parallel(s.x, s.y, s.z, 0.0015, 1.0, 50, s.mass)] == ref


def test_dense_lattices_and_random_clusters_property(cuda):
    rng = np.random.default_rng(17)
    for trial in range(6):
        n = int(rng.integers(2_000, 40_000))
        pts = rng.normal(0, rng.uniform(0.001, 0.02), (n, 3)) + rng.uniform(-50, 50, 3)
        ll = float(rng.uniform(0.0002, 0.002))
        lab = fof.fof_labels(pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), ll)
        assert np.array_equal(lab, oracle.fof_labels(pts[:, 0], pts[:, 1], pts[:, 2], ll)), trial
    # ties: lattice spacing equal to the linking length at large coordinates
    pts = synth.lattice_points(24, 0.0015, origin=(37.1, -12.3, 4.4), jitter_ulps=1, seed=4)
    lab = fof.fof_labels(pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), 0.0015)
    assert np.array_equal(lab, oracle.fof_labels(pts[:, 0], pts[:, 1], pts[:, 2], 0.0015))


def test_far_offsets_and_elongated_boxes(cuda):
    """Cell keys stay exact far from the origin (a cloud 3e4 Mpc away) and on grids millions of
    cells long on one axis (a chain of particles 0.5-1.2 LL apart)."""
    rng = np.random.default_rng(23)
    pts = rng.normal(0, 0.003, (20_000, 3)) + np.array([1.0e4, -2.5e4, 7.5e3])
    lab = fof.fof_labels(pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), 0.0007)
    assert np.array_equal(lab, oracle.fof_labels(pts[:, 0], pts[:, 1], pts[:, 2], 0.0007))
    n = 6000
    chain = np.zeros((n, 3))
    chain[:, 0] = 3.0e3 + np.cumsum(rng.uniform(0.5, 1.2, n)) * 0.001
    chain[:, 1] = rng.normal(0, 2e-5, n)
    chain[:, 2] = -4.0e2 + rng.normal(0, 2e-5, n)
    chain = np.concatenate([chain, chain[::7] + np.array([0.0, 1.0, 0.0])])   # a second, sparser line
    lab = fof.fof_labels(chain[:, 0].copy(), chain[:, 1].copy(), chain[:, 2].copy(), 0.001)
    assert np.array_equal(lab, oracle.fof_labels(chain[:, 0], chain[:, 1], chain[:, 2], 0.001))


def test_flat_and_thin_grids(cuda):
    """Grids one cell thick on one or two axes (planes and lines of particles): the neighbour
    keys of the padded key grid wrap across a row or column end there on every cell, and must
    land on the pad, never on a cell of the next row."""
    rng = np.random.default_rng(29)
    ll = 0.001
    cases = []
    # planes z = const (one cell in z), y = const (one cell in y)
    pl = rng.uniform(0, 0.2, (20_000, 3))
    cases.append((pl[:, 0], pl[:, 1], np.full(len(pl), 0.5)))
    cases.append((pl[:, 0], np.full(len(pl), -0.25), pl[:, 1]))
    # lines along x, y and z with steps of 0.5-1.2 LL and a parallel line 1.5 LL away
    for axis in range(3):
        t = np.cumsum(rng.uniform(0.5, 1.2, 5000)) * ll
        a = [np.full(len(t), 0.3), np.full(len(t), 0.3), np.full(len(t), 0.3)]
        a[axis] = t
        b = [v.copy() for v in a]
        b[(axis + 1) % 3] = b[(axis + 1) % 3] + 1.5 * ll
        cases.append(tuple(np.concatenate([u, v]) for u, v in zip(a, b)))
    for k, (x, y, z) in enumerate(cases):
        x, y, z = (np.ascontiguousarray(v, dtype=np.float64) for v in (x, y, z))
        lab = fof.fof_labels(x, y, z, ll)
        assert np.array_equal(lab, oracle.fof_labels(x, y, z, ll)), k


def test_integer_and_fma_key_maps(cuda):
    """Both maps from coordinates to quarter cells: the integer one (coordinates and grid within
    2^37 quarter cells) on a cloud straddling zero with signed zeros, subnormals and points on
    multiples of the linking length, and the FP64 FMA one on a cloud 1e8 length units from the
    origin (4e11 quarter cells), each against the oracle."""
    rng = np.random.default_rng(31)
    ll = 0.001
    pts = rng.normal(0, 0.004, (30_000, 3))
    special = np.array([[0.0, -0.0, 5e-324], [-5e-324, 0.0, -0.0], [2.2e-308, -2.2e-308, 0.0],
                        [ll, -ll, 0.0], [2 * ll, 0.0, -3 * ll], [-ll, -ll, -ll], [0.5 * ll, 0.5 * ll, 0.0]])
    grid = np.stack(np.meshgrid(*(np.arange(-4, 5) * ll,) * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    pts = np.concatenate([pts, special, grid, grid + np.array([ll * (1 + 2 ** -40), 0.0, 0.0])])
    lab = fof.fof_labels(pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), ll)
    assert np.array_equal(lab, oracle.fof_labels(pts[:, 0], pts[:, 1], pts[:, 2], ll))
    far = rng.normal(0, 0.004, (20_000, 3)) + np.array([1.0e8, -3.0e7, 2.0e8])
    lab = fof.fof_labels(far[:, 0].copy(), far[:, 1].copy(), far[:, 2].copy(), ll)
    assert np.array_equal(lab, oracle.fof_labels(far[:, 0], far[:, 1], far[:, 2], ll))


def test_groups_reject_labels_that_are_not_particle_indices(cuda):
    """Labels index the per-group counters; one outside [-1, n) is refused by the kernel that
    reads it (host and device labels), and the next call works as before."""
    import torch
    for bad in (np.array([0, 0, 5, -1, 2], dtype=np.int32), np.array([0, 0, -2, -1, 2], dtype=np.int32)):
        with pytest.raises(ValueError, match="labels"):
            fof.fof_groups(bad)
        with pytest.raises(ValueError, match="labels"):
            fof.fof_groups(torch.from_numpy(bad).to(cuda))
    off, mem = fof.fof_groups(np.array([0, 0, -1, 3, 3, 3], dtype=np.int32))
    assert off.tolist() == [0, 2, 5] and mem.tolist() == [0, 1, 3, 4, 5]


def _clumps(n, sep, spread, seed):
    """Two clumps of n points on x = 0 and x = sep (Mpc), spread in y and z only."""
    rng = np.random.default_rng(seed)
    p = np.zeros((2 * n, 3))
    p[n:, 0] = sep
    p[:, 1:] = rng.uniform(0.0, spread, (2 * n, 2))
    return np.ascontiguousarray(p[rng.permutation(2 * n)].T)


@pytest.mark.parametrize("n,sep,spread", [
    (31, 1.5e-3, 1e-4), (33, 1.5001e-3, 1e-4), (700, 1.49999e-3, 2e-4), (3000, 1.4999999e-3, 5e-4),
    (3000, 1.50001e-3, 5e-4), (20000, 1.50001e-3, 6e-4)])
def test_crowded_half_cells_a_linking_length_apart(cuda, n, sep, spread):
    """Pairs of nodes with more than a thread's share of tests, with few links or none between them."""
    ll = 1.5e-3
    x, y, z = _clumps(n, sep, spread, 3)
    x += 0.11
    lab = fof.fof_labels(x, y, z, ll)
    # a clump is one group (its spread is below the linking length); they join where a pair is near enough
    left = x < 0.11 + sep / 2
    d2 = np.inf
    for b in range(0, n, 2000):   # the smallest separation squared, in the predicate's own order of operations
        i, j = np.nonzero(left)[0][b:b + 2000], np.nonzero(~left)[0]
        dx, dy, dz = (a[i][:, None] - a[j][None, :] for a in (x, y, z))
        d2 = min(d2, ((dx * dx + dy * dy) + dz * dz).min())
    first = [np.nonzero(left)[0][0], np.nonzero(~left)[0][0]]
    want = np.where(left, first[0], first[1]) if d2 > ll * ll else np.zeros(2 * n, dtype=np.int64)
    assert np.array_equal(lab, want)


@pytest.mark.parametrize("ll,box,n", [(0.0, 1.0, 9000), (4.0 / 1.45e6, 4.0, 5000), (5000.0 / 1.4e6, 5000.0, 20000)])
def test_particles_as_nodes(cuda, ll, box, n):
    """No half-cells in the key: coincident points only (ll = 0, crowded cells), and grids whose keys leave
    no room for them."""
    rng = np.random.default_rng(11)
    p = rng.uniform(0.0, box, (n // 3, 3))
    p = np.concatenate([p, p[rng.integers(0, len(p), n // 3)], np.full((n // 3, 3), box / 3)])
    if ll > 0:
        p[n // 3:2 * (n // 3)] += rng.normal(0.0, 0.4 * ll, (n // 3, 3))
    p = p[rng.permutation(len(p))]
    x, y, z = (np.ascontiguousarray(c) for c in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), oracle.fof_labels(x, y, z, ll))


def _filled(x, y, z, ll, total):
    """The points followed by isolated ones beyond them, `total` in all: past the limit of the small path."""
    k = total - len(x)
    step = 4.0 * ll if ll > 0 else 1.0
    fx = (x.max() if len(x) else 0.0) + step * (1.0 + np.arange(k))
    f = lambda a, b: np.ascontiguousarray(np.concatenate([a, b]))
    return f(x, fx), f(y, np.zeros(k)), f(z, np.zeros(k))


@pytest.mark.parametrize("total", [8192, 8193, 16384, 16385])
def test_both_sides_of_the_small_path(golden, cuda, total):
    """The reference's own cases on the all-pairs path and, filled up past its limit, on the cell path."""
    d = golden("fof_cases.npz")
    for name in _cases(d):
        x, y, z = (np.ascontiguousarray(c) for c in d[f"{name}__xyz"].astype(np.float64).T)
        ll = float(d[f"{name}__ll"])
        if len(x) > total:
            continue
        want = oracle.fof_labels(x, y, z, ll)
        fx, fy, fz = _filled(x, y, z, ll, total)
        lab = fof.fof_labels(fx, fy, fz, ll)
        assert np.array_equal(lab[:len(x)], want), name
        assert (lab[len(x):] == -1).all(), name
        off, mem = fof.fof_groups(lab, 2)
        woff, wmem = fof.fof_groups(want, 2)
        assert np.array_equal(off, woff) and np.array_equal(mem, wmem), name


@pytest.mark.parametrize("far,ll", [(0.0, 1.5e-3), (3e5, 1.5e-3), (1e300, 1e290), (5.0, 1e-310)])
def test_small_path_on_far_coordinates(cuda, far, ll):
    """Coordinates beyond 2^24 linking lengths of the first particle are tested in FP64."""
    rng = np.random.default_rng(4)
    s = min(ll, 1e290) if ll > 1e-300 else 1e-310
    p = rng.uniform(0.0, 12.0, (1500, 3)) * s
    p[700:] += far
    x, y, z = (np.ascontiguousarray(c) for c in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), _brute(p, ll))


def _brute(p, ll):
    n = len(p)
    lab = np.arange(n)
    with np.errstate(all="ignore"):
        adj = [np.nonzero(((p[i, 0] - p[:, 0]) ** 2 + (p[i, 1] - p[:, 1]) ** 2) + (p[i, 2] - p[:, 2]) ** 2 <= ll * ll)[0]
               for i in range(n)]
    while True:
        new = np.array([lab[a].min() if len(a) else lab[i] for i, a in enumerate(adj)])
        if np.array_equal(new, lab):
            break
        lab = new
    alone = np.array([len(a) <= 1 for a in adj])
    return np.where(alone, -1, lab)


@pytest.mark.parametrize("n", [1, 31, 1023, 1025, 5000, 8192, 8193, 30000])
def test_groups_of_given_labels(cuda, n):
    """Groups from labels alone, in the order of their smallest members, on both sides of the one-block path."""
    rng = np.random.default_rng(n)
    head = np.minimum(np.arange(n), (rng.uniform(0, 1, n) ** 3 * n).astype(np.int64))
    while not np.array_equal(head, head[head]):
        head = head[head]
    lab = np.where(rng.random(n) < 0.1, -1, head).astype(np.int32)
    lab[np.unique(lab[lab >= 0])] = np.unique(lab[lab >= 0])
    for minp in (1, 2, 7):
        off, mem = fof.fof_groups(lab, minp)
        heads, count = np.unique(lab[lab >= 0], return_counts=True)
        heads = heads[count >= minp]
        assert len(off) == len(heads) + 1
        for g, h in enumerate(heads):
            assert np.array_equal(mem[off[g]:off[g + 1]], np.nonzero(lab == h)[0])


@pytest.mark.parametrize("ll", [1e200, 1e-170])
def test_small_path_where_the_predicate_leaves_the_range(cuda, ll):
    """The FP64 predicate overflows (or underflows) on both sides at the linking length: it, not the floats, decides."""
    rng = np.random.default_rng(4)
    p = rng.uniform(0.0, 12.0, (1500, 3)) * ll
    x, y, z = (np.ascontiguousarray(c) for c in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), _brute(p, ll))


@pytest.mark.parametrize("reach", [2.0 ** 19, 2.0 ** 21, 3.0 ** 14, 2.0 ** 23.5, 2.0 ** 27, 2.0 ** 36, 2.0 ** 45])
def test_small_path_with_an_outlier(cuda, reach):
    """Friends around the linking length, half of them `reach` linking lengths from the other half: looked at by one
    float, by both, and beyond that in FP64."""
    rng = np.random.default_rng(14)
    ll = 1.5e-3
    p = rng.uniform(0.0, 12.0, (1500, 3)) * ll
    p[::2] += reach * ll / np.sqrt(3.0)
    p[3] = p[2] + np.array([ll, 0.0, 0.0])
    p[5] = p[2] + np.array([0.0, ll * (1 + 1e-15), 0.0])
    x, y, z = (np.ascontiguousarray(c) for c in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), _brute(p, ll))


@pytest.mark.parametrize("what", ["outlier", "zero linking length"])
def test_small_path_is_not_quadratic_in_friends(cuda, what):
    """A crowd of 16,384 friends with one particle 1e8 linking lengths away takes about as long as the crowd alone, and
    coordinates far below one unit with linking length 0 as long as ordinary ones."""
    import torch
    rng = np.random.default_rng(15)
    n, ll = 16_384, 1.5e-3
    p = rng.normal(0.0, 2.0 * ll, (3, n))
    far = p.copy()
    if what == "outlier":
        far[:, 7] = 1e8 * ll
    else:
        ll, p, far = 0.0, 1e3 * p, 1e-9 * p

    def ms(a):
        x, y, z = (torch.tensor(c, device=cuda) for c in a)
        fof.fof_labels(x, y, z, ll)
        best = np.inf
        for _ in range(3):
            torch.cuda.synchronize()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            lab = fof.fof_labels(x, y, z, ll)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best, lab.cpu().numpy()
    (alone, _), (took, lab) = ms(p), ms(far)
    assert took < 3.0 * alone + 0.1, (took, alone)
    x, y, z = (np.ascontiguousarray(c) for c in far)
    keep = np.arange(n) != 7
    want = oracle.fof_labels(x[keep], y[keep], z[keep], ll)
    idx = np.nonzero(keep)[0]
    assert np.array_equal(lab[keep], np.where(want >= 0, idx[want], -1))


@pytest.mark.parametrize("n", [500, 16_384, 16_385])
def test_labels_are_not_touched_by_a_refused_call(cuda, n):
    import torch
    from pyhalma_gb300 import _lib
    rng = np.random.default_rng(16)
    x, y, z = (torch.tensor(c, device=cuda) for c in rng.uniform(0.0, 1.0, (3, n)))
    y[n // 3] = float("inf")
    lab = torch.full((n,), 77, dtype=torch.int32, device=cuda)
    st = _lib.lib().halma_fof(n, _lib.ptr(x), _lib.ptr(y), _lib.ptr(z), 0.05, _lib.ptr(lab), None, _lib.stream_of(x))
    assert st == _lib.ERR_INVALID
    assert bool((lab == 77).all())


def test_member_count_of_the_last_call(cuda):
    """halma_last_group_members(): what the thread's last successful call stored; 0 after an empty one, and as it was after
    one that failed."""
    import ctypes
    from pyhalma_gb300 import _lib
    L = _lib.lib()
    lab = np.array([0, 0, -1, 3, 3, 3], dtype=np.int32)
    off, mem, ng = np.zeros(7, dtype=np.int64), np.zeros(6, dtype=np.int32), ctypes.c_int64()
    call = lambda n, l: L.halma_fof_groups(n, _lib.ptr(l), 2, _lib.ptr(off), _lib.ptr(mem), ctypes.byref(ng), None)
    assert call(6, lab) == 0 and L.halma_last_group_members() == 5
    bad = np.array([0, 0, 9, 3, 3, 3], dtype=np.int32)
    assert call(6, bad) == _lib.ERR_INVALID and L.halma_last_group_members() == 5
    assert call(0, lab) == 0 and L.halma_last_group_members() == 0
    from pyhalma_gb300.unbinding import find_haloes
    assert call(6, lab) == 0 and L.halma_last_group_members() == 5
    e = np.zeros(0)
    find_haloes(e, e, e, e, e, e, e, 0.0015)
    assert L.halma_last_group_members() == 0


@pytest.mark.parametrize("n", [8, 9, 60, 181, 182, 300])
@pytest.mark.parametrize("sep", [1.4e-3, 1.4999999e-3, 1.50001e-3])
def test_pairs_of_nodes_by_a_lane_a_warp_and_a_block(cuda, n, sep):
    """Many pairs of clumps at the numbers of tests where a lane (64), a warp (32,768) and a block take over, linked by few
    particles, by pairs at the linking length, or not at all."""
    rng = np.random.default_rng(n)
    ll, k = 1.5e-3, max(20, 20_000 // n)
    c = np.stack(np.meshgrid(np.arange(40), np.arange(40), np.arange(40), indexing="ij"), -1).reshape(-1, 3)[:k] * (8 * ll)
    a = c[:, None, :] + rng.uniform(-1.0, 1.0, (k, n, 3)) * [0.0, 2e-4, 2e-4]
    b = c[:, None, :] + [sep, 0.0, 0.0] + rng.uniform(-1.0, 1.0, (k, n, 3)) * [1e-8, 2e-4, 2e-4]
    p = np.concatenate([a.reshape(-1, 3), b.reshape(-1, 3)])
    if len(p) <= 16_384:   # past the all-pairs limit
        p = np.concatenate([p, np.stack([1.0 + 0.01 * np.arange(17_000 - len(p))] * 3, 1)])
    p = p[rng.permutation(len(p))]
    x, y, z = (np.ascontiguousarray(q) for q in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), oracle.fof_labels(x, y, z, ll))


@pytest.mark.parametrize("copies", [8, 9, 64, 65, 256, 257, 1000])
@pytest.mark.parametrize("ll", [0.0, 1e-6])
def test_copies_of_particles(cuda, copies, ll):
    """Coincident particles, with linking length 0 (particles as nodes) and a small one, around the sizes at which a lane, a warp
    and a block take a pair of cells; some copies a little apart."""
    rng = np.random.default_rng(copies)
    p = np.repeat(rng.uniform(0.0, 1.0, (24_000 // copies, 3)), copies, axis=0)
    p[rng.random(len(p)) < 0.1] += 0.5e-6
    p = p[rng.permutation(len(p))]
    x, y, z = (np.ascontiguousarray(q) for q in p.T)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), oracle.fof_labels(x, y, z, ll))


@pytest.mark.parametrize("what", ["clumps", "lattice", "sheets", "copies"])
def test_crowded_cells_take_no_longer_than_spread_ones(cuda, what):
    """Particles crowded in half-cells that are not linked to their neighbours, or only here and there, against as many
    spread out."""
    import torch
    rng = np.random.default_rng(18)
    n, ll = 400_000, 1.0
    if what == "clumps":
        p = np.repeat(rng.uniform(0.0, 45.0, (n // 200, 3)), 200, axis=0) + rng.normal(0.0, 0.05, (n, 3))
    elif what == "lattice":
        p = np.round(rng.uniform(0.0, 20.0, (n, 3))) * 0.5
    elif what == "sheets":
        n = 100_000
        p = rng.uniform(0.0, 0.3, (n, 3)) * [0.0, 1.0, 1.0]
        p[::2, 0] = 1.3
    else:
        p, ll = np.repeat(rng.uniform(0.0, 10.0, (n // 500, 3)), 500, axis=0), 0.0

    def ms(q, ll):
        x, y, z = (torch.tensor(np.ascontiguousarray(c), device=cuda) for c in q.T)
        fof.fof_labels(x, y, z, ll)
        best = np.inf
        for _ in range(3):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            fof.fof_labels(x, y, z, ll)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best
    spread, took = ms(rng.uniform(0.0, 70.0, (n, 3)), 1.0), ms(p, ll)
    assert took < 4.0 * spread, (took, spread)


@pytest.mark.parametrize("sigma", [0.3, 1.0, 3.0])
def test_crowded_cells_of_a_grid_without_room_for_half_cells(cuda, sigma):
    """A crowd whose box is 1.5e6 linking lengths wide for the sake of one particle: particles are the nodes."""
    rng = np.random.default_rng(19)
    n, ll = 60_000, 1.0
    p = rng.normal(0.0, sigma, (3, n))
    p[:, 7] = 1.5e6
    x, y, z = (np.ascontiguousarray(c) for c in p)
    assert np.array_equal(fof.fof_labels(x, y, z, ll), oracle.fof_labels(x, y, z, ll))
