"""Device memory that calls keep or cannot do without: the scratch stays in proportion to what is computed, and a call
whose faster form does not fit in what is left of the memory takes the smaller one."""
import numpy as np
import pytest

import oracle
from pyhalma_gb300 import _lib, fof, halo_gas, halo_properties, synth

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _scratch(call):
    """Bytes of the library's scratch after one call on empty workspaces (the second, so that kernels are loaded)."""
    call()
    _lib.lib().halma_release_workspace()
    before = _free()
    call()
    return before - _free()


class _Leave:
    """All of the device's memory taken but for `nbytes`, with empty workspaces."""
    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __enter__(self):
        import torch
        _lib.lib().halma_release_workspace()
        torch.cuda.empty_cache()
        self.held = torch.empty(max(_free() - self.nbytes, 0), dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        self.held = None
        torch.cuda.empty_cache()
        _lib.lib().halma_release_workspace()


def test_fof_of_few_cells(cuda):
    """The cell pairs take their place by the cells, not by the particles."""
    import torch
    s = synth.plummer_snapshot(4_000_000, 40, seed=1, box_mpc=10.0, contaminant_frac=0.05)
    x, y, z = (torch.from_numpy(a).to(cuda) for a in (s.x, s.y, s.z))
    assert _scratch(lambda: fof.fof_labels(x, y, z, 0.0015)) < 190 * s.n


def test_gradients_where_partial_sums_do_not_fit(cuda):
    """Both ends in one sweep (34 MB of partial sums), in slices (100 MB) or with none: 12 MB are left here."""
    import torch
    ns, nt = 20_000, 20_100
    g = torch.Generator(device=cuda).manual_seed(3)
    P = _lib.ptr

    def make(ns, nt):
        T = lambda n: 0.02 * torch.randn(n, device=cuda, generator=g)
        ins = (ns, [T(ns).abs()] + [T(ns) for _ in range(3)], nt, [T(nt) for _ in range(4)])
        return ins, [torch.empty(k, device=cuda) for k in (ns, 3 * ns, 3 * nt)]

    def run(ins, out):
        ns, s, nt, t = ins
        _lib.check(_lib.lib().halma_potential_grad_f32(ns, *[P(a) for a in s], nt, *[P(a) for a in t], 1e-8, _lib.MASK_NONE,
                                                       0, *[P(a) for a in out], _lib.stream_of(s[0])), "gradients")
    ins, out = make(ns, nt)
    run(ins, out)
    want = [o.clone() for o in out]
    for k in ((1000, nt), (300, 200)):   # the kernels that are called below, loaded while there is room
        run(*make(*k))
    for o in out:
        o.zero_()
    with _Leave(12 << 20):
        run(ins, out)
        torch.cuda.synchronize()
    for o, w in zip(out, want):
        assert float((o - w).norm() / w.norm()) < 1e-6


def test_reference_potential_of_many_sources(cuda):
    import torch
    ns = 1 << 24
    x, y, z = (torch.rand(ns, device=cuda) for _ in range(3))
    m = x + 1.0
    t = [torch.full((8,), 0.3 + k, device=cuda) for k in range(3)]
    assert _scratch(lambda: halo_gas.bf_potential(m, x, y, z, *t, mode="reference")) < 100 << 20


def test_half_mass_radii_where_four_sets_do_not_fit(cuda):
    """The four half-mass radii one after another where one run for all has no room."""
    rng = np.random.default_rng(4)
    sizes = rng.integers(1000, 9000, 80)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    cols = rng.normal(0.0, 0.01, (6, n))
    m = rng.uniform(0.5, 2.0, n)
    cen = np.zeros((len(sizes), 5))
    cen[:, 3] = np.add.reduceat(m, off[:-1])
    cen[:, 4] = 0.06
    call = lambda: halo_properties.halo_property_table(off, np.arange(n, dtype=np.int32), *cols, m, cen, 0.002)
    want = call()
    used = _scratch(call)
    one = 60 * n                       # one set's scratch, of which the run of four takes four
    with _Leave(used - 2 * one):
        got = call()
    assert np.array_equal(got, want, equal_nan=True)
