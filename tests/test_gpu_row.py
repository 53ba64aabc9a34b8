"""The row kernels (a warp on the bra pairs of one A shell times 32 kets), the
pack kernels (a warp on one bra and several kets) and the graph replay of
short builds, against the oracle and against the thread, warp and team kernels
pinned class by class, through the C ABI.

Sizes: one molecule (segments of one bra, chunks of fewer than 32 kets), a few
(full segments, ragged last chunks), d and f shells beside the row classes."""
import numpy as np
import pytest

from dalton_b200 import _lib, molecules
from dalton_b200.basis import Molecule, build_basis
from dalton_b200.fock import FockBuilder

pytestmark = pytest.mark.gpu


def _hydrogen():
    return Molecule.from_bohr(["H", "H"], [[0.0, 0.0, -0.7], [0.0, 0.1, 0.7]])


MOLS = {
    "h2_dz": (_hydrogen, "cc-pVDZ"),
    "h2o_dz": (molecules.water_dalton_test, "cc-pVDZ"),
    "h2o3_dz": (lambda: molecules.water_cluster(3, seed=4), "cc-pVDZ"),
    "h2o7_dz": (lambda: molecules.water_cluster(7, seed=9), "cc-pVDZ"),
    "h2o2_aug": (lambda: molecules.water_cluster(2, seed=5), "aug-cc-pVDZ"),
    "c2h6_tz": (lambda: molecules.alkane(2, seed=6), "cc-pVTZ"),
}


def _density(n, seed, scale=0.1):
    d = np.random.default_rng(seed).normal(size=(n, n)) * scale
    return d + d.T


def _pin(fb, variant, fallback=None):
    """Pin every class with kernel `variant` (-5 row, -6 pack) to it, or to
    `fallback` (0: the thread kernel, or the class's next default)."""
    n = 0
    for la in range(4):
        for lb in range(la + 1):
            for lc in range(la + 1):
                for ld in range(lc + 1):
                    if la * (la + 1) // 2 + lb < lc * (lc + 1) // 2 + ld:
                        continue
                    try:
                        fb.set_class_kernel((la, lb, lc, ld), variant)
                    except _lib.DgfError:
                        continue
                    n += 1
                    if fallback is not None:
                        for v in (fallback, -3, -1):
                            try:
                                fb.set_class_kernel((la, lb, lc, ld), v)
                                break
                            except _lib.DgfError:
                                pass
    return n


OPTIONS = [{}, {"hfxfac": 0.0}, {"hfxfac": 0.3}, {"ifthrs": 9, "icedif": 0}, {"ifthrs": 11}, {"ifctyp": 23}, {"ifctyp": 11},
           {"hfxmu": 0.5, "hfxatt": 0.4}, {"thrs": 1e-8}]


@pytest.mark.parametrize("variant", [-5, -6])
@pytest.mark.parametrize("name", list(MOLS))
def test_tiled_kernels_match_quartet_kernels(cuda, name, variant):
    mol, basis = MOLS[name]
    bs = build_basis(mol(), basis)
    fb, ft = FockBuilder(bs), FockBuilder(bs)
    assert _pin(fb, variant) > 0 or name == "h2_dz"  # no d shells: no pack kernels
    for v in (-5, -6):
        _pin(ft, v, 0)
    d = _density(bs.nbf, 11)
    for o in OPTIONS:
        o = dict(o)
        dm = np.triu(d, 1) - np.triu(d, 1).T if o.get("ifctyp") == 23 else d
        ict = o.pop("ifctyp", 13)
        f, g = fb.herfck(dm, ict, **o), ft.herfck(dm, ict, **o)
        assert fb.last_stats["quartets_total"] == ft.last_stats["quartets_total"]
        assert fb.last_stats["quartets_skipped"] == ft.last_stats["quartets_skipped"]
        # the same quartets in another order of summation: rounding of sums
        # of up to nbf^2 terms of the matrices' size
        tol = 1e-15 * bs.nbf * max(1.0, np.abs(g).max())
        if "ifthrs" in o and "icedif" not in o:
            # ICEDIF looks at the integrals of a thread's chunk of A functions,
            # which the kernels cut differently: parts below the threshold may
            # be dropped or kept
            tol += 10.0 ** -o["ifthrs"] * bs.nbf
        assert np.abs(f - g).max() < tol, (o, np.abs(f - g).max(), tol)


@pytest.mark.parametrize("name", ["h2o_dz", "h2o3_dz", "h2o2_aug", "c2h6_tz"])
def test_default_kernels_match_oracle(cuda, orc, name):
    mol, basis = MOLS[name]
    bs = build_basis(mol(), basis)
    d = _density(bs.nbf, 3)
    f = FockBuilder(bs).herfck(d, 13)
    assert np.abs(f - orc.fock(bs, d, 13, 1.0, 1e-12)).max() < 1e-10


@pytest.mark.parametrize("name", ["h2o3_dz", "c2h6_tz"])
def test_several_densities(cuda, name):
    """More than one density slot: the pack kernels digest the slots one after
    the other, the row classes launch once per slot; against one build per density."""
    mol, basis = MOLS[name]
    bs = build_basis(mol(), basis)
    fb = FockBuilder(bs)
    rng = np.random.default_rng(2)
    d = rng.normal(size=(9, bs.nbf, bs.nbf)) * 0.1
    ift = [3, 13, 23, 11, 12, 1, 2, 3, 13]
    f = fb.herfck(d, ift)
    for k in range(9):
        g = fb.herfck(d[k], ift[k])
        assert np.abs(f[k] - g).max() < 1e-15 * bs.nbf * max(1.0, np.abs(g).max())


@pytest.mark.parametrize("ifctyp", [[13, 3, 3, 3, 3], [22, 2, 1, 11, 23, 3], [13] * 7 + [3, 3, 13]])
def test_general_density_at_the_slot_limit(cuda, ifctyp):
    """A general density whose two slots would be the last of one pass over the
    quartets and the first of the next; against one build per density."""
    bs = build_basis(molecules.water_cluster(2, seed=4), "cc-pVDZ")
    fb = FockBuilder(bs)
    d = np.random.default_rng(2).normal(size=(len(ifctyp), bs.nbf, bs.nbf)) * 0.1
    f = fb.herfck(d, ifctyp)
    for k, i in enumerate(ifctyp):
        g = fb.herfck(d[k], i)
        assert np.abs(f[k] - g).max() < 1e-15 * bs.nbf * max(1.0, np.abs(g).max())


@pytest.mark.parametrize("name", ["h2o3_dz", "h2o2_aug", "c2h6_tz"])
def test_several_densities_by_slot(cuda, name):
    """Several slots through the row kernels, one launch per slot, against the
    thread kernels that take all slots at once: screens over all densities,
    slots without Coulomb or exchange part, the attenuated pass, the counts."""
    mol, basis = MOLS[name]
    bs = build_basis(mol(), basis)
    fb, ft = FockBuilder(bs), FockBuilder(bs)
    _pin(fb, -5)
    for v in (-5, -6):
        _pin(ft, v, 0)
    scale = np.array([1.0, 1e-3, 1.0, 1e-2, 1.0])[:, None, None] * 0.1
    d = np.random.default_rng(12).normal(size=(5, bs.nbf, bs.nbf)) * scale
    ift = [3, 13, 22, 11, 12]
    for o in ({}, {"hfxfac": 0.0}, {"hfxfac": 0.3}, {"ifthrs": 9, "icedif": 0}, {"hfxmu": 0.5, "hfxatt": 0.4}):
        f, g = fb.herfck(d, ift, **o), ft.herfck(d, ift, **o)
        for key in ("quartets_total", "quartets_skipped", "prim_quartets"):
            assert fb.last_stats[key] == ft.last_stats[key], (o, key)
        # another order of summation of up to nbf^2 terms of the matrices' size
        assert np.abs(f - g).max() < 1e-15 * bs.nbf * max(1.0, np.abs(g).max()), o


@pytest.mark.parametrize("nshard", [2, 5])
def test_row_shards_tile(cuda, nshard):
    """Shards add up to the whole build, also when one rank's tuning pinned
    other kernels than the others'."""
    bs = build_basis(molecules.water_cluster(3, seed=4), "cc-pVDZ")
    d = _density(bs.nbf, 5)
    ref = FockBuilder(bs).herfck(d, 13)
    fbs = [FockBuilder(bs) for _ in range(nshard)]
    _pin(fbs[0], -5, 0)
    _pin(fbs[0], -6, 0)
    f = sum(fb.herfck(d, 13, shard=(r, nshard)) for r, fb in enumerate(fbs))
    assert np.abs(f - ref).max() < 1e-12 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("basis", ["6-31G*", "cc-pVTZ"])
def test_shards_tile_with_a_pinned_rank(cuda, basis):
    """The same in a segmented basis, whose whole builds run in the contracted
    form once a kernel is pinned, and with the pack kernels of f shells: one
    rank pinned, one autotuned, one with a copied tuning, the others as made."""
    import torch

    bs = build_basis(molecules.water_cluster(2, seed=4), basis)
    d = _density(bs.nbf, 5)
    ref = FockBuilder(bs).herfck(d, 13)
    fbs = [FockBuilder(bs) for _ in range(5)]
    fbs[0].set_class_kernel((1, 0, 0, 0), 0)
    fbs[1].autotune(torch.tensor(d, device=cuda))
    fbs[2].copy_tuning_from(fbs[0])
    f = sum(fb.herfck(d, 13, shard=(r, 5)) for r, fb in enumerate(fbs))
    # every quartet in one shard: only the order of the sums differs
    assert np.abs(f - ref).max() < 1e-15 * bs.nbf * max(1.0, np.abs(ref).max())


def test_graph_replay(cuda):
    """Repeated short builds (replayed as graphs from the second call on):
    new densities, buffers, streams and options between the calls, plan and
    tuning changes, against a fresh context each time."""
    import torch

    bs = build_basis(molecules.water_cluster(2, seed=8), "cc-pVDZ")
    fb = FockBuilder(bs)
    side = torch.cuda.Stream()
    opts = [{}, {"hfxfac": 0.25}, {"ifthrs": 9}, {"mixed_cutoff": 1e-6}, {"thrs": 1e-9}, {"hfxmu": 0.4, "hfxatt": 0.5}, {}]
    for i, o in enumerate(opts * 2):
        for rep in range(3):
            d = torch.tensor(_density(bs.nbf, 100 + 7 * i + rep), device=cuda)
            if rep == 2:
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    f = fb.herfck_device(d, stats=False, **o)
                torch.cuda.current_stream().wait_stream(side)
            else:
                f = fb.herfck_device(d, stats=rep == 1, **o)
            ref = FockBuilder(bs).herfck_device(d, **o)
            assert float((f - ref).abs().max()) < 1e-11 * max(1.0, float(ref.abs().max())), (o, rep)
        if i == 6:
            fb.set_class_kernel((1, 0, 1, 0), 0)


def test_capture_by_the_caller(cuda):
    """A build recorded into the caller's own CUDA graph: the launches fork
    and join inside the capture."""
    import torch

    bs = build_basis(molecules.water_cluster(2, seed=8), "cc-pVDZ")
    fb = FockBuilder(bs)
    d = torch.tensor(_density(bs.nbf, 1), device=cuda)
    f = torch.empty_like(d)
    fb.herfck_device(d, fmat=f, stats=False)  # plan and buffers
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fb.herfck_device(d, fmat=f, stats=False)
    for seed in (2, 3):
        d.copy_(torch.tensor(_density(bs.nbf, seed), device=cuda))
        g.replay()
        torch.cuda.synchronize()
        ref = FockBuilder(bs).herfck_device(d)
        assert float((f - ref).abs().max()) < 1e-11 * max(1.0, float(ref.abs().max()))
