"""One-electron integrals and gradient on the working-basis pairs, the
two-electron gradient's row and warp kernels, and the resolved form of
contracted bases, against the oracle.

Sizes and bases: s, p, d and f shells, spherical and Cartesian, general and
segmented contractions, one molecule (tasks of one bra) and three."""
import numpy as np
import pytest

from dalton_b200 import molecules
from dalton_b200.basis import Molecule, build_basis
from dalton_b200.fock import FockBuilder

pytestmark = pytest.mark.gpu


def _methane():
    r = 0.63
    return Molecule.from_angstrom(["C", "H", "H", "H", "H"],
                                  [[0, 0, 0], [r, r, r], [-r, -r, r], [-r, r, -r], [r, -r, -r]])


MOLS = {
    "h2o_sto3g": (molecules.water_dalton_test, "STO-3G", True),
    "h2o2_631gs": (lambda: molecules.water_cluster(2, seed=3), "6-31G*", True),
    "h2o_631gs_cart": (molecules.water_dalton_test, "6-31G*", False),
    "h2o3_dz": (lambda: molecules.water_cluster(3, seed=4), "cc-pVDZ", True),
    "h2o_dz_cart": (molecules.water_dalton_test, "cc-pVDZ", False),
    "h2o_aug": (molecules.water_dalton_test, "aug-cc-pVDZ", True),
    "ch4_tz": (_methane, "cc-pVTZ", True),
    "ch4_tz_cart": (_methane, "cc-pVTZ", False),
}


def _basis(name):
    mol, basis, sph = MOLS[name]
    return build_basis(mol(), basis, spherical=sph)


def _density(n, seed, scale=0.1):
    d = np.random.default_rng(seed).normal(size=(n, n)) * scale
    return d + d.T


@pytest.mark.parametrize("name", list(MOLS))
def test_one_electron(cuda, orc, name):
    bs = _basis(name)
    fb = FockBuilder(bs)
    for _ in range(2):  # the scratch is kept between calls
        for x, y in zip(fb.oneint(), orc.oneint(bs)):
            # rounding of contractions of up to ten primitives
            assert np.abs(x - y).max() < 1e-13 * max(1.0, np.abs(y).max())
        d, w = _density(bs.nbf, 1), _density(bs.nbf, 2)
        g, ref = fb.grad1e(d, w), orc.grad1e(bs, d, w)
        assert np.abs(g - ref).max() < 1e-14 * bs.nbf * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("basis", ["cc-pVDZ", "6-31G*", "STO-3G"])
def test_kinetic_energy_of_s_functions(cuda, basis):
    """T between s functions against its closed form, a b / p (3 - 2 mu R^2) S,
    in extended precision: some fifteen roundings of each primitive's term
    (2e-15 of the terms' sum), also where a tight function meets a diffuse
    one."""
    bs = build_basis(molecules.water_dalton_test(), basis)
    ld = np.longdouble
    fun = []
    for i in np.nonzero(np.asarray(bs.block_l) == 0)[0]:
        c = np.asarray(bs.block_coefs(i)).astype(ld)
        x = bs.molecule.coords[int(bs.block_atom[i])].astype(ld)
        fun += [(int(bs.block_ao_offset[i]) + k, np.asarray(bs.block_exps(i)).astype(ld), c[:, k], x)
                for k in range(c.shape[1])]
    T = FockBuilder(bs).oneint()[1]
    pi = ld("3.14159265358979323846264338327950288")
    for m, a, ca, xa in fun:
        for n, b, cb, xb in fun:
            p = a[:, None] + b[None, :]
            mu = a[:, None] * b[None, :] / p
            r2 = ((xa - xb) ** 2).sum()
            t = ca[:, None] * cb[None, :] * np.exp(-mu * r2) * (pi / p) ** ld(1.5) * mu * (3 - 2 * mu * r2)
            assert abs(float(T[m, n] - t.sum())) < 2e-15 * float(np.abs(t).sum()), (m, n)


@pytest.mark.parametrize("sph", [True, False])
def test_one_electron_of_distant_shells(cuda, orc, sph):
    """Two atoms 10.3 bohr apart: the overlap distributions of their f shells
    have mu R^2 just above 40, beyond the two-electron pair lists, but their
    polynomials keep the integrals far above the block's rounding."""
    bs = build_basis(Molecule.from_bohr(["C", "C"], [[0.1, -0.2, 0.3], [10.36, 0.3, 0.8]]), "cc-pVTZ", spherical=sph)
    fb = FockBuilder(bs)
    n1 = bs.nbf // 2
    d, w = _density(bs.nbf, 1), _density(bs.nbf, 2)
    for _ in range(2):
        for x, y in zip(fb.oneint(), orc.oneint(bs)):
            # the block of the two atoms by itself: elements up to 0.05
            assert np.abs(x[:n1, n1:] - y[:n1, n1:]).max() < 1e-15
            assert np.abs(x - y).max() < 1e-13 * max(1.0, np.abs(y).max())
        # only the densities that couple the two atoms: the forces of far pairs alone
        dd, ww = d.copy(), w.copy()
        for m in (dd, ww):
            m[:n1, :n1] = m[n1:, n1:] = 0.0
        g, ref = fb.grad1e(dd, ww), orc.grad1e(bs, dd, ww)
        assert np.abs(g - ref).max() < 1e-14


@pytest.mark.parametrize("name", [n for n in MOLS if not n.startswith("ch4")])
@pytest.mark.parametrize("hfx", [1.0, 0.0, 0.3])
def test_bilinear_gradient(cuda, orc, name, hfx):
    """K(D1, D2) = [K(D1 + D2, D1 + D2) - K(D1 - D2, D1 - D2)] / 4 with the
    oracle's quadratic form; D1 = D2 through the same entry point."""
    import torch

    from dalton_b200.grad import grad2e_bilinear

    bs = _basis(name)
    fb = FockBuilder(bs)
    d1, d2 = _density(bs.nbf, 5, 0.05), _density(bs.nbf, 6, 0.05)
    dev = lambda m: torch.tensor(m, device=cuda)
    ref = (orc.grad2e(bs, d1 + d2, hfx, 1e-12) - orc.grad2e(bs, d1 - d2, hfx, 1e-12)) / 4
    # Schwarz-screened quartets differ (working basis, primitives): 1e-10 as
    # the gradient's parity elsewhere
    for _ in range(2):
        assert np.abs(grad2e_bilinear(fb, dev(d1), dev(d2), hfx).cpu().numpy() - ref).max() < 1e-10
    same = grad2e_bilinear(fb, dev(d1), dev(d1), hfx).cpu().numpy()
    assert np.abs(same - orc.grad2e(bs, d1, hfx, 1e-12)).max() < 1e-10


@pytest.mark.parametrize("name", ["h2o_sto3g", "h2o2_631gs", "h2o_631gs_cart"])
def test_resolved_contractions(cuda, orc, name):
    """Direct builds and gradients of segmented bases run in the resolved
    form until a kernel is pinned on the context; both against the oracle's
    unscreened build, the resolved one to the accuracy of its tighter
    threshold."""
    import torch

    bs = _basis(name)
    res, con = FockBuilder(bs), FockBuilder(bs)
    con.set_class_kernel((1, 0, 0, 0), 0)  # what it would choose anyway: now serves all calls itself
    d = _density(bs.nbf, 8)
    ref = orc.fock(bs, d, 13, 1.0, 0.0)
    f, g = res.herfck(d, 13), con.herfck(d, 13)
    assert res.last_stats["prim_quartets"] == res.last_stats["quartets_total"]
    assert con.last_stats["prim_quartets"] > con.last_stats["quartets_total"]
    assert np.abs(g - ref).max() < 1e-10
    assert np.abs(f - ref).max() < 1e-12 * max(1.0, np.abs(ref).max())
    assert np.abs(res.herfck(d, 13, ifthrs=10) - con.herfck(d, 13, ifthrs=10)).max() < 1e-7
    assert np.abs(res.grad2e(d) - con.grad2e(d)).max() < 1e-10
    # a store keeps contracted blocks; stored and direct builds agree
    n = res.store_integrals()
    assert n == con.store_integrals()
    dt = torch.tensor(d, device=cuda)
    assert float((res.herfck_stored(dt) - res.herfck_device(dt)).abs().max()) < 1e-11


# dgf_class_time.kernel of each kernel variant (thread variants: 0)
KERNEL_OF = {-6: 10, -5: 8, -4: 6, -3: 4, -2: 2, -1: 1}


def _kernels(fb, d, **o):
    fb.set_profiling(True)
    fb.herfck_device(d, **o)
    fb.set_profiling(False)
    return {((r["la"], r["lb"], r["lc"], r["ld"]), r["precision"]): r["kernel"] for r in fb.profile()}


@pytest.mark.parametrize("basis", ["6-31G*", "STO-3G", "cc-pVDZ"])
def test_autotune_reaches_the_builds(cuda, basis):
    """A build after the autotuner runs the kernels that its report has as the
    fastest, also where the basis is resolved, on the tuned context and on one
    that took the tuning over before or after its own first build; the mixed
    form splits the classes that the tuner split."""
    import torch

    bs = build_basis(molecules.water_cluster(2, seed=3), basis)
    d = torch.tensor(_density(bs.nbf, 8), device=cuda)
    fb, early, late = FockBuilder(bs), FockBuilder(bs), FockBuilder(bs)
    late.herfck_device(d)
    ref = early.herfck_device(d) if basis == "cc-pVDZ" else FockBuilder(bs).herfck_device(d)
    report = fb.autotune(d, mixed_cutoff=1e-6)
    for other in (early, late):
        other.copy_tuning_from(fb)
    ms, best = {}, {}
    for r in report:
        if r.get("precision") == 64:
            ms.setdefault(tuple(r["class"]), {})[KERNEL_OF.get(r["variant"], 0), r["variant"]] = r["ms"]
    for c, t in ms.items():  # the report's times are rounded: kernels at the least one are all the fastest
        best[c, 64] = {k for (k, _), x in t.items() if x == min(t.values())}
    split = {tuple(r["class"]) for r in report if r.get("split")}
    assert best
    for b in (fb, early, late):
        used = _kernels(b, d)
        assert used.keys() == best.keys() and all(used[c] in best[c] for c in used)
        mixed = _kernels(b, d, mixed_cutoff=1e-6)
        assert {c for c, p in mixed if p == 32} == split
        assert float((b.herfck_device(d) - ref).abs().max()) < 1e-15 * bs.nbf * max(1.0, float(ref.abs().max()))


@pytest.mark.parametrize("basis", ["6-31G*", "cc-pVDZ"])
def test_batch_rows(cuda, basis):
    """Batched builds with the row kernels: molecules of one to five waters,
    FP64 and mixed, replayed with new densities."""
    import torch

    from dalton_b200.batch import BatchBuilder

    fbs = [FockBuilder(build_basis(molecules.water_cluster(n, seed=n), basis)) for n in (1, 5, 2, 1, 3)]
    bb = BatchBuilder(fbs)
    out = None
    for seed in (1, 2):
        ds = [torch.tensor(_density(fb.nbf, 10 * seed + k), device=cuda) for k, fb in enumerate(fbs)]
        ref = [fb.herfck_device(d) for fb, d in zip(fbs, ds)]
        for graph in (False, True, True):
            fp = bb.herfck_batch(bb.pack(ds), out, use_graph=graph)
            for a, b in zip(bb.unpack(fp), ref):
                assert float((a - b).abs().max()) < 1e-14 * a.shape[0] * max(1.0, float(b.abs().max()))
        fm = bb.unpack(bb.herfck_batch(bb.pack(ds), use_graph=False, mixed_cutoff=1e-7))
        assert max(float((a - b).abs().max()) for a, b in zip(fm, ref)) < 1e-6


def test_capture_after_a_store(cuda):
    """A build captured into the caller's graph when only the integral store
    made a plan before: the contracted context serves it."""
    import torch

    bs = build_basis(molecules.water_cluster(2, seed=3), "6-31G*")
    fb = FockBuilder(bs)
    warm = FockBuilder(bs)
    warm.set_class_kernel((1, 0, 0, 0), 0)
    warm.herfck_device(torch.zeros((bs.nbf, bs.nbf), dtype=torch.float64, device=cuda))  # loads the kernels
    fb.store_integrals()
    d = torch.tensor(_density(bs.nbf, 1), device=cuda)
    f = torch.empty_like(d)
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
