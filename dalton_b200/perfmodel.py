"""Algorithmic FLOP model of the McMurchie-Davidson J/K quartet kernels.

One fixed count per class (la lb|lc ld), independent of how a kernel
organises the work, used as the numerator of the FP64-pipe roofline:

per primitive quartet (L = la+lb+lc+ld, N3(L) = (L+1)(L+2)(L+3)/6)
  Boys function + prefactor      40 + 3 L
  Hermite R_tuv recursion        3 * sum_{j=1..L} N3(j)
  ket contraction                2 N3(Lab) N3(Lcd) ncart_c ncart_d
  bra contraction                2 N3(Lab) ncart_a ncart_b ncart_c ncart_d
per contracted quartet
  Cartesian -> spherical         2 * (sum over transformed indices of in x out sizes x rest)
  digestion                      2 (2 + 4) n_int   (two Coulomb, four exchange blocks)
"""
from __future__ import annotations


def n3(L: int) -> int:
    return (L + 1) * (L + 2) * (L + 3) // 6


def ncart(l: int) -> int:
    return (l + 1) * (l + 2) // 2


def nsph(l: int, spherical: bool = True) -> int:
    return 2 * l + 1 if (spherical and l >= 2) else ncart(l)


def flops_per_primitive(la, lb, lc, ld) -> float:
    L, lab, lcd = la + lb + lc + ld, la + lb, lc + ld
    boys = 40 + 3 * L
    rtuv = 3 * sum(n3(j) for j in range(1, L + 1))
    ket = 2 * n3(lab) * n3(lcd) * ncart(lc) * ncart(ld)
    bra = 2 * n3(lab) * ncart(la) * ncart(lb) * ncart(lc) * ncart(ld)
    return float(boys + rtuv + ket + bra)


def flops_per_contracted(la, lb, lc, ld, spherical=True) -> float:
    ls = [la, lb, lc, ld]
    dims = [ncart(l) for l in ls]
    sph = 0
    for k, l in enumerate(ls):
        if spherical and l >= 2:
            rest = 1
            for m, d in enumerate(dims):
                if m != k:
                    rest *= d
            sph += 2 * dims[k] * (2 * l + 1) * rest
            dims[k] = 2 * l + 1
    nint = 1
    for l in ls:
        nint *= nsph(l, spherical)
    return float(sph + 2 * 6 * nint)


def class_flops(la, lb, lc, ld, prim_quartets, quartets, spherical=True) -> float:
    return prim_quartets * flops_per_primitive(la, lb, lc, ld) + quartets * flops_per_contracted(la, lb, lc, ld,
                                                                                                   spherical)


# Two-electron gradient in relative coordinates, one fixed count per class:
# per primitive quartet the Boys function and R_tuv to L+1 and, for each ket
# component, its transform to Hermite indices up to Lab+1, the contraction of
# the density product with the bra coefficients and with the lowered ones of
# each direction, the energy and the three dE/dP sums, and the three sums over
# lowered ket coefficients; per contracted quartet the density product (16
# flops per Cartesian integral).  Coefficient ranges are those of the
# components (t <= i + j in each direction).
def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _ranges(l1, l2):
    """For each component pair: the number of Hermite indices, and their
    number with one direction lowered, summed over the directions."""
    out = []
    for c in _cart(l1):
        for d in _cart(l2):
            s = [c[k] + d[k] + 1 for k in range(3)]
            full = s[0] * s[1] * s[2]
            out.append((full, sum(full // s[k] * (s[k] - 1) for k in range(3))))
    return out


def grad_flops_per_primitive(la, lb, lc, ld) -> float:
    L, lab = la + lb + lc + ld + 1, la + lb
    f = 40 + 3 * L + 3 * sum(n3(j) for j in range(1, L + 1))
    bra = sum(2 * full + 2 * low for full, low in _ranges(la, lb))
    for full, low in _ranges(lc, ld):
        f += 2 * full * n3(lab + 1) + bra + 8 * n3(lab) + 2 * low * n3(lab)
    return float(f)


def grad_flops_per_contracted(la, lb, lc, ld) -> float:
    return float(16 * ncart(la) * ncart(lb) * ncart(lc) * ncart(ld))


def grad_class_flops(la, lb, lc, ld, prim_quartets, quartets) -> float:
    return prim_quartets * grad_flops_per_primitive(la, lb, lc, ld) + quartets * grad_flops_per_contracted(la, lb, lc,
                                                                                                            ld)
