"""The rule by which the neighbor kernels' FP32 pass settles a pair, by the
species of its sites (k_neighbors.cu: prefilter, fp32_decides, pair_test),
on the host with the same single-precision operations (numpy float32 rounds
each as the kernels do: that translation unit is compiled without FMA
contraction).

d^2 is held against rc^2 for every pair, and against a shell threshold only
where the kernels read the class it bounds: both for two Pd sites (shell
counts), the lower one for two H sites (first H shell), neither for a Pd and
an H site.  What a settled pair contributes -- its acceptance, and that part
of its class -- must be what the FP64 test gives, and a rejected pair must be
one the FP64 test rejects: on a lattice, whose Pd-H shells lie on the
thresholds, and on pairs placed within 1e-9 to 1e-1 A^2 of them."""
import numpy as np
import pytest

f32 = np.float32
RC, A = 5.35, 3.89
A75, A125 = 0.75 * A * A, 1.25 * A * A
PD, H = True, False
MAGIC = f32(12582912.0)  # 1.5 2^23


def shell_class(d2, a75, a125):
    return np.where(d2 < a75, 0, np.where((d2 > a75) & (d2 < a125), 1, 2))


def fp32_pass(xi, xj, box, iPd, jPd):
    fi, fj = xi.astype(f32), xj.astype(f32)
    boxf, inv = box.astype(f32), (1.0 / box).astype(f32)
    qmax = np.nextafter(f32(np.max(np.abs(np.concatenate([fi, fj])))), f32(np.inf))
    rcf = f32(RC)
    guard = f32(f32(1e-4) + f32(f32(1.9073486328125e-6) * f32(f32(qmax + f32(boxf.max())) + rcf)))
    lim = f32(rcf + guard)
    dd = fj - fi
    t = f32(f32(dd * inv) + MAGIC)  # rounded to an integer by the addition
    n = f32(t - MAGIC)
    dd = f32(dd - f32(n * boxf))
    m = -n.astype(np.int64)
    d2 = f32(f32(f32(dd[:, 0] * dd[:, 0]) + f32(dd[:, 1] * dd[:, 1])) + f32(dd[:, 2] * dd[:, 2]))
    near = (np.max(np.abs(dd), axis=1) <= lim) & (d2 <= f32(lim * lim))
    g = f32(lim - rcf)
    band = f32(f32(f32(f32(2.0) * g) * f32(rcf + f32(1.0))) + f32(1e-5))
    off75, off125 = np.abs(f32(d2 - f32(A75))) > band, np.abs(f32(d2 - f32(A125))) > band
    settled = near & np.all(np.abs(dd) < f32(rcf - g), axis=1) & (d2 < f32(f32(RC * RC) - band))
    if iPd == jPd:
        settled &= off75 & off125 if iPd else off75
    return near, settled & np.all(np.abs(m) <= 1, axis=1), m, d2


def check(xi, xj, box, iPd, jPd):
    near, settled, m, d2f = fp32_pass(xi, xj, box, iPd, jPd)
    dd = (xj + m * box) - xi
    d2 = dd[:, 0] * dd[:, 0] + dd[:, 1] * dd[:, 1] + dd[:, 2] * dd[:, 2]
    accepted = np.all(np.abs(dd) <= RC, axis=1) & (d2 <= RC * RC)
    assert not np.any(accepted & ~near)
    assert np.all(accepted[settled])
    c32, c64 = shell_class(d2f[settled], f32(A75), f32(A125)), shell_class(d2[settled], A75, A125)
    if iPd and jPd:
        assert np.array_equal(c32, c64)
    elif not iPd and not jPd:
        assert np.array_equal(c32 == 0, c64 == 0)
    return int(settled.sum()), int((near & ~settled).sum())


@pytest.mark.parametrize("iPd,jPd", [(PD, PD), (PD, H), (H, PD), (H, H)])
def test_lattice_pairs(iPd, jPd):
    rng = np.random.default_rng(7)
    ncell = 30  # box 116.7 A
    box = np.full(3, ncell * A)
    xi = rng.integers(0, ncell, (500, 3)) * A
    offs = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    odd = offs.sum(axis=1) % 2 != 0  # Pd and H sites: an odd number of half edges apart
    offs = offs[odd if iPd != jPd else ~odd] * (A / 2)
    xj = np.mod((xi[:, None, :] + offs[None, :, :]).reshape(-1, 3), box)
    xi = np.repeat(xi, len(offs), axis=0)
    for std in (0.0, 1e-4, 0.02):
        a, b = np.mod(xi + rng.normal(0, std, xi.shape) if std else xi, box), xj + (rng.normal(0, std, xj.shape) if std else 0)
        settled, open_ = check(a, b, box, iPd, jPd)
        assert settled > 10 * open_  # the rule leaves little to FP64


@pytest.mark.parametrize("iPd,jPd", [(PD, PD), (PD, H), (H, PD), (H, H)])
def test_pairs_at_the_thresholds(iPd, jPd):
    rng = np.random.default_rng(11)
    box = np.full(3, 30 * A)
    n = 10000
    for t2 in (A75, A125, RC * RC):
        for delta in (1e-9, 1e-7, 1e-5, 1e-3, 1e-2, 1e-1):
            u = rng.normal(size=(n, 3))
            u /= np.linalg.norm(u, axis=1)[:, None]
            xi = rng.uniform(0, box[0], (n, 3))
            d2 = t2 + delta * rng.choice([-1.0, 1.0], n)
            settled, _ = check(xi, np.mod(xi + u * np.sqrt(d2)[:, None], box), box, iPd, jPd)
            if delta == 1e-9 and iPd == jPd and not (t2 == A125 and not iPd):
                assert settled == 0  # on a threshold that is read: always FP64's
