"""Permuted sums, assignments, dots and weights of blocks against numpy: equal layouts (one long
row), rows of 16 or more elements, 32 x 32 tiles where the fastest positions differ, and the
element-wise rest, at extents around those limits."""
import numpy as np
import pytest

import aquarius_b200 as A

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 7), (3, 8), (5, 16), (7, 33), (17, 31), (33, 9)]
ORDERS = ["abij", "baij", "abji", "baji"]


def plain(ctx, vrt, occ, rng):
    """Three plain [a, b, i, j] tensors with random symmetric blocks."""
    out = []
    for name in "xyz":
        t = ctx.tensor(name, (2, 0), (0, 2), plain=True)
        alpha = t.spin_cases()[0]
        n = len(vrt)
        for h in np.ndindex(n, n, n, n):
            if h[0] ^ h[1] ^ h[2] ^ h[3] == 0 and t.block_size(alpha, h):
                t.write_block(alpha, rng.standard_normal(t.block_shape(alpha, h)), h)
        out.append(t)
    return out


@pytest.mark.parametrize("split", [1, 2], ids=["c1", "two-irreps"])
@pytest.mark.parametrize("o,v", SIZES, ids=[f"o{o}v{v}" for o, v in SIZES])
def test_sums_dots_weights(o, v, split):
    rng = np.random.default_rng(100 * o + v)
    part = lambda n: [n] if split == 1 else [n - n // 3, n // 3]
    vrt, occ = part(v), part(o)
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=vrt, occ=occ)
        x, y, z = plain(ctx, vrt, occ, rng)
        fx, fy = x.to_full(), y.to_full()
        for ix in ORDERS:
            perm = [ix.index(c) for c in "abij"]
            px = fx.transpose(perm)
            # one addition per element: the two roundings of alpha * x + z bound the difference
            z["abij"] = 0.5 * x[ix]
            assert np.abs(z.to_full() - 0.5 * px).max() == 0.0, ix
            z["abij"] += -2.0 * y["abij"]
            z["abij"] += 3.0 * x[ix]
            ref = 0.5 * px - 2.0 * fy + 3.0 * px
            assert np.abs(z.to_full() - ref).max() <= 4e-16 * 16 * max(1.0, np.abs(ref).max()), ix
            z["abij"] = x[ix] if ix == "abij" else 1.0 * x[ix]
            z["abij"] -= x["abij"]
            assert np.abs(z.to_full() - (px - fx)).max() <= 1e-15 * 8, ix
            # n products in another order
            n = fx.size
            assert abs(ctx.dot(x, ix, y, "abij") - (px * fy).sum()) <= 2.3e-16 * n * np.abs(px * fy).sum() + 1e-300, ix
        dv, do = 0.5 + rng.random(v), 0.5 + rng.random(o)
        z["abij"] = y["abij"]
        ctx.weight(z, dv, do)
        den = dv[:, None, None, None] + dv[None, :, None, None] + do[None, None, :, None] + do[None, None, None, :]
        assert np.abs(z.to_full() - fy / den).max() <= 1e-15 * np.abs(fy).max()


@pytest.mark.parametrize("group", ["1", "0"], ids=["batched", "one-by-one"])
@pytest.mark.parametrize("split", [1, 2], ids=["c1", "two-irreps"])
def test_assignments_over_stale_and_shared_storage(split, group, monkeypatch):
    """C = alpha A is one pass that does not read C: what was in C, NaN included, is gone.  Sources that
    are views (<ab||ij> of <ij||ab>) are read through their strides, and a view of C itself as the source
    is not folded: C is zeroed first, as it is statement by statement."""
    monkeypatch.setenv("CCSD_GROUP_GEMMS", group)
    o, v = 5, 9
    eps, B, occ, vrt, aux = A.synth_problem(11, o, v, nirrep=split)
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=vrt, occ=occ)
        H = ctx.hamiltonian_from_factor(B, eps, aux_per_irrep=aux if split > 1 else None)
        ref = H["VABIJ"].to_full()
        assert np.array_equal(ref, H["VMNEF"].to_full().transpose(2, 3, 0, 1)) and ref.any()
        z, w = ctx.tensor("z", (2, 0), (0, 2)), ctx.tensor("w", (0, 2), (2, 0))
        for t in (z, w):
            t.fill(float("nan"))
        z["abij"] = H["VABIJ"]["abij"]
        assert np.array_equal(z.to_full(), ref)
        w["ijab"] = -2.0 * H["VABIJ"]["abij"]
        assert np.array_equal(w.to_full(), -2.0 * ref.transpose(2, 3, 0, 1))
        z.fill(float("nan"))
        ctx.sum(0.5, H["VMNEF"], "ijab", 0.0, z, "abij")
        assert np.array_equal(z.to_full(), 0.5 * ref)
        ctx.sum(0.5, H["VMNEF"], "ijab", 2.0, z, "abij")          # a scaling that is not to zero
        assert np.array_equal(z.to_full(), 1.5 * ref)
        H["VMNEF"]["mnef"] = 3.0 * H["VABIJ"]["efmn"]
        assert not H["VMNEF"].to_full().any()
