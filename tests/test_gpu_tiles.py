"""The tiled FP64 kernel at the edges of its tiles (32 and 64 rows), of its k chunks (16) and
of its shared tiles (a tile's k range cut between CTAs), odd extents included, where the two
neighbours of a copy are misaligned.  Plain tensors, so that the extents of a statement are
the orbital counts themselves; CCSD_FP64_TILED keeps narrow products on this kernel."""
import numpy as np
import pytest

import aquarius_b200 as A

pytestmark = pytest.mark.gpu

SHAPES = {"ae": ((1, 0), (1, 0)), "mi": ((0, 1), (0, 1)), "abij": ((2, 0), (0, 2)), "mnij": ((0, 2), (0, 2))}
CASES = [
    # C, idxC, A, idxA, B, idxB
    ("ae", "ae", "abij", "afmn", "abij", "efmn"),     # M = N = v, K = v o^2: shared tiles
    ("mnij", "mnij", "abij", "efmn", "abij", "efij"),  # M = N = o^2, K = v^2, both along k
    ("abij", "abij", "ae", "ae", "abij", "ebij"),     # M = v, N = v o^2, K = v
    ("abij", "abij", "mi", "mi", "abij", "abmj"),     # M = o, K = o: one short chunk
]


@pytest.mark.parametrize("o,v", [(1, 16), (3, 31), (4, 33), (5, 64), (6, 65), (9, 96), (8, 129)])
@pytest.mark.parametrize("case", CASES, ids=[f"{c[1]}+={c[3]}*{c[5]}" for c in CASES])
def test_tiles_match_numpy(case, o, v, monkeypatch):
    cs, ic, as_, ia, bs, ib = case
    monkeypatch.setenv("CCSD_FP64_TILED", "1")
    rng = np.random.default_rng(5 * o + v)
    ctx = A.Context(0)
    try:
        ctx.set_spaces(vrt=[v], occ=[o])
        host, dev = [], []
        for name, s in (("A", as_), ("B", bs), ("C", cs)):
            t = ctx.tensor(name, *SHAPES[s], plain=True)
            alpha = t.spin_cases()[0]
            x = rng.standard_normal(t.block_shape(alpha))
            t.write_block(alpha, x)
            host.append(x)
            dev.append(t)
        ctx.contract(0.5, dev[0], ia, dev[1], ib, 1.0, dev[2], ic)
        got = dev[2].to_full()
    finally:
        ctx.close()
    spec = f"{ia},{ib}->{ic}"
    ref = 0.5 * np.einsum(spec, host[0], host[1], optimize=True) + host[2]
    # two sums of K terms in any order differ by at most 2 (K + 1) u sum |a b| (the running
    # error bound of each, u = 2^-53)
    k = np.prod([v if c in "abef" else o for c in set(ia) & set(ib) - set(ic)])
    bound = 2 * (k + 2) * 2.0**-53 * (0.5 * np.einsum(spec, abs(host[0]), abs(host[1]), optimize=True) + abs(host[2]))
    assert (np.abs(got - ref) <= bound).all()
