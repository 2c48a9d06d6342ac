"""Split (BF16 and INT8 slice) tcgen05 contractions against the native-FP64 path and the oracle.

Tolerances: a single contraction agrees with FP64 to 2e-6 of max|C| with three BF16 slices
per operand (8 bits each, the leading product exact, errors unbiased), 1e-8 with four;
INT8 slices carry 7.99 bits each (3e-5, 3e-7, 3e-9 for three, four, five).  A full CCSD solve
agrees with the FP64 oracle to |dE| <= 1e-8 Eh and max|dT| <= 1e-7 at every iteration with
three BF16 or four INT8 slices.
"""
import time

import numpy as np
import pytest

import aquarius_b200 as A
from oracle import ccsd_oracle as O
from tests.helpers import random_so, write_full

pytestmark = pytest.mark.gpu

SHAPES = {"abij": ((2, 0), (0, 2)), "abef": ((2, 0), (2, 0)), "amei": ((1, 1), (1, 1)), "mnef": ((0, 2), (2, 0))}


def _contract(precision, o, v, ia, sa, ib, sb, ic, sc, seed, packed_a=False, slices=0):
    rng = np.random.default_rng(seed)
    ctx = A.Context(0)
    try:
        ctx.set_spaces(vrt=[v], occ=[o])
        if precision != "fp64":
            ctx.set_precision(precision, slices=slices)
            ctx.set_split_routing("all")   # these sizes would stay on FP64 otherwise
        tA = ctx.tensor("A", *SHAPES[sa], packed=packed_a)
        tB = ctx.tensor("B", *SHAPES[sb])
        tC = ctx.tensor("C", *SHAPES[sc])
        write_full(tA, random_so(ctx, *SHAPES[sa], rng, scale=0.05))
        write_full(tB, random_so(ctx, *SHAPES[sb], rng, scale=0.01))
        ctx.contract(0.5, tA, ia, tB, ib, 0.0, tC, ic)
        if precision != "fp64":
            assert ctx.split_launches() > 0
        else:
            assert ctx.split_launches() == 0
        return tC.to_full()
    finally:
        ctx.close()


@pytest.mark.parametrize("case", [
    ("abef", "abef", "abij", "efij", "abij", "abij", True),     # particle ladder
    ("amei", "amei", "abij", "ebjm", "abij", "abij", False),    # ring with antisymmetriser images
    ("mnef", "mnef", "abij", "afni", "amei", "amei", False),    # W(am,ei) build
], ids=["ladder", "ring", "wamei"])
@pytest.mark.parametrize("precision,slices,tol", [
    ("split", 3, 2e-6), ("split", 4, 1e-8), ("split_i8", 3, 3e-5), ("split_i8", 4, 3e-7), ("split_i8", 5, 3e-9),
], ids=["bf16x3", "bf16x4", "i8x3", "i8x4", "i8x5"])
def test_split_contraction_matches_fp64(case, precision, slices, tol):
    """BF16: three slices 2e-6 of max|C| (FP32-like inputs), four 1e-8 (2^-8 finer);
    INT8: 7.99 bits per slice."""
    sa, ia, sb, ib, sc, ic, packed = case
    o, v = 6, 40
    ref = _contract("fp64", o, v, ia, sa, ib, sb, ic, sc, 11, packed)
    got = _contract(precision, o, v, ia, sa, ib, sb, ic, sc, 11, packed, slices=slices)
    scale = np.abs(ref).max()
    assert scale > 0
    assert np.abs(got - ref).max() <= tol * scale


@pytest.mark.parametrize("precision,slices,etol,ttol", [
    ("split", 3, 1e-8, 1e-7), ("split", 4, 1e-10, 1e-9), ("split_i8", 3, 2e-7, 2e-6), ("split_i8", 4, 1e-8, 1e-7),
    ("split_i8", 5, 1e-10, 1e-9),
], ids=["bf16x3", "bf16x4", "i8x3", "i8x4", "i8x5"])
@pytest.mark.parametrize("o,v,seed", [(4, 40, 21), (6, 48, 22)])
def test_split_solve_matches_oracle_every_iteration(o, v, seed, precision, slices, etol, ttol):
    eps, B, *_ = A.synth_problem(seed, o, v)
    ref = O.CCSD(O.hamiltonian_from_factor(B, eps, o), diis_order=8)
    ctx = A.Context(0)
    try:
        ctx.set_spaces(vrt=[v], occ=[o])
        ctx.set_split_routing("all")
        H = ctx.hamiltonian_from_factor(B, eps)
        s = ctx.solver(H, diis_order=8, precision=precision, slices=slices)
        for it in range(10):
            e_ref, _ = ref.iterate()
            e, _ = s.iterate()
            assert abs(e - e_ref) <= etol, (it, e, e_ref)
        assert ctx.split_launches() > 0
        assert np.abs(s.T2.to_full() - ref.T.T2).max() <= ttol
        assert np.abs(s.T1.to_full() - ref.T.T1).max() <= ttol
        s.close()
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", ["split", "split_i8"])
def test_refinement_moves_to_four_slices_and_converges(precision):
    """refine_tol: 3-slice contractions until conv < refine_tol, then 4 slices (and 5 INT8
    slices on a stall); the solve reaches conv_tol and the oracle's converged energy."""
    o, v, seed = 4, 40, 23
    eps, B, *_ = A.synth_problem(seed, o, v)
    ref = O.CCSD(O.hamiltonian_from_factor(B, eps, o), diis_order=8)
    e_ref = ref.run(1e-10, 80)
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=[v], occ=[o])
        ctx.set_split_routing("all")
        H = ctx.hamiltonian_from_factor(B, eps)
        s = ctx.solver(H, diis_order=8, precision=precision, conv_tol=1e-10, max_iter=80, refine_tol=1e-6)
        e, c, it = s.run()
        assert c < 1e-10
        assert abs(e - e_ref) < 1e-10, (e, e_ref)
        s.close()


SHAPES.update(amef=((1, 1), (2, 0)), amij=((1, 1), (0, 2)))


@pytest.mark.parametrize("slices", [3, 4, 5])
@pytest.mark.parametrize("o,v", [(3, 11), (5, 27), (7, 34)], ids=lambda x: str(x))
def test_int8_slices_at_odd_extents(o, v, slices):
    """Rows and k that end inside a packed group of four, both orientations of the gather, and a bound
    that a lost slice does not meet.  An operand of standard deviation s and row maxima up to m is
    rounded to multiples of u = m / 127 / 254^(n-1), so that it is off by u / sqrt(12), independently;
    the products left out (n - 1 of them at level n) are of two digits of 127 / sqrt(3) each, weight
    254^-n (m / 127)^2.  K terms add as sqrt(K), four images at most add to an element, and the largest
    of some 10^5 elements stays within six deviations."""
    sa, sb, m = 0.05, 0.01, 5.0                       # m: row maximum in standard deviations

    def bound(n, K):
        rounding = 2 * m / 127 / 254.0 ** (n - 1) / 12**0.5
        left_out = (n - 1) ** 0.5 * (127 / 3**0.5) ** 2 * 254.0**-n * (m / 127) ** 2
        return 6 * 0.5 * (4 * K) ** 0.5 * sa * sb * (rounding + left_out)

    for xa, ia, xb, ib, xc, ic, K in (("amei", "amei", "abij", "ebjm", "abij", "abij", 2 * o * v),
                                      ("amef", "amef", "abij", "efij", "amij", "amij", 4 * v * v)):
        ref = _contract("fp64", o, v, ia, xa, ib, xb, ic, xc, 5, False)
        err = lambda n: np.abs(_contract("split_i8", o, v, ia, xa, ib, xb, ic, xc, 5, False, slices=n) - ref).max()
        assert err(slices) <= bound(slices, K), xa
        if slices > 3:
            assert err(slices - 1) > bound(slices, K), xa     # one slice less is seen


@pytest.mark.parametrize("precision,slices", [("split", 3), ("split", 4), ("split_i8", 3), ("split_i8", 4), ("split_i8", 5)],
                         ids=["bf16x3", "bf16x4", "i8x3", "i8x4", "i8x5"])
def test_tiles_of_one_cta_follow_one_another(precision, slices):
    """2401 x 2401 x 16641: 361 tiles of 128 x 128 (722 of 128 x 64), two and more per CTA, the last of
    each row and column ragged, and 2 (INT8) to 33 (BF16) drained chunks of k per tile, so that stages,
    accumulator buffers and their phases go on from one tile to the next.  Rounding and products left
    out as in the test of the odd extents, BF16 slices with units of 2^(2 - 8 n) of the row maximum."""
    torch = pytest.importorskip("torch")
    o, v = 49, 129
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=[v], occ=[o])
        x, y, z = (ctx.tensor(n, *sh, plain=True) for n, sh in
                   (("x", ((0, 2), (2, 0))), ("y", ((2, 0), (0, 2))), ("z", ((0, 2), (0, 2)))))
        g = torch.Generator(device="cuda").manual_seed(slices)
        for t in (x, y):
            alpha = t.spin_cases()[0]
            t.write_block(alpha, torch.rand(t.block_shape(alpha), generator=g, device="cuda", dtype=torch.float64)
                          .sub_(0.5).cpu().numpy())
        out = {}
        for p, n in (("fp64", 0), (precision, slices)):
            ctx.set_precision(p, slices=n)
            ctx.set_split_routing("all")
            ctx.contract(1.0, x, "mnef", y, "efij", 0.0, z, "mnij")
            out[p] = z.read_block(z.spin_cases()[0])
        ctx.set_precision("fp64")
    K, sd = v * v, 12**-0.5
    if precision == "split_i8":
        unit = 0.5 / 127 / 254.0 ** (slices - 1)
        left = (slices - 1) ** 0.5 * (127 / 3**0.5) ** 2 * 254.0**-slices * (0.5 / 127) ** 2
    else:
        # 2^(e-6) 2^(-8 (n-1)) with 2^e <= max; FP32 sums of the lower products: 2^-24 of sums below
        # 2^-8 K max^2, once per product of a chunk
        unit = 0.25 * 2.0 ** (-6 - 8 * (slices - 1)) * 2
        left = (slices - 1) ** 0.5 * (2.0**8 / 12**0.5) ** 2 * 2.0 ** (-8 * slices) * 2.0**-14 * 4 + 2.0**-31
    bound = 7 * K**0.5 * (2 * unit * sd / 12**0.5 + left)
    err = np.abs(out[precision] - out["fp64"]).max()
    assert 0 < err <= bound, (err, bound)


def test_first_slices_of_a_deeper_slicing_are_unbiased():
    """A constant operand sliced four times serves a contraction with three slices.  Every element here
    sits half a unit of the third slice beside a multiple of it: rounded all to one side, the K
    contributions to an element add up to K / 2 units; rounded independently, to sqrt(K) / 2."""
    o, v = 3, 24
    rng = np.random.default_rng(4)
    eps, B, *_ = A.synth_problem(3, o, v)
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=[v], occ=[o])
        H = ctx.rhf_hamiltonian_from_factor(B, eps)
        s = ctx.solver(H)                       # the integrals are its constants: their slices are kept
        V = H["VABCD"]
        alpha = V.spin_cases()[0]
        n = 254 * rng.integers(-127 * 254**2 + 1, 127 * 254**2, size=(v, v, v, v)) - 127
        n[:, :, 0, 0] = 127 * 254**3            # the row maximum, a multiple
        x = n / (127 * 254.0**3)
        V.write_block(alpha, x)
        t = ctx.tensor("t", (2, 0), (0, 2), plain=True)
        t.fill(1.0)                             # one digit: the other operand is exact
        z = ctx.tensor("z", (2, 0), (0, 2), plain=True)
        ctx.set_split_routing("all")
        err = {}
        for slices in (4, 3):
            ctx.set_precision("split_i8", slices=slices)
            ctx.contract(1.0, V, "abef", t, "efij", 0.0, z, "abij")
            err[slices] = np.abs(z.to_full() - x.sum((2, 3))[:, :, None, None]).max()
        ctx.set_precision("fp64")
        s.close()
    K, unit = v * v, 1 / 127 / 254.0**2
    assert err[4] <= 6 * K**0.5 * unit / 254
    assert 0.01 * unit < err[3] <= 5 * 0.5 * K**0.5 * unit, (err[3] / unit, K)


def test_a_small_product_gets_in_beside_a_large_one():
    """A split product of 40000 tiles on a stream of low priority gives its SMs back as it goes: a CTA
    takes 10 of an SM's 270 tiles.  A small split product on a stream of high priority (five kernels, each
    of which may wait for such a CTA), queued when 0.4 of the large one's time has gone, is there
    within 0.3 of it; one that kept its SMs held the small one up to its end, 0.6 later."""
    torch = pytest.importorskip("torch")
    streams = [torch.cuda.Stream(priority=p) for p in (0, -5)]
    ctxs = [A.Context(0, s.cuda_stream) for s in streams]
    try:
        runs = []
        for ctx, (o, v) in zip(ctxs, [(160, 64), (16, 64)]):
            ctx.set_spaces(vrt=[v], occ=[o])
            ctx.set_precision("split_i8", slices=4)
            ctx.set_split_routing("all")
            x, y, z = (ctx.tensor(n, *sh, plain=True) for n, sh in
                       (("x", ((0, 2), (2, 0))), ("y", ((2, 0), (0, 2))), ("z", ((0, 2), (0, 2)))))
            runs.append(lambda ctx=ctx, x=x, y=y, z=z: ctx.contract(1.0, x, "mnef", y, "efij", 0.0, z, "mnij"))
        large, small = runs
        wait = lambda: [ctx.synchronize() for ctx in ctxs]
        for _ in range(3):
            large(), small(), wait()
        t0 = time.perf_counter()
        large(), wait()
        whole = time.perf_counter() - t0
        late = []
        for _ in range(5):
            large()
            time.sleep(0.4 * whole)
            t0 = time.perf_counter()
            small(), ctxs[1].synchronize()
            late.append(time.perf_counter() - t0)
            wait()
        assert sorted(late)[2] < 0.3 * whole, (late, whole)
    finally:
        for ctx in ctxs:
            ctx.close()
