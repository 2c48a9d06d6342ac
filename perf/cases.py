"""Performance cases of the CCSD engine: what its users run, over the range of sizes they run.

Every case enters through the public binding: statements on a context (the way a program that keeps
its own iteration uses the engine), the solvers, the DIIS object, and whole programs from a
three-index factor to converged amplitudes.  Inputs are closed-shell problems of the shape the
synthetic benchmark uses (o occupied and v virtual spatial orbitals, v = 4 to 9 times o, a factor of
3 (o + v) auxiliary functions); results come back in page-locked host buffers through the C entry
point that reads a block, as a program that keeps its results would fetch them.
"""
import itertools
import math
import random

import numpy as np
import torch

import aquarius_b200 as A

# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------


def listed():
    return [
        # the smallest calls: the 44 statements of one residual of a water molecule in cc-pVDZ (the
        # known-answer test), where every launch and every call on the host counts
        {"name": "residual-fp64-o5v19", "kind": "residual", "o": 5, "v": 19, "nirrep": 1, "precision": "fp64"},
        # an ordinary molecule with odd sizes, native FP64 (the default precision)
        {"name": "residual-fp64-o13v94", "kind": "residual", "o": 13, "v": 94, "nirrep": 1, "precision": "fp64"},
        # point-group symmetry (D2h): thousands of small ragged blocks in each statement
        {"name": "residual-fp64-d2h-o16v96", "kind": "residual", "o": 16, "v": 96, "nirrep": 8, "precision": "fp64"},
        # a caller's own iteration on the tensor cores (4 INT8 slices), no operand kept sliced
        {"name": "residual-i8-o20v144", "kind": "residual", "o": 20, "v": 144, "nirrep": 1, "precision": "split_i8"},
        # the particle ladder alone in FP64: the largest single product
        {"name": "ladder-fp64-o20v160", "kind": "ladder", "o": 20, "v": 160, "nirrep": 1, "precision": "fp64"},
        # the one-body intermediates and the T1 residual: long thin products that stream <am||ef>
        {"name": "singles-fp64-o20v160", "kind": "singles", "o": 20, "v": 160, "nirrep": 1, "precision": "fp64"},
        # the tail of a caller's own iteration: denominators, update, DIIS over 8 pairs, energy
        {"name": "update-o20v144", "kind": "update", "o": 20, "v": 144, "nirrep": 1, "precision": "fp64"},
        # a small solve with the iteration replayed as a graph (the serving mix's small end)
        {"name": "solve-fp64-o9v60", "kind": "solve", "o": 9, "v": 60, "nirrep": 1, "precision": "fp64"},
        # iterations of a solver at the benchmark's scale, INT8 slices, constants kept sliced: the
        # headline metric, largest size
        {"name": "iterate-i8-o24v184", "kind": "iterate", "o": 24, "v": 184, "nirrep": 1, "precision": "split_i8"},
        # the same of a symmetry-blocked problem of the serving mix, replayed as a graph
        {"name": "iterate-i8-d2h-o24v180", "kind": "iterate", "o": 24, "v": 180, "nirrep": 8, "precision": "split_i8"},
        # closed-shell spin-adapted CCSD, native FP64
        {"name": "iterate-rhf-fp64-o16v128", "kind": "rhf", "o": 16, "v": 128, "nirrep": 1, "precision": "fp64"},
        # the whole program, host factor to converged amplitudes (3 then 4 INT8 slices, as served)
        {"name": "program-i8-o14v112", "kind": "program", "o": 14, "v": 112, "nirrep": 1, "precision": "split_i8"},
    ]


def draw(rng):
    kind = rng.choice(["residual", "residual", "residual", "solve", "iterate", "iterate", "rhf", "ladder", "singles",
                       "update", "program"])
    nirrep = rng.choice([1, 1, 2, 4, 8]) if kind in ("residual", "iterate") else 1
    precision = rng.choice(["fp64", "fp64", "split_i8", "split"]) if kind in ("residual", "solve", "iterate", "program") else "fp64"
    low = {"ladder": 9, "singles": 9, "update": 7}.get(kind, 4)
    high = {"solve": 13, "program": 13}.get(kind, 18)
    if nirrep > 1:
        low, high = 9, 20
    o = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    v = int(round(o * rng.uniform(4.0, 8.0)))
    return {"kind": kind, "o": o, "v": max(v, nirrep), "nirrep": nirrep, "precision": precision}


# a solve of these problems to 1e-9 takes about this many iterations
ITERATIONS = 14
# iterations between two looks at the amplitudes, in the cases that keep a solver
STEPS = 4


def work(case):
    o, v, h = case["o"], case["v"], case["nirrep"]
    kind = case["kind"]
    # stored elements of the spin-orbital blocks that an iteration reads (pairs of <ab||ef> once)
    vvvv = v**4 + 2 * (v * (v - 1) // 2) ** 2
    t2 = 3 * v * v * o * o
    rest = 6 * v**3 * o + 9 * v * v * o * o + 6 * v * o**3 + 3 * o**4
    ladder = 2 * v**4 * o * o + 4 * (v * (v - 1) // 2) ** 2 * (o * (o - 1) // 2)
    rings = 24 * 2 * (o * v) ** 3
    if kind == "ladder":
        return {"bytes": 8 * (vvvv + 2 * t2), "flops": ladder}
    if kind == "singles":
        return {"bytes": 8 * (6 * v**3 * o + 3 * t2 + 9 * v * v * o * o), "flops": 20 * 2 * v**3 * o * o}
    if kind == "update":
        # Z and T read and written, the ring's other seven pairs read, two pairs written back
        return {"bytes": 8 * t2 * (4 + 14 + 4), "flops": 2 * t2 * 24}
    if kind == "rhf":
        return {"bytes": 8 * (v**4 + 2 * v**3 * o + 6 * v * v * o * o), "flops": STEPS * (2 * v**4 * o * o + 16 * (o * v) ** 3)}
    byt, fl = 8 * (vvvv + rest + 2 * t2) / h, (ladder + rings) / (h * h)
    if kind == "residual":
        return {"bytes": byt, "flops": fl}
    if kind == "program":
        n = o + v
        return {"bytes": byt + 8 * 3 * n**3, "flops": ITERATIONS * fl + 2 * 3 * n * vvvv}
    return {"bytes": byt, "flops": (STEPS if kind == "iterate" else ITERATIONS) * fl}


def tolerance(case):
    """FP64 statements: sums in another order.  Split statements: the slices' truncation.  Converged
    amplitudes: two solves of one problem that each stop at a residual of 1e-9."""
    if case["kind"] in ("solve", "program"):
        return {"rel": 5e-7, "max": 2e-5}
    if case["kind"] == "iterate" and case["precision"] != "fp64":
        return {"rel": 4e-7, "max": 2e-5}   # the residual's largest element carries the slices' truncation
    if case["precision"] == "split_i8":
        return {"rel": 3e-8, "max": 1e-6}
    if case["precision"] == "split":
        return {"rel": 1e-7, "max": 4e-6}
    return {"rel": 1e-12, "max": 4e-11}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------


def irrep_counts(total, nirrep, salt):
    """An uneven split of `total` orbitals over the irreps, at least one in each, fixed by the sizes."""
    if nirrep == 1:
        return [total]
    r = random.Random(1000 * total + 10 * nirrep + salt)
    share = [r.gammavariate(1.5, 1.0) for _ in range(nirrep)]
    counts = [1 + int((total - nirrep) * s / sum(share)) for s in share]
    for k in range(total - sum(counts)):
        counts[k % nirrep] += 1
    return counts


def problem(case, seed):
    """(occ, vrt, aux counts, eps, B) with the benchmark generator's distributions; B on the GPU."""
    o, v, h = case["o"], case["v"], case["nirrep"]
    n, naux = o + v, 3 * (o + v)
    occ, vrt, aux = irrep_counts(o, h, 1), irrep_counts(v, h, 2), irrep_counts(naux, h, 3)
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    eo = -1.2 + 0.8 * u[:o]
    ev = 0.3 + 3.7 * u[o:]
    at = 0
    for c in occ:
        eo[at:at + c] = eo[at:at + c].sort().values
        at += c
    at = 0
    for c in vrt:
        ev[at:at + c] = ev[at:at + c].sort().values
        at += c
    eps = torch.cat([eo, ev])
    B = torch.randn(naux, n, n, generator=g, device="cuda", dtype=torch.float64)
    p = torch.arange(n, device="cuda", dtype=torch.float64)
    B *= (0.25 / math.sqrt(naux)) * torch.exp(-(p[None, :] - p[:, None]).abs() / n)
    B = B.triu()
    B += B.triu(1).transpose(1, 2).clone()
    if h > 1:
        orb = torch.tensor(labels(occ) + labels(vrt), device="cuda")
        B *= ((orb[:, None] ^ orb[None, :])[None] == torch.tensor(labels(aux), device="cuda")[:, None, None])
    return occ, vrt, aux, eps, B


def labels(counts):
    return [h for h, c in enumerate(counts) for _ in range(c)]


def singles_guess(case, seed, occ, vrt):
    """Spatial T1[a, i] of the size that a correlated singles vector has, symmetry kept."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 5)
    t = 0.02 * torch.randn(case["v"], case["o"], generator=g, device="cuda", dtype=torch.float64)
    if case["nirrep"] > 1:
        a, i = torch.tensor(labels(vrt), device="cuda"), torch.tensor(labels(occ), device="cuda")
        t *= a[:, None] == i[None, :]
    return t


def mixing(case, seed):
    """Sets of denominators that give the update case residual vectors of its own making."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 31337 + 3)
    return [(0.5 + torch.rand(case["v"], generator=g, device="cuda", dtype=torch.float64),
             0.5 + torch.rand(case["o"], generator=g, device="cuda", dtype=torch.float64)) for _ in range(9)]


# ---------------------------------------------------------------------------------------------
# results: every block of a tensor, case by case, in one page-locked buffer
# ---------------------------------------------------------------------------------------------


def symmetric(nirrep, ndim):
    for irr in itertools.product(range(nirrep), repeat=ndim):
        x = 0
        for h in irr:
            x ^= h
        if x == 0:
            yield irr


class Reader:
    def __init__(self, ctx, tensor):
        self.at, n = [], 0
        for alpha in tensor.spin_cases():
            for irr in symmetric(ctx.nirrep, tensor.ndim):
                size = math.prod(tensor.block_shape(alpha, irr))
                if size:
                    self.at.append((np.array(alpha, np.int32), np.array(irr, np.int32), n))
                    n += size
        self.out = torch.empty(n, dtype=torch.float64, pin_memory=True)

    def read(self, ctx, tensor):
        lib, base = A.lib(), self.out.data_ptr()
        for alpha, irr, at in self.at:
            code = lib.ccsd_tensor_read_block(ctx.c, tensor.h, alpha.ctypes.data, irr.ctypes.data, base + 8 * at)
            if code:
                raise A.CcsdError(code, (lib.ccsd_last_error(ctx.c) or b"").decode())
        return self.out


class State:
    """What the program keeps: the context and what lives on it.  The context goes last."""

    ctx = solver = diis = None

    def __del__(self):
        for x in (self.solver, self.diis, self.ctx):
            if x is not None:
                x.close()


SOLVER = {"fp64": {}, "split_i8": {"slices": 3, "refine_tol": 1e-5}, "split": {"slices": 3, "refine_tol": 1e-6}}


def prepare(case, seed):
    kind = case["kind"]
    occ, vrt, aux, eps, B = problem(case, seed)
    s = State()
    s.case, s.occ, s.vrt = case, occ, vrt
    s.aux = aux if case["nirrep"] > 1 else None
    host = torch.empty(B.shape, dtype=torch.float64, pin_memory=True)
    host.copy_(B)
    s.B, s.eps = host.numpy(), eps.cpu().numpy()
    del B
    if kind == "program":
        # the sizes are known, so the result buffers are there before the solve
        with A.Context(0) as ctx:
            ctx.set_spaces(vrt=vrt, occ=occ)
            s.read1 = Reader(ctx, ctx.tensor("t1", (1, 0), (0, 1)))
            s.read2 = Reader(ctx, ctx.tensor("t2", (2, 0), (0, 2)))
        return s
    s.ctx = ctx = A.Context(0)
    ctx.set_spaces(vrt=vrt, occ=occ)
    if kind == "rhf":
        s.H = ctx.rhf_hamiltonian_from_factor(s.B, s.eps, s.aux)
        t1, t2 = ctx.tensor("t1", (1, 0), (0, 1), plain=True), ctx.tensor("t2", (2, 0), (0, 2), plain=True)
    else:
        s.H = ctx.hamiltonian_from_factor(s.B, s.eps, s.aux)
        t1, t2 = ctx.tensor("T1", (1, 0), (0, 1)), ctx.tensor("T2", (2, 0), (0, 2))
    s.B = None
    s.read1, s.read2 = Reader(ctx, t1), Reader(ctx, t2)
    if kind in ("rhf", "iterate"):
        # a solver and the guess that every pass starts from; DIIS keeps its ring and waits
        p = case["precision"]
        s.solver = ctx.solver(s.H, diis_order=8, diis_start=1 << 30, precision=p, slices=0 if p == "fp64" else 4,
                              use_graph=case["o"] < 12 or case["nirrep"] > 1)
        s.guess1, s.guess2 = t1, t2
        t1["ai"], t2["abij"] = s.solver.T1["ai"], s.solver.T2["abij"]
        return s
    if kind == "solve":
        return s
    if case["precision"] != "fp64":
        ctx.set_precision(case["precision"], 4)
    o = case["o"]
    s.T1, s.T2, s.Z1, s.Z2 = t1, t2, ctx.tensor("Z1", (1, 0), (0, 1)), ctx.tensor("Z2", (2, 0), (0, 2))
    t1["ai"] = s.H["fAI"]["ai"]
    t2["abij"] = s.H["VABIJ"]["abij"]
    ctx.weight(t2, -s.eps[o:], s.eps[:o])
    if kind == "update":
        prepare_update(s, case, seed)
        return s
    guess, at_a, at_i = singles_guess(case, seed, occ, vrt).cpu().numpy(), 0, 0
    for h, (na, ni) in enumerate(zip(vrt, occ)):
        for alpha in t1.spin_cases():
            t1.write_block(alpha, guess[at_a:at_a + na, at_i:at_i + ni], [h, h])
        at_a, at_i = at_a + na, at_i + ni
    s.Tau = ctx.tensor("Tau", (2, 0), (0, 2))
    make_tau(s)
    s.F = {n: ctx.tensor(n, *A.H_SHAPES[m]) for n, m in
           (("FME", "fME"), ("FMI", "fMI"), ("FAE", "fAE"))}
    if kind == "residual":
        s.F.update({n: ctx.tensor(n, *A.H_SHAPES[m]) for n, m in
                    (("WMNIJ", "VMNIJ"), ("WMNEJ", "VMNEJ"), ("WAMIJ", "VAMIJ"), ("WAMEI", "VAMEI"))})
    if kind == "singles":
        s.readf = [Reader(ctx, s.F[n]) for n in ("FMI", "FAE")]
    return s


def prepare_update(s, case, seed):
    """Nine amplitude pairs and residuals in hand, and a DIIS ring that is full, as in mid-solve."""
    ctx = s.ctx
    s.sets = []
    for k, (dv, do) in enumerate(mixing(case, seed)):
        z1, z2 = ctx.tensor("z1_%d" % k, (1, 0), (0, 1)), ctx.tensor("z2_%d" % k, (2, 0), (0, 2))
        z2["abij"] = s.H["VABIJ"]["abij"]
        ctx.weight(z2, dv.cpu().numpy(), do.cpu().numpy())
        g = singles_guess(case, 16 * int(seed) + k, s.occ, s.vrt).cpu().numpy()
        for alpha in z1.spin_cases():
            z1.write_block(alpha, g, [0, 0])
        s.sets.append((z1, z2))
    s.base1, s.base2 = ctx.tensor("b1", (1, 0), (0, 1)), ctx.tensor("b2", (2, 0), (0, 2))
    s.base1["ai"], s.base2["abij"] = s.T1["ai"], s.T2["abij"]
    s.diis = ctx.diis(order=8)
    s.count = 0
    for _ in range(8):
        step_update(s)


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------


def run(s):
    return {"residual": run_residual, "ladder": run_ladder, "singles": run_singles, "update": run_update,
            "solve": run_solve, "rhf": run_iterate, "iterate": run_iterate, "program": run_program}[s.case["kind"]](s)


def make_tau(s):
    s.Tau["abij"] = s.T2["abij"]
    s.Tau["abij"] += 0.5 * s.T1["ai"] * s.T1["bj"]


def run_residual(s):
    H, T1, T2, Z1, Z2, Tau = s.H, s.T1, s.T2, s.Z1, s.Z2, s.Tau
    FME, FMI, FAE = s.F["FME"], s.F["FMI"], s.F["FAE"]
    WMNIJ, WMNEJ, WAMIJ, WAMEI = s.F["WMNIJ"], s.F["WMNEJ"], s.F["WAMIJ"], s.F["WAMEI"]
    make_tau(s)
    FME["me"] = H["fME"]["me"]
    FME["me"] += H["VMNEF"]["mnef"] * T1["fn"]
    FMI["mi"] = H["fMI"]["mi"]
    FMI["mi"] += 0.5 * H["VMNEF"]["mnef"] * T2["efin"]
    FMI["mi"] += FME["me"] * T1["ei"]
    FMI["mi"] += H["VMNEJ"]["nmfi"] * T1["fn"]
    FAE["ae"] = H["fAE"]["ae"]
    FAE["ae"] -= 0.5 * H["VMNEF"]["mnef"] * T2["afmn"]
    FAE["ae"] -= FME["me"] * T1["am"]
    FAE["ae"] += H["VAMEF"]["amef"] * T1["fm"]
    WMNIJ["mnij"] = H["VMNIJ"]["mnij"]
    WMNIJ["mnij"] += 0.5 * H["VMNEF"]["mnef"] * Tau["efij"]
    WMNIJ["mnij"] += H["VMNEJ"]["mnej"] * T1["ei"]
    WMNEJ["mnej"] = H["VMNEJ"]["mnej"]
    WMNEJ["mnej"] += H["VMNEF"]["mnef"] * T1["fj"]
    WAMIJ["amij"] = H["VAMIJ"]["amij"]
    WAMIJ["amij"] += 0.5 * H["VAMEF"]["amef"] * Tau["efij"]
    WAMIJ["amij"] += H["VAMEI"]["amej"] * T1["ei"]
    WAMEI["amei"] = H["VAMEI"]["amei"]
    WAMEI["amei"] += 0.5 * H["VMNEF"]["mnef"] * T2["afni"]
    WAMEI["amei"] += H["VAMEF"]["amef"] * T1["fi"]
    WAMEI["amei"] -= WMNEJ["nmei"] * T1["an"]
    Z1["ai"] = H["fAI"]["ai"]
    Z1["ai"] += H["fAE"]["ae"] * T1["ei"]
    Z1["ai"] -= FMI["mi"] * T1["am"]
    Z1["ai"] -= H["VAMEI"]["amei"] * T1["em"]
    Z1["ai"] += FME["me"] * T2["aeim"]
    Z1["ai"] += 0.5 * H["VAMEF"]["amef"] * Tau["efim"]
    Z1["ai"] -= 0.5 * WMNEJ["mnei"] * T2["eamn"]
    Z2["abij"] = H["VABIJ"]["abij"]
    Z2["abij"] += H["VABEJ"]["abej"] * T1["ei"]
    Z2["abij"] -= WAMIJ["amij"] * T1["bm"]
    Z2["abij"] += FAE["ae"] * T2["ebij"]
    Z2["abij"] -= FMI["mi"] * T2["abmj"]
    Z2["abij"] += 0.5 * H["VABEF"]["abef"] * Tau["efij"]
    Z2["abij"] += 0.5 * WMNIJ["mnij"] * Tau["abmn"]
    Z2["abij"] += WAMEI["amei"] * T2["ebjm"]
    return {"Z1": s.read1.read(s.ctx, Z1), "Z2": s.read2.read(s.ctx, Z2)}


def run_ladder(s):
    s.Z2["abij"] = 0.5 * s.H["VABEF"]["abef"] * s.Tau["efij"]
    return {"Z2": s.read2.read(s.ctx, s.Z2)}


def run_singles(s):
    H, T1, T2, Tau, Z1 = s.H, s.T1, s.T2, s.Tau, s.Z1
    FMI, FAE = s.F["FMI"], s.F["FAE"]
    FMI["mi"] = H["fMI"]["mi"]
    FMI["mi"] += 0.5 * H["VMNEF"]["mnef"] * T2["efin"]
    FMI["mi"] += H["VMNEJ"]["nmfi"] * T1["fn"]
    FAE["ae"] = H["fAE"]["ae"]
    FAE["ae"] -= 0.5 * H["VMNEF"]["mnef"] * T2["afmn"]
    FAE["ae"] += H["VAMEF"]["amef"] * T1["fm"]
    Z1["ai"] = H["fAI"]["ai"]
    Z1["ai"] += FAE["ae"] * T1["ei"]
    Z1["ai"] -= FMI["mi"] * T1["am"]
    Z1["ai"] -= H["VAMEI"]["amei"] * T1["em"]
    Z1["ai"] += 0.5 * H["VAMEF"]["amef"] * Tau["efim"]
    Z1["ai"] -= 0.5 * H["VMNEJ"]["mnei"] * T2["eamn"]
    return {"Z1": s.read1.read(s.ctx, Z1), "FMI": s.readf[0].read(s.ctx, FMI), "FAE": s.readf[1].read(s.ctx, FAE)}


def step_update(s):
    ctx, T1, T2, Z1, Z2, H, o = s.ctx, s.T1, s.T2, s.Z1, s.Z2, s.H, s.case["o"]
    z1, z2 = s.sets[s.count % len(s.sets)]
    s.count += 1
    Z1["ai"], Z2["abij"] = z1["ai"], z2["abij"]
    ctx.weight(Z1, -s.eps[o:], s.eps[:o])
    ctx.weight(Z2, -s.eps[o:], s.eps[:o])
    T1["ai"], T2["abij"] = s.base1["ai"], s.base2["abij"]
    T1["ai"] += Z1["ai"]
    T2["abij"] += Z2["abij"]
    residual = max(Z1.norm(0), Z2.norm(0))
    s.diis.extrapolate([T1, T2], [Z1, Z2])
    energy = ctx.dot(H["fAI"], "ai", T1, "ai") + 0.25 * ctx.dot(H["VABIJ"], "abij", T2, "abij")
    return energy, residual


def run_update(s):
    energy, residual = step_update(s)
    return {"energy": energy, "residual": residual, "T1": s.read1.read(s.ctx, s.T1), "T2": s.read2.read(s.ctx, s.T2)}


def run_iterate(s):
    T1, T2 = s.solver.T1, s.solver.T2
    T1["ai"], T2["abij"] = s.guess1["ai"], s.guess2["abij"]
    for _ in range(STEPS):
        energy, residual = s.solver.iterate()
    return {"energy": energy, "residual": residual, "T1": s.read1.read(s.ctx, T1), "T2": s.read2.read(s.ctx, T2)}


def solve(s, ctx, H, **kw):
    p = s.case["precision"]
    solver = ctx.solver(H, conv_tol=1e-9, max_iter=60, diis_order=8, precision=p, **SOLVER[p], **kw)
    try:
        energy, _, _ = solver.run()
        return {"energy": energy, "T1": s.read1.read(ctx, solver.T1), "T2": s.read2.read(ctx, solver.T2)}
    finally:
        solver.close()


def run_solve(s):
    return solve(s, s.ctx, s.H, use_graph=s.case["o"] < 12)


def run_program(s):
    with A.Context(0) as ctx:
        ctx.set_spaces(vrt=s.vrt, occ=s.occ)
        H = ctx.hamiltonian_from_factor(s.B, s.eps, s.aux)
        return solve(s, ctx, H)


# ---------------------------------------------------------------------------------------------
# the same in 64 bits with plain torch: closed-shell CCSD over spatial orbitals, the singles folded
# into the integrals (Koch, Christiansen, Kobayashi, Jorgensen and Helgaker, 1994)
# ---------------------------------------------------------------------------------------------


def chem(L, R, p, q, r, s):
    """(pq|rs) from the dressed factors, as [p, q, r, s]."""
    return torch.einsum("Ppq,Prs->pqrs", L[:, p, q], R[:, r, s])


class Spatial:
    def __init__(self, case, seed):
        self.occ, self.vrt, _, self.eps, self.B = problem(case, seed)
        self.o, self.n = case["o"], case["o"] + case["v"]
        self.O, self.V = slice(0, self.o), slice(self.o, self.n)
        O, V, B = self.O, self.V, self.B
        # <ab|ij> = (ai|bj) as [a, b, i, j]
        self.abij = torch.einsum("Pai,Pbj->abij", B[:, V, O], B[:, V, O])
        # h of the canonical orbitals with these energies
        J = torch.einsum("Ppq,P->pq", B, B[:, range(self.o), range(self.o)].sum(1))
        K = torch.einsum("Ppk,Pkq->pq", B[:, :, O], B[:, O, :])
        self.h = torch.diag(self.eps) - 2 * J + K

    def ladder(self, B, tau, V):
        """sum_cd (ac|bd) tau[c, d, i, j], a few a at a time."""
        v = self.n - self.o
        out = torch.empty_like(tau)
        flat = tau.reshape(v * v, -1)
        step = max(1, int(2e9 // (8 * v**3)))
        for a in range(0, v, step):
            aa = slice(self.o + a, self.o + min(v, a + step))
            w = torch.einsum("Pac,Pbd->abcd", B[:, aa, V], B[:, V, V])
            out[a:a + step] = (w.reshape(-1, v * v) @ flat).reshape(w.shape[0], *tau.shape[1:])
        return out

    def residual(self, t1, t2):
        """The full (unweighted) residuals [a, i] and [a, b, i, j] at these amplitudes."""
        o, n, O, V = self.o, self.n, self.O, self.V
        eye = torch.eye(n, dtype=torch.float64, device="cuda")
        t = torch.zeros_like(eye)
        t[V, O] = t1
        X, Y = eye - t, eye + t.T
        B = torch.einsum("pr,Prs,qs->Ppq", X, self.B, Y)
        h = X @ self.h @ Y.T
        F = h + 2 * torch.einsum("Ppq,P->pq", B, B[:, range(o), range(o)].sum(1)) - torch.einsum("Ppk,Pkq->pq", B[:, :, O], B[:, O, :])
        ii = torch.einsum
        u = 2 * t2 - t2.transpose(2, 3)
        ovov = chem(B, B, O, V, O, V)                                # (kc|ld)
        G = 2 * ovov - ovov.transpose(1, 3)                          # L_kcld
        x1 = ii("Pkc,cdki->Pdi", B[:, O, V], u)                      # sum_kc (.|kc) u[c, d, k, i]
        r1 = F[V, O] + ii("kc,acik->ai", F[O, V], u) + ii("Pad,Pdi->ai", B[:, V, V], x1) - ii("Pki,Pak->ai", B[:, O, O], x1)
        r2 = self.ladder(B, t2, V) + ii("Pai,Pbj->abij", B[:, V, O], B[:, V, O])
        w = chem(B, B, O, O, O, O) + ii("cdij,kcld->kilj", t2, ovov)  # (ki|lj)
        r2 += ii("abkl,kilj->abij", t2, w)
        # C: -(1/2 + P_ij) sum_ck t[b, c, k, j] ((ki|ac) - 1/2 sum_dl t[a, d, l, i] (kd|lc))
        c = chem(B, B, O, O, V, V) - 0.5 * ii("adli,kdlc->kiac", t2, ovov)
        y = ii("bckj,kiac->abij", t2, c)
        half = -0.5 * y - y.transpose(2, 3)
        # D: 1/2 sum_ck u[b, c, j, k] (L_aikc + 1/2 sum_dl u[a, d, i, l] L_ldkc)
        d = 2 * chem(B, B, V, O, O, V) - ii("Pac,Pki->aikc", B[:, V, V], B[:, O, O]) + 0.5 * ii("adil,ldkc->aikc", u, G)
        half += 0.5 * ii("bcjk,aikc->abij", u, d)
        # E: the dressed Fock matrices
        fbc = F[V, V] - ii("bdkl,ldkc->bc", u, ovov)
        fkj = F[O, O] + ii("cdlj,kdlc->kj", u, ovov)
        half += ii("acij,bc->abij", t2, fbc) - ii("abik,kj->abij", t2, fkj)
        return r1, r2 + half + half.transpose(0, 1).transpose(2, 3)

    def denominators(self):
        e, o = self.eps, self.o
        d1 = e[None, :o] - e[o:, None]
        return d1, d1[:, None, :, None] + d1[None, :, None, :]

    def energy(self, t1, t2):
        tau = t2 + t1[:, None, :, None] * t1[None, :, None, :]
        return float(((2 * self.abij - self.abij.transpose(2, 3)) * tau).sum())

    def solve(self):
        d1, d2 = self.denominators()
        t1, t2 = torch.zeros_like(d1), self.abij / d2
        xs, es = [], []
        for _ in range(80):
            r1, r2 = self.residual(t1, t2)
            z1, z2 = r1 / d1, r2 / d2
            t1, t2 = t1 + z1, t2 + z2
            if max(z1.abs().max(), z2.abs().max()) < 2e-13:
                break
            xs, es = ([(t1, t2)] + xs)[:6], ([(z1, z2)] + es)[:6]
            c = diis_weights([[float((p[0] * q[0]).sum() + (p[1] * q[1]).sum()) for q in es] for p in es])
            t1 = sum(w * x[0] for w, x in zip(c, xs))
            t2 = sum(w * x[1] for w, x in zip(c, xs))
        return self.energy(t1, t2), t1, t2

    # the block layout: spin cases by their alpha count, then irreps, first index fastest
    def starts(self, counts):
        return list(itertools.accumulate([0] + counts))

    def flat1(self, x, rows, cols):
        a, i, parts = self.starts(rows), self.starts(cols), []
        for _ in range(2):
            parts += [x[a[h]:a[h + 1], i[h]:i[h + 1]].T.reshape(-1) for h in range(len(rows))]
        return torch.cat(parts).cpu()

    def flat2(self, ab, plain=False):
        """All spin cases (bb, ab, aa) of a closed-shell [a, b, i, j] array; `plain`: the one array."""
        a, i, parts = self.starts(self.vrt), self.starts(self.occ), []
        same = ab - ab.transpose(0, 1)
        for x in ([ab] if plain else [same, ab, same]):
            for h in symmetric(len(self.vrt), 4):
                b = x[a[h[0]]:a[h[0] + 1], a[h[1]]:a[h[1] + 1], i[h[2]]:i[h[2] + 1], i[h[3]]:i[h[3] + 1]]
                parts.append(b.permute(3, 2, 1, 0).reshape(-1))
        return torch.cat([p.cpu() for p in parts])


def diis_weights(e):
    m = len(e)
    a = np.zeros((m + 1, m + 1))
    scale = max(abs(e[k][k]) for k in range(m)) or 1.0
    a[:m, :m] = np.array(e) / scale
    a[m, :m] = a[:m, m] = -1.0
    rhs = np.zeros(m + 1)
    rhs[m] = -1.0
    return np.linalg.lstsq(a, rhs, rcond=1e-15)[0][:m]


def exact(case, seed):
    x, kind = Spatial(case, seed), case["kind"]
    if kind in ("solve", "program"):
        energy, t1, t2 = x.solve()
        return {"energy": energy, "T1": x.flat1(t1, x.vrt, x.occ), "T2": x.flat2(t2)}
    if kind in ("rhf", "iterate"):
        return exact_iterate(x, kind == "rhf")
    if kind == "update":
        return exact_update(x, case, seed)
    t2 = x.abij / x.denominators()[1]
    t1 = singles_guess(case, seed, x.occ, x.vrt)
    if kind == "residual":
        r1, r2 = x.residual(t1, t2)
        return {"Z1": x.flat1(r1, x.vrt, x.occ), "Z2": x.flat2(r2)}
    tau = t2 + t1[:, None, :, None] * t1[None, :, None, :]
    if kind == "ladder":
        return {"Z2": x.flat2(x.ladder(x.B, tau, x.V))}
    return exact_singles(x, t1, t2, tau)


def exact_iterate(x, plain):
    d1, d2 = x.denominators()
    t1, t2 = torch.zeros_like(d1), x.abij / d2
    for _ in range(STEPS):
        r1, r2 = x.residual(t1, t2)
        t1, t2, residual = t1 + r1 / d1, t2 + r2 / d2, max(float((r1 / d1).abs().max()), float((r2 / d2).abs().max()))
    if not plain:   # the same-spin residual counts too
        z2 = r2 / d2
        residual = max(residual, float((z2 - z2.transpose(0, 1)).abs().max()))
    flat = x.flat1(t1, x.vrt, x.occ)
    half = flat[:flat.numel() // 2] if plain else flat
    return {"energy": x.energy(t1, t2), "residual": residual, "T1": half, "T2": x.flat2(t2, plain)}


def exact_singles(x, t1, t2, tau):
    B, O, V, ii = x.B, x.O, x.V, torch.einsum
    ov, vv, oo = B[:, O, V], B[:, V, V], B[:, O, O]
    u, ut = 2 * t2 - t2.transpose(2, 3), 2 * tau - tau.transpose(2, 3)
    Q = ii("Pnf,fn->P", ov, t1)
    y = ii("Pnf,efin->Pei", ov, u)                                   # <mn|ef> = (me|nf)
    fmi = torch.diag(x.eps[O]) + ii("Pme,Pei->mi", ov, y) + 2 * ii("Pmi,P->mi", oo, Q) - ii("Pni,Pmf,fn->mi", oo, ov, t1)
    fae = torch.diag(x.eps[V]) - ii("Pme,Pam->ae", ov, y) + 2 * ii("Pae,P->ae", vv, Q) - ii("Paf,Pme,fm->ae", vv, ov, t1)
    z1 = ii("ae,ei->ai", fae, t1) - ii("mi,am->ai", fmi, t1) + 2 * ii("Pia,P->ai", ov, Q) - ii("Pae,Pmi,em->ai", vv, oo, t1)
    z1 += ii("Pae,Pmf,efim->ai", vv, ov, ut) - ii("Pme,Pni,eamn->ai", ov, oo, u)
    return {"Z1": x.flat1(z1, x.vrt, x.occ), "FMI": x.flat1(fmi, x.occ, x.occ), "FAE": x.flat1(fae, x.vrt, x.vrt)}


def exact_update(x, case, seed):
    d1, d2 = x.denominators()
    t0 = x.abij / d2
    xs, es = [], []
    for k, (dv, do) in enumerate(mixing(case, seed)):
        z2 = x.abij / (dv[:, None, None, None] + dv[None, :, None, None] + do[None, None, :, None] + do[None, None, None, :]) / d2
        z1 = singles_guess(case, 16 * int(seed) + k, x.occ, x.vrt) / d1
        xs, es = ([(z1, t0 + z2)] + xs)[:8], ([(z1, z2)] + es)[:8]

    def dot(p, q):   # <T1, T1'> + 1/4 <T2, T2'> over spin orbitals
        same = p[1] - p[1].transpose(0, 1)
        return float(2 * (p[0] * q[0]).sum() + (p[1] * q[1]).sum() + 0.5 * (same * (q[1] - q[1].transpose(0, 1))).sum())

    c = diis_weights([[dot(p, q) for q in es] for p in es])
    t1, t2 = (sum(w * v[k] for w, v in zip(c, xs)) for k in (0, 1))
    energy = float(((2 * x.abij - x.abij.transpose(2, 3)) * t2).sum())
    residual = max(float(es[0][0].abs().max()), float(es[0][1].abs().max()), float((es[0][1] - es[0][1].transpose(0, 1)).abs().max()))
    return {"energy": energy, "residual": residual, "T1": x.flat1(t1, x.vrt, x.occ), "T2": x.flat2(t2)}
