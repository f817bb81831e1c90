"""The mixed-radix line passes (flups_b200/csrc/mix_dft_impl.cuh): every
operation against the FP64 oracle and the general line pass, in both kernel
classes, at lengths of two, three and four stages, odd sizes, partial tiles
and pairs without a partner; and, without a GPU, which passes take them and
that the cases meet every radix in every place."""
import numpy as np
import pytest

from gpu_helpers import from_user, make_solver, oracle_solve, rel_l2, to_user
from oracle.plans import CELL_CENTER, NODE_CENTER, CHAT_2, HEJ_2, HEJ_4
from flups_b200 import pyflups as pf

E, O, P, U = 0, 1, 3, 4


def _bc(s, lda=1):
    code = {"E": E, "O": O, "P": P, "U": U}
    return [[[code[s[2 * d]]] * lda, [code[s[2 * d + 1]]] * lda] for d in range(3)]


# (grid, lda, boundary conditions, centre, kernel)
CASES = [
    # free space, x r2c rows / y columns / fused z columns: 2 (9 x 2 ...), 3 and 4 stages, all radices
    ([33, 18, 20], 1, "UUUUUU", CELL_CENTER, HEJ_2),
    ([55, 26, 21], 1, "UUUUUU", CELL_CENTER, CHAT_2),
    ([50, 35, 49], 1, "UUUUUU", CELL_CENTER, HEJ_4),
    ([540, 9, 10], 1, "UUUUUU", CELL_CENTER, HEJ_2),
    ([10, 9, 1001], 1, "UUUUUU", CELL_CENTER, HEJ_2),
    ([14, 700, 9], 1, "UUUUUU", CELL_CENTER, HEJ_2),
    ([27, 25, 33], 1, "UUUUUU", NODE_CENTER, CHAT_2),
    # three components (pairs stay within a component)
    ([21, 15, 18], 3, "UUUUUU", CELL_CENTER, HEJ_2),
    # periodic: odd lengths, the node-centred copy, an odd outer extent of a folded fused pass, fused rows
    ([25, 27, 30], 1, "PPPPUU", CELL_CENTER, HEJ_2),
    ([24, 42, 25], 1, "PPUUPP", CELL_CENTER, HEJ_2),
    ([28, 16, 22], 1, "UUPPPP", NODE_CENTER, CHAT_2),
    ([121, 26, 23], 1, "PPPPUU", NODE_CENTER, HEJ_2),
    ([169, 15, 14], 1, "PPPPPP", CELL_CENTER, CHAT_2),
    # walls: types II / III (cell), I (node), IV and III / II (one even, one odd wall)
    ([45, 30, 21], 1, "EEOOPP", CELL_CENTER, CHAT_2),
    ([40, 44, 50], 1, "EOOEPP", CELL_CENTER, CHAT_2),
    ([31, 41, 29], 1, "EEOOUU", NODE_CENTER, HEJ_2),
    ([29, 22, 41], 1, "EOOEUU", NODE_CENTER, CHAT_2),
    # real last directions
    ([20, 18, 25], 1, "EEEEPP", CELL_CENTER, CHAT_2),
    ([22, 15, 21], 1, "OOEEOO", CELL_CENTER, CHAT_2),
    ([15, 20, 28], 1, "EEOOEE", CELL_CENTER, CHAT_2),
    ([20, 28, 36], 1, "OEEOOE", CELL_CENTER, CHAT_2),
    ([20, 28, 44], 1, "OEOOEO", CELL_CENTER, CHAT_2),
    ([19, 25, 31], 1, "EEOOEE", NODE_CENTER, CHAT_2),
    ([19, 25, 28], 1, "EEOOOO", NODE_CENTER, CHAT_2),
    ([19, 26, 31], 1, "OEEEEO", NODE_CENTER, CHAT_2),
    ([19, 26, 29], 1, "OEEEOE", NODE_CENTER, CHAT_2),
    # one wall, one open end
    ([30, 21, 25], 1, "EUUUUU", CELL_CENTER, HEJ_2),
    ([20, 18, 22], 1, "UUUUUO", CELL_CENTER, HEJ_2),
    ([21, 19, 26], 1, "UUUUOU", NODE_CENTER, HEJ_2),
    ([18, 20, 15], 1, "EUOUUE", CELL_CENTER, CHAT_2),
    # rows of the operations that x meets last or second only
    ([18, 20, 22], 1, "UUPPUU", CELL_CENTER, CHAT_2),
    ([22, 15, 20], 1, "UUEEOO", CELL_CENTER, CHAT_2),
    ([21, 20, 18], 1, "EUEEOO", CELL_CENTER, CHAT_2),
    ([22, 19, 15], 1, "EUOOEE", NODE_CENTER, CHAT_2),
]
# y and z lines of n points: (n, walls along x) with r2c / c2r columns along y, without c2c ones; fused columns
# along z.  First those of two stages of large radices (MIX_TWO), then radices of the other class that CASES miss
COLUMNS = [(n, True) for n in (75, 81, 98, 100, 108, 112, 125, 126, 135, 144, 160, 162, 200, 224, 264)] + \
    [(n, False) for n in (112, 126, 140, 168, 198, 210, 224, 260, 264, 270, 288, 324, 352, 400, 600, 625)] + \
    [(n, True) for n in (4, 8, 121, 169, 225, 243, 338, 500, 1008, 1125)]
COLUMN_CASES = [([6, n, n], 1, "EEPPPP" if w else "PPPPPP", CELL_CENTER, CHAT_2) for n, w in COLUMNS] + \
    [([n, 6, 6], 1, "PPPPPP", CELL_CENTER, CHAT_2) for n in (81, 108, 112, 320)]
# near the longest lines that a plan takes (the general pass has to fit them too)
LONG_CASES = [([6, 4840, 8], 64), ([3600, 6, 8], 64), ([6, 9680, 8], 32), ([7200, 6, 8], 32)]


def _lengths(nglob, center):
    n0 = nglob[0] - (0 if center == CELL_CENTER else 1)
    h = [1.0 / n0] * 3
    return h, [h[d] * (nglob[d] - (0 if center == CELL_CENTER else 1)) for d in range(3)]


def _rhs(nglob, lda, bc, center, seed=5):
    rhs = np.random.default_rng(seed).standard_normal((lda,) + tuple(nglob))
    if center == NODE_CENTER:
        for d in range(3):
            if bc[2 * d] == "P":
                rhs = np.moveaxis(rhs, d + 1, 0)
                rhs[-1] = rhs[0]
                rhs = np.moveaxis(rhs, 0, d + 1)
    return rhs


def _solve(s, u, kind=0):
    import torch
    du = torch.from_numpy(u).cuda()
    out = torch.full_like(du, float("nan"))
    s.solve(out, du, kind)
    torch.cuda.synchronize()
    assert s.last_error() == 0
    return out.cpu().numpy()


def _id(c):
    return f"{c[0][0]}x{c[0][1]}x{c[0][2]}_{c[2]}_{'cell' if c[3] == CELL_CENTER else 'node'}_lda{c[1]}"


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=[_id(c) for c in CASES])
def test_mixed_radix_matches_oracle_and_general_pass(case):
    nglob, lda, bc, center, kernel = case
    h, L = _lengths(nglob, center)
    rhs = _rhs(nglob, lda, bc, center)
    ref = oracle_solve(nglob, lda, _bc(bc, lda), h, L, center, kernel, rhs)
    u = to_user(rhs)
    for precision, tol in ((64, 1e-12), (32, 2e-6)):
        _, s = make_solver(nglob, lda, _bc(bc, lda), h, L, center, kernel, precision=precision)
        kinds = [p["fast"] for p in s.plan_json()["passes"] if p["name"] != "green"]
        assert 6 in kinds and 0 not in kinds, kinds
        got = from_user(_solve(s, u), lda, nglob)
        pf.load_library().flups_b200_set_fast_kernels(s._solver, 0)
        gen = from_user(_solve(s, u), lda, nglob)
        assert rel_l2(got, ref) <= tol
        assert rel_l2(got, gen) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("case", COLUMN_CASES, ids=[_id(c) for c in COLUMN_CASES])
def test_mixed_radix_columns_match_oracle(case):
    nglob, lda, bc, center, kernel = case
    h, L = _lengths(nglob, center)
    rhs = _rhs(nglob, lda, bc, center)
    ref = oracle_solve(nglob, lda, _bc(bc, lda), h, L, center, kernel, rhs)
    for precision, tol in ((64, 1e-12), (32, 2e-6)):
        _, s = make_solver(nglob, lda, _bc(bc, lda), h, L, center, kernel, precision=precision)
        assert rel_l2(from_user(_solve(s, to_user(rhs)), lda, nglob), ref) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("nglob,precision", LONG_CASES)
def test_mixed_radix_long_lines_match_oracle(nglob, precision):
    h, L = _lengths(nglob, CELL_CENTER)
    rhs = _rhs(nglob, 1, "PPPPPP", CELL_CENTER)
    ref = oracle_solve(nglob, 1, _bc("PPPPPP"), h, L, CELL_CENTER, CHAT_2, rhs)
    _, s = make_solver(nglob, 1, _bc("PPPPPP"), h, L, CELL_CENTER, CHAT_2, precision=precision)
    long_passes = [p for p in s.plan_json()["passes"] if p["st"][0]["M"] >= 3600]
    assert long_passes and all(p["fast"] == 6 for p in long_passes)
    assert rel_l2(from_user(_solve(s, to_user(rhs)), 1, nglob), ref) <= (1e-12 if precision == 64 else 2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("lda,type_", [(1, 0), (3, 1)])
@pytest.mark.parametrize("precision", [32, 64])
def test_mixed_radix_batch_equals_single_solves(precision, lda, type_):
    """Pairs of lines stay within a right-hand side: a batch gives the bits of
    its solves one by one (an odd number of lines per plane, 3 of them)."""
    import torch
    nglob, nb = [21, 25, 18], 3
    h, L = _lengths(nglob, CELL_CENTER)
    _, s = make_solver(nglob, lda, _bc("UUUUUU", lda), h, L, CELL_CENTER, HEJ_2, odiff=1 if type_ else 0, precision=precision)
    us = [to_user(_rhs(nglob, lda, "UUUUUU", CELL_CENTER, seed=k)) for k in range(nb)]
    single = np.concatenate([_solve(s, u, type_) for u in us])
    rhs = torch.from_numpy(np.concatenate(us)).cuda()
    out = torch.full_like(rhs, float("nan"))
    s.solve_batch(out, rhs, nb, type_)
    torch.cuda.synchronize()
    assert s.last_error() == 0 and np.array_equal(out.cpu().numpy(), single)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-6)])
def test_mixed_radix_lines_of_very_different_size(precision, tol):
    """Real lines that travel in pairs and differ by up to six orders of
    magnitude: the solution's error stays that of the largest."""
    nglob = [45, 42, 39]
    h, L = _lengths(nglob, CELL_CENTER)
    rhs = _rhs(nglob, 1, "UUUUUU", CELL_CENTER)
    rhs *= 10.0 ** np.random.default_rng(9).uniform(-6, 0, (1, 1, nglob[1], nglob[2]))
    ref = oracle_solve(nglob, 1, _bc("UUUUUU"), h, L, CELL_CENTER, HEJ_2, rhs)
    _, s = make_solver(nglob, 1, _bc("UUUUUU"), h, L, CELL_CENTER, HEJ_2, precision=precision)
    assert rel_l2(from_user(_solve(s, to_user(rhs)), 1, nglob), ref) <= tol


ROT_CASES = [([20, 18, 25], "UUUUUU", 1), ([21, 50, 27], "UUUUUU", 2), ([27, 22, 14], "UUUUUU", 6),
             # walls along x, a periodic direction, fused rows
             ([20, 25, 18], "EOPPUU", 1), ([21, 20, 27], "PPPPUU", 4), ([25, 20, 18], "UUPPPP", 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("nglob,bc,odiff", ROT_CASES)
def test_mixed_radix_rot_matches_oracle(nglob, bc, odiff):
    h, L = _lengths(nglob, CELL_CENTER)
    rhs = _rhs(nglob, 3, bc, CELL_CENTER)
    kernel = HEJ_2 if bc == "UUUUUU" else CHAT_2
    ref = oracle_solve(nglob, 3, _bc(bc, 3), h, L, CELL_CENTER, kernel, rhs, type_=1, odiff=odiff)
    for precision, tol in ((64, 1e-12), (32, 2e-6)):
        _, s = make_solver(nglob, 3, _bc(bc, 3), h, L, CELL_CENTER, kernel, odiff=odiff, precision=precision)
        assert [p["fast"] for p in s.plan_json(1)["passes"] if p["name"] != "green"] == [6] * 5
        got = from_user(_solve(s, to_user(rhs), 1), 3, nglob)
        assert rel_l2(got, ref) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("nglob", [[50, 60, 54], [70, 50, 63]])
def test_mixed_radix_rot_forms_the_curl_in_fp64(nglob):
    """The curl of a gradient is zero, so what an FP32 ROT solve leaves of one
    is rounding: of the spectrum, the same in both families, and of the curl.
    The general pass forms the curl in FP64.  The mixed-radix pass leaves no
    more than it (0.93 and 0.76 of it); formed in FP32 from FP32 symbols it
    left 1.16 and 1.14 times as much."""
    h = 1.0 / nglob[0]
    x = np.meshgrid(*[(np.arange(m) + 0.5) * h for m in nglob], indexing="ij")
    r = [x[d] - 0.5 * nglob[d] * h * (1 + 0.02 * d) for d in range(3)]
    phi = np.exp(-sum(v ** 2 for v in r) / (2 * (3 * h) ** 2))
    u = to_user(np.stack([-r[d] / (3 * h) * phi for d in range(3)]))
    _, s = make_solver(nglob, 3, _bc("UUUUUU", 3), [h] * 3, [h * m for m in nglob], CELL_CENTER, HEJ_2, odiff=1, precision=32)
    got = np.linalg.norm(_solve(s, u, 1))
    pf.load_library().flups_b200_set_fast_kernels(s._solver, 0)
    assert got <= 1.03 * np.linalg.norm(_solve(s, u, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [20, 32])
def test_solve_captured_by_the_caller_equals_the_plain_one(n):
    """Back-to-back solves (passes launched behind each other) and the same
    solve captured in a graph of the caller's own give the same bits."""
    import torch
    h, L = _lengths([n] * 3, CELL_CENTER)
    _, s = make_solver([n] * 3, 1, _bc("UUUUUU"), h, L, CELL_CENTER, HEJ_2)
    rhs = torch.from_numpy(to_user(_rhs([n] * 3, 1, "UUUUUU", CELL_CENTER))).cuda()
    st = torch.cuda.Stream()
    s.set_stream(st)
    s.set_async(True)
    plain, out = torch.zeros_like(rhs), torch.zeros_like(rhs)
    torch.cuda.synchronize()
    for _ in range(5):
        s.solve(plain, rhs)
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        s.solve(out, rhs)
    g.replay()
    torch.cuda.synchronize()
    assert s.last_error() == 0 and torch.equal(out, plain)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-6)])
@pytest.mark.parametrize("lda,type_", [(1, 0), (3, 1)])
def test_odd_folded_outer_extent_of_a_register_fused_pass(precision, tol, lda, type_):
    """64-point fused y columns whose outer direction (z, periodic, 25 points)
    is folded: the order in mirror pairs visits every plane once."""
    nglob = [16, 32, 25]
    h, L = _lengths(nglob, CELL_CENTER)
    bc = _bc("PPUUPP", lda)
    rhs = _rhs(nglob, lda, "PPUUPP", CELL_CENTER)
    ref = oracle_solve(nglob, lda, bc, h, L, CELL_CENTER, HEJ_2, rhs, type_=type_, odiff=1 if type_ else 0)
    _, s = make_solver(nglob, lda, bc, h, L, CELL_CENTER, HEJ_2, odiff=1 if type_ else 0, precision=precision)
    fused = [p for p in s.plan_json(type_)["passes"] if p["fused"]]
    assert [(p["axis"], p["fast"]) for p in fused] == [(1, 1)]
    assert rel_l2(from_user(_solve(s, to_user(rhs), type_), lda, nglob), ref) <= tol


def _kinds(nglob, bc, center, precision=32):
    t = pf.Topology(0, 1, list(nglob))
    h, L = _lengths(nglob, center)
    code = {"E": E, "O": O, "P": P, "U": U}
    s = pf.Solver(t, [[code[bc[2 * d]], code[bc[2 * d + 1]]] for d in range(3)], h, L, center_type=[center] * 3)
    s.set_precision(precision)
    return s, [p["fast"] for p in s.plan_json()["passes"] if p["name"] != "green"]


def _met(nglob, lda, bc, center, type_=0, odiff=0):
    """(precision, two-stage class, operation, rows, place, radix) of the mixed-radix passes of a solve."""
    h, L = _lengths(nglob, center)
    met = set()
    for precision in (32, 64):
        s = pf.Solver(pf.Topology(0, lda, list(nglob)), _bc(bc, lda), h, L, order_diff=odiff, center_type=[center] * 3)
        s.set_precision(precision)
        for p in s.plan_json(type_)["passes"]:
            if p["fast"] == 6:
                r = p["mix"]["radices"]
                for i, radix in enumerate(r):
                    place = "last" if i == len(r) - 1 else ("first" if i == 0 else "middle")
                    met.add((precision, p["mix"]["two"], p["mix"]["op"], p["axis"] == 0, place, radix))
    return met


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def test_cases_meet_every_radix():
    """Of the lengths up to 1200: class TWO with every radix in every place of
    each of its operations, class MULTI with every radix in every place (the
    last one apart where it takes several butterflies), and every operation
    in rows and columns that any set of boundary conditions leads to."""
    met = set()
    for c in CASES + COLUMN_CASES:
        met |= _met(*c[:4])
    for nglob, bc, odiff in ROT_CASES:
        met |= _met(nglob, 3, bc, CELL_CENTER, 1, odiff)
    small_last = {2, 3, 5, 6, 9, 10, 11, 14}  # k and M - k, or three components, in one thread

    def two(m):
        return {x for x in m if x[1]}

    def multi(m):
        return {(x[0], x[4], x[4] == "last" and x[2] in small_last, x[5]) for x in m if not x[1]}

    could = set()
    for n in filter(_smooth, range(4, 1200)):
        for bc in ("EEPPPP", "PPPPPP"):
            could |= _met([6, n, n], 1, bc, CELL_CENTER)
        could |= _met([n, 6, 6], 1, "PPPPPP", CELL_CENTER)
    assert not two(could) - two(met)
    assert not multi(could) - multi(met)
    # rows of types III / II and IV / IV in a fused pass: x is never the last of three walls
    ops = {(op, rows) for op in range(15) for rows in (False, True)} - {(11, True), (13, True)}
    for precision in (32, 64):
        assert not ops - {(x[2], x[3]) for x in met if x[0] == precision}


def test_lengths_outside_the_radices_stay_on_the_general_pass():
    """A prime factor above 13, a length of one radix and a type-IV line of odd
    size are not split; power-of-two lines keep the register DFTs; with the
    fast kernels off every pass is the general one."""
    for precision in (32, 64):
        assert _kinds([51, 20, 20], "UUUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]  # 102 = 2 3 17
        assert _kinds([21, 20, 20], "EOUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]
        assert _kinds([13, 20, 20], "PPUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]
        # 3 5^4: no four radices up to 13, and 15 and 25 are FP32 ones
        assert _kinds([6, 1875, 6], "PPPPPP", CELL_CENTER, precision)[1] == [6, 0 if precision == 64 else 6, 6, 0 if precision == 64 else 6, 6]
        assert _kinds([64, 64, 64], "UUUUUU", CELL_CENTER, precision)[1] == [3, 1, 5, 1, 3]
        s, kinds = _kinds([20, 20, 20], "UUUUUU", CELL_CENTER, precision)
        assert kinds == [6] * 5
        pf.load_library().flups_b200_set_fast_kernels(s._solver, 0)
        assert [p["fast"] for p in s.plan_json()["passes"] if p["name"] != "green"] == [0] * 5


def test_one_module_per_mixed_radix_operation():
    """A module is loaded whole at its first launch: each operation, precision
    and direction is a translation unit of its own."""
    import re
    from flups_b200 import build
    ops = re.findall(r"^    MX_\w+ = (\d+),", (build.CSRC / "mix_dft.h").read_text(), re.M)
    assert sorted(map(int, ops)) == list(range(build.MIX_OPS))
    units = [d for s, _, d in build.units() if s.name == "mix_unit.cu"]
    assert len(units) == len(set(units)) == 4 * build.MIX_OPS
    names = [n for _, n, _ in build.units()]
    assert len(names) == len(set(names))
    others = [s for s in build.CSRC.glob("*.cu") if s.name != "mix_unit.cu" and '#include "mix_dft_impl.cuh"' in s.read_text()]
    assert not others
