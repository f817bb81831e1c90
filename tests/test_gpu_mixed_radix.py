"""The mixed-radix line passes (flups_b200/csrc/mix_dft_impl.cuh): every
operation against the FP64 oracle and the general line pass, at lengths of
two, three and four stages, every radix, odd sizes, partial tiles and pairs
without a partner; and, without a GPU, which passes take them."""
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
]


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
@pytest.mark.parametrize("nglob,odiff", [([20, 18, 25], 1), ([21, 50, 27], 2), ([27, 22, 14], 6)])
def test_mixed_radix_rot_matches_oracle(nglob, odiff):
    h, L = _lengths(nglob, CELL_CENTER)
    bc = _bc("UUUUUU", 3)
    rhs = _rhs(nglob, 3, "UUUUUU", CELL_CENTER)
    ref = oracle_solve(nglob, 3, bc, h, L, CELL_CENTER, HEJ_2, rhs, type_=1, odiff=odiff)
    for precision, tol in ((64, 1e-12), (32, 2e-6)):
        _, s = make_solver(nglob, 3, bc, h, L, CELL_CENTER, HEJ_2, odiff=odiff, precision=precision)
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


def test_lengths_outside_the_radices_stay_on_the_general_pass():
    """A prime factor above 13, a length of one radix and a type-IV line of odd
    size are not split; power-of-two lines keep the register DFTs; with the
    fast kernels off every pass is the general one."""
    for precision in (32, 64):
        assert _kinds([51, 20, 20], "UUUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]  # 102 = 2 3 17
        assert _kinds([21, 20, 20], "EOUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]
        assert _kinds([13, 20, 20], "PPUUUU", CELL_CENTER, precision)[1] == [0, 6, 6, 6, 0]
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
