"""Solves on the caller's own non-blocking stream, the first one captured in a
graph among them: tables reach the device before the passes that read them."""
import re
from pathlib import Path

import numpy as np
import pytest

from gpu_helpers import make_solver, to_user
from oracle.plans import CELL_CENTER, CHAT_2

CSRC = Path(__file__).resolve().parent.parent / "flups_b200" / "csrc"


def test_no_upload_outside_the_solvers_stream():
    """A cudaMemcpy from pageable memory may return before its data has
    arrived, and a non-blocking stream is not ordered behind it: uploads name
    the stream of the passes."""
    for src in sorted(CSRC.iterdir()):
        assert not re.search(r"\bcudaMemcpy\(", src.read_text()), src.name


def _problem(n, bc, lda=1):
    code = {"E": 0, "O": 1, "P": 3, "U": 4}
    b = [[[code[bc[2 * d]]] * lda, [code[bc[2 * d + 1]]] * lda] for d in range(3)]
    h = [1.0 / n[0]] * 3
    return b, h, [h[d] * n[d] for d in range(3)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n,bc", [([3003, 12, 10], "PPPPUU"), ([64, 1024, 8], "UUUUUU"), ([2100, 20, 22], "EOOEPP")])
def test_first_solve_on_a_side_stream_equals_the_next(n, bc, precision):
    import torch
    b, h, L = _problem(n, bc)
    st = torch.cuda.Stream()
    rhs = torch.from_numpy(to_user(np.random.default_rng(3).standard_normal([1] + n))).cuda()
    first, second = torch.full_like(rhs, float("nan")), torch.full_like(rhs, float("nan"))
    torch.cuda.synchronize()
    _, s = make_solver(n, 1, b, h, L, CELL_CENTER, CHAT_2, precision=precision)
    s.set_stream(st)
    s.set_async(True)
    s.solve(first, rhs)
    s.solve(second, rhs)
    st.synchronize()
    assert s.last_error() == 0 and torch.equal(first, second)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n,bc,type_", [([20, 30, 22], "UUUUUU", 0), ([64, 64, 64], "UUUUUU", 0), ([45, 30, 21], "EEOOPP", 0),
                                        ([20, 28, 36], "OEEOOE", 0), ([34, 20, 18], "UUUUUU", 0), ([20, 30, 22], "UUUUUU", 1),
                                        ([64, 64, 64], "UUUUUU", 1)])
def test_first_solve_may_be_captured(n, bc, type_, precision):
    """Set-up makes every table a solve of device arrays reads, so the first
    solve allocates nothing and its caller may capture it; replayed, it gives
    the bits of a plain solve."""
    import torch
    lda = 3 if type_ else 1
    b, h, L = _problem(n, bc, lda)
    rhs = torch.from_numpy(to_user(np.random.default_rng(5).standard_normal([lda] + n))).cuda()
    out, plain = torch.full_like(rhs, float("nan")), torch.full_like(rhs, float("nan"))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    _, s = make_solver(n, lda, b, h, L, CELL_CENTER, CHAT_2, odiff=1 if type_ else 0, precision=precision)
    s.set_stream(st)
    s.set_async(True)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        s.solve(out, rhs, type_)
    g.replay()
    torch.cuda.synchronize()
    s.solve(plain, rhs, type_)
    st.synchronize()
    assert s.last_error() == 0 and not torch.isnan(out).any() and torch.equal(out, plain)
