"""The rule of fem_launch.cuh for kernels that may start before their predecessor has
ended: what the predecessor writes is read with plain loads.  A read-only load (__ldg, or
one the compiler makes of a const __restrict__ argument) needs data that nobody writes
while the kernel is resident."""
import os
import re

import numpy as np
import pytest

import moris_gb300 as mg
from tests.common import RTOL, csr_row_rel_err, problem, uniform01

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moris_gb300", "csrc")

# kernels launched with overlap (and the helpers their work is in): file, and what a
# kernel before them in the same chain writes
OVERLAPPED = {
    "lattice_project": ("fem_lattice.cu", ["p.S"]),
    "lattice_rows": ("fem_lattice.cu", ["S"]),
    "lattice_restrict": ("fem_lattice.cu", ["rn"]),
    "lattice_product": ("fem_lattice.cu", ["p.u", "p.r"]),
    "const_blocks": ("fem_lattice.cu", ["p.u", "p.r"]),
    "neighbours": ("fem_lattice.cu", ["p.u"]),
    "hex_cells": ("fem_hex.cuh", ["p.u", "p.r", "p.S", "p.vals"]),
    "hex_residual": ("fem_hex.cuh", ["p.u", "p.r"]),
    "k_pair_product": ("fem_solver.cu", ["z", "pa", "pb", "q", "st"]),
    "k_pair_update": ("fem_solver.cu", ["x", "r", "z", "pa", "pb", "q", "st"]),
    "stencil_sweep": ("fem_multigrid.cu", ["x"]),
    "mg_cheb_init": ("fem_multigrid.cu", ["b"]),
    "mg_cheb_step": ("fem_multigrid.cu", ["din", "r", "x"]),
    "mg_residual_update": ("fem_multigrid.cu", ["d", "r"]),
    "mg_post_first": ("fem_multigrid.cu", ["e", "r", "x"]),
    "mg_restrict": ("fem_multigrid.cu", ["r"]),
    "mg_prolong": ("fem_multigrid.cu", ["xc"]),
    "mg_gemv": ("fem_multigrid.cu", ["b"]),
    "mg_convert": ("fem_multigrid.cu", ["a"]),
}


def _function(text, name):
    """Argument list and body of the definition of `name`."""
    for m in re.finditer(r"\b%s\(" % name, text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        rest = re.match(r"\s*(const\s*)?\{", text[i:])
        if not rest:
            continue  # a call
        args, start = text[m.end():i - 1], i + rest.end()
        i, depth = start, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        return args, text[start:i]
    raise AssertionError("no definition of " + name)


def _mentions(expr, names):
    return any(re.search(r"(?<![\w.>])%s(?!\w)" % re.escape(n), expr) for n in names)


@pytest.mark.parametrize("name", sorted(OVERLAPPED))
def test_no_read_only_loads_of_what_a_predecessor_writes(name):
    file, written = OVERLAPPED[name]
    with open(os.path.join(CSRC, file)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    args, body = _function(text, name)
    for a in args.split(","):
        assert not ("__restrict__" in a and _mentions(a, written)), a
    names = set(written)
    while True:  # pointers formed from them
        more = {m.group(1) for m in re.finditer(r"\*\s*(\w+)\s*=\s*([^;,]+)", body) if _mentions(m.group(2), names)}
        if more <= names:
            break
        names |= more
    for m in re.finditer(r"__ldg\(", body):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(body[i], 0)
            i += 1
        assert not _mentions(body[m.end():i - 1], names), body[m.start():i]


def test_every_overlapped_kernel_is_listed():
    """Kernels with a wait on their predecessor; the two side kernels read nothing of it."""
    found = set()
    for file in sorted(os.listdir(CSRC)):
        if not file.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, file)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__[^;{]*?(\w+)\(", text):
            name = m.group(1)
            if name == "__launch_bounds__":
                name = re.match(r"[^{;]*?\)\s*(\w+)\(", text[m.end():]).group(1)
            if "cudaGridDependencySynchronize" in _function(text, name)[1]:
                found.add(name)
    assert found - set(OVERLAPPED) == {"side_cta_kernel", "lattice_plane_sides"}


@pytest.mark.gpu
@pytest.mark.parametrize("shape,density", [(mg.SHAPE_RECTANGULAR, False), (mg.SHAPE_RECTANGULAR, True),
                                           (mg.SHAPE_GENERAL, False)], ids=["bricks", "density", "distorted"])
def test_projection_reads_the_stencil_of_its_own_set(shape, density):
    """Without a residual the projection follows the kernel that writes the stencil
    directly.  Two sets of different moduli share the stencil's memory, so stale values of
    one would show in the other."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m, _, mesh = problem(3, (13, 12, 11), 2, shape, mg.RULE_HEX_2x2x2, density=density)
    nc = len(mesh["cells"])
    m.add_bulk_set(np.arange(nc, dtype=np.int32), 10.0 + uniform01(8, nc), 0.1, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
    m.finalize()
    rp, _ = m.graph()
    out = []
    for k in range(6):
        vals = torch.full((m.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        m.assemble(None, vals, None, mg.NO_RESIDUAL)
        out.append(vals.cpu().numpy())
    m.set_variant(0, 2)
    m.set_variant(1, 2)
    vals = torch.full((m.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    m.assemble(None, vals, None, mg.NO_RESIDUAL)
    ref = vals.cpu().numpy()
    for v in out:
        assert csr_row_rel_err(rp, v, ref) <= RTOL
