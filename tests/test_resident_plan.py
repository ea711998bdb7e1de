"""The launch shapes of the resident BiCGStab (csrc/resident_plan.h), on the CPU: every plan's
launch is one that the kernel it names accepts, whatever the system's rows and width."""
import itertools
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
SMS, SMEM = 152, 227 * 1024
FIELDS = ("ok", "two", "cluster", "mats", "recomp", "x_in_smem", "ctas", "threads", "rc", "smem", "bound", "gmres")


@pytest.fixture(scope="session")
def plan(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "resident_plan_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(REPO / "tnl-mhfem_gb300" / "csrc"),
                        str(REPO / "tests" / "resident_plan_check.cpp"), "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(systems):
        text = "".join(f"{rows} {width} {real} {SMS} {SMEM}\n" for rows, width, real in systems)
        r = subprocess.run([str(out)], input=text, capture_output=True, text=True)
        assert r.returncode == 0
        return [dict(zip(FIELDS, map(int, line.split()))) for line in r.stdout.splitlines()]

    return run


def test_every_launch_is_within_its_kernels_bounds(plan):
    """Block size within the launch bound, whole warps, shared memory within
    the device's, at most one CTA per SM, every row owned by one CTA."""
    rows = sorted({r + d for r in [1, 128, 1024, 4096, *range(5000, 1_700_000, 9973), 622_592, 262_144]
                   for d in (0, 1)})
    systems = list(itertools.product(rows, [0, 1, 2, 3, 4, 5, 6, 8, 9, 10, 13, 17, 25, 40], [4, 8]))
    for (r, w, real), P in zip(systems, plan(systems)):
        if not P["ok"]:
            continue
        at = (r, w, real, P)
        assert P["threads"] <= P["bound"] and P["threads"] % 32 == 0 and P["threads"] >= 128, at
        assert P["smem"] <= SMEM, at
        assert 1 <= P["ctas"] <= (16 if P["cluster"] else SMS), at
        assert P["ctas"] * P["rc"] >= r, at
        if not P["cluster"]:
            assert (P["ctas"] - 1) * P["rc"] < r, at


def _form(P):
    if not P["ok"]:
        return "five kernels"
    if P["two"]:
        return "cluster" if P["cluster"] else "two"
    if P["mats"]:
        return "three, s recomputed" if P["recomp"] else "three"
    return "streamed" if P["x_in_smem"] else "x in memory"


# (rows, width, bytes per value) -> the form that takes the system: the sizes by which the GPU tests
# reach each form
FORMS = {
    (3_960, 4, 8): "cluster", (4_181, 4, 8): "two", (124_033, 4, 8): "two", (126_485, 4, 8): "three, s recomputed",
    (249_408, 4, 8): "three, s recomputed", (252_880, 4, 8): "three", (357_765, 4, 8): "streamed",
    (677_825, 4, 8): "x in memory", (812_240, 4, 8): "x in memory", (821_633, 4, 8): "five kernels",
    (297_714, 6, 8): "streamed", (777_600, 6, 8): "x in memory",
    (346_560, 9, 8): "streamed", (686_816, 9, 8): "x in memory", (736_400, 9, 8): "five kernels",
    (382_500, 10, 8): "streamed", (658_800, 10, 8): "five kernels",
    (196_800, 13, 8): "streamed", (536_256, 13, 8): "five kernels", (312_132, 21, 8): "five kernels",
    (459_425, 4, 4): "three, s recomputed", (555_560, 4, 4): "streamed", (1_388_560, 4, 4): "x in memory",
    (1_648_725, 4, 4): "five kernels", (1_626_560, 4, 4): "five kernels",
    (437_778, 6, 4): "streamed", (1_515_000, 6, 4): "x in memory", (1_703_520, 6, 4): "five kernels",
    (240_800, 9, 4): "three, s recomputed", (346_560, 9, 4): "streamed", (1_060_080, 9, 4): "five kernels",
    (227_556, 10, 4): "three, s recomputed", (382_500, 10, 4): "streamed", (957_168, 10, 4): "five kernels",
    (143_856, 13, 4): "three, s recomputed", (261_360, 13, 4): "streamed", (726_516, 13, 4): "five kernels",
    (488_136, 21, 4): "five kernels",
}


def test_forms_at_the_sizes_of_the_gpu_tests(plan):
    assert {k: _form(P) for k, P in zip(FORMS, plan(FORMS))} == FORMS


def test_gmres_route_follows_rows_and_width(plan):
    """On the faster side at the sizes where both routes were measured, and resident up to 2^18 rows
    whatever the width."""
    resident = [(262_144, 4), (262_144, 40), (766_085, 4), (720_954, 6), (694_960, 9), (595_428, 13), (287_712, 21)]
    kernels = [(786_433, 4), (779_040, 9), (726_516, 13), (455_112, 21), (677_376, 21)]
    plans = plan([(r, w, 8) for r, w in resident + kernels])
    assert [P["gmres"] for P in plans] == [1] * len(resident) + [0] * len(kernels)


@pytest.mark.gpu
def test_mixed_form_without_off_diagonal_entries():
    """217,800 triangles that share no face, every face Dirichlet: 653,400 rows of ELL width 0, the
    widest CTAs of the mixed form's inner solve.  The traces are the boundary values."""
    import numpy as np
    from helpers import rel_err, variant
    from mhfem import _lib as L
    from mhfem import problems
    from oracle.oracle import OracleModel

    p = variant(problems.heat2d(N=330, steps=1), form=L.FORM_MIXED)
    p.coords = p.coords[p.cells.ravel()]
    p.cells = np.arange(3 * p.C, dtype=p.cells.dtype).reshape(-1, 3)
    p.tol = 1e-13

    def bc(face_verts, face_cells):
        F = face_cells.shape[0]
        return np.zeros(F, np.uint8), np.zeros(F), np.linspace(-0.7, 1.1, F)

    p.bc_fn = bc
    s = problems.make_solver(p)
    assert s.F == 653_400
    assert s.step(0.0, p.dt)["residual"] < 1e-13
    m = OracleModel.from_problem(p)
    m.step(0.0, p.dt, 1e-13)
    zf, zk = s.state()
    assert rel_err(zf, m.Z_iF) < 1e-10 and rel_err(zk, m.Z_iK) < 1e-10
    s.close()
