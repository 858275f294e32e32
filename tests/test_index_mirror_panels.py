"""CPU replay of the memory indexing of today's panel kernels (tests/index_mirror/k_panels_mirror.c) for every
size that their launchers admit; the block sizes and limits are read from k_inv.cu, so that a change there
reaches the replay."""
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(os.path.dirname(HERE), "gaspacho2_b200", "csrc", "k_inv.cu")).read()


def _const(name):
    m = re.search(rf"\b{name} = (\d+)\b", SRC)
    assert m, f"{name} not found in k_inv.cu"
    return int(m.group(1))


@pytest.fixture(scope="module")
def mirror(tmp_path_factory):
    def build(**over):
        exe = str(tmp_path_factory.mktemp("mirror") / "k_panels_mirror")
        defs = {n: _const(n) for n in ("IB", "IS", "NB", "CW", "RB", "RC", "kPotrfHalfP")}
        defs.update(over)
        subprocess.run(["gcc", "-O2", "-std=c11"] + [f"-D{k}={v}" for k, v in defs.items()] +
                       ["-o", exe, os.path.join(HERE, "index_mirror", "k_panels_mirror.c")], check=True)
        return exe
    return build


def test_layouts_are_the_sources():
    """The shared-memory layouts that the replay builds on, as the source states them."""
    for line in ("const int rows_pad = max(IB, (P + 15) / 16 * 16);",
                 "const int SP = rows_pad + 2, space = ns * CW * (rows_pad + 4);",
                 "return (int)sizeof(double) * (IB * (rows_pad + 2) + ns * CW * (rows_pad + 4) + IB);",
                 "return 2 * (potrf_panel_smem(P, 3) + extra + 1536) <= 228 * 1024 ? 3 : 2;",
                 "return (int)sizeof(double) * (IB * (nb * IB + 4) + IB * IS + NB * IB * IS);",
                 "const int nb = (P + IB - 1) / IB, SY = nb * IB + 4;",
                 "constexpr int kRowsSmem = (int)sizeof(double) * (RB * IS + 2 * RC * (RSA + RSB) + IB * DS + IB);"):
        assert line in SRC, line


@pytest.mark.parametrize("kernel,first,last", [("potrf", 1, "kPotrfMaxP"), ("rows", 289, 700), ("trtri", 1, "kInverseMaxP"),
                                               ("lauum", 1, "kInverseMaxP")])
def test_every_size_stays_in_bounds(mirror, kernel, first, last):
    last = _const(last) if isinstance(last, str) else last
    r = subprocess.run([mirror(), kernel, str(first), str(last)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == f"ok {kernel} {first}..{last}"


def test_replay_notices_rows_left_out(mirror):
    """One size past the panel kernel's range, and 128 threads past theirs: rows without an update."""
    top = _const("kPotrfMaxP")
    r = subprocess.run([mirror(), "potrf", str(top + 1), str(top + 1)], capture_output=True, text=True)
    assert r.returncode == 1 and "updated 0 times" in r.stderr
    half = _const("kPotrfHalfP")
    r = subprocess.run([mirror(kPotrfHalfP=half + 1), "potrf", str(half + 1), str(half + 1)], capture_output=True, text=True)
    assert r.returncode == 1 and "updated 0 times" in r.stderr


def test_split_products(tmp_path):
    """tests/index_mirror/k_splits_mirror.c: the split products' ranges and the Gram's tiles; with odd range
    starts or a partial sum too few it must fail."""
    exe = str(tmp_path / "k_splits_mirror")
    subprocess.run(["gcc", "-O2", "-std=c11", "-o", exe, os.path.join(HERE, "index_mirror", "k_splits_mirror.c")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
    for arg in ("odd", "short"):
        assert subprocess.run([exe, arg], capture_output=True).returncode == 1
