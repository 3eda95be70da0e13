"""Index arithmetic of the several-row raw-block kernel, walked on the host (csrc/qb_kqrows_units.hpp compiled as plain C++)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "quactlize_b200", "csrc")


def _build(tmp_path_factory, name):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path_factory.mktemp(name) / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, os.path.join(HERE, name + ".cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    exe = _build(tmp_path_factory, "kqrows_units_probe")

    def run(rows, tiles, parts, off):
        text = " ".join(map(str, [rows, len(off) - 1, tiles, parts, *off]))
        r = subprocess.run([exe], input=text, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        return tuple(map(int, r.stdout.split()))
    return run


@pytest.mark.parametrize("rows,experts,n", [(65536, 1024, 14336), (32768, 1024, 16384), (9, 5, 40), (1, 1, 16)])
def test_units_stay_in_bounds_whatever_the_offsets_hold(units, rows, experts, n):
    """The kernel may run before its offsets are checked: sawtooth offsets must not make more groups than the host bounded."""
    rng = np.random.default_rng(rows)
    odd = [0 if i % 2 == 0 else rows for i in range(experts + 1)]
    for off in (odd, odd[::-1], [2**31 - 1] * (experts + 1), [-2**31] * (experts + 1), [rows] * (experts + 1),
                rng.integers(-2**31, 2**31 - 1, experts + 1).tolist(), rng.integers(0, rows + 1, experts + 1).tolist()):
        got, most = units(rows, (n + 15) // 16, 148, off)
        assert got <= most


def test_units_of_valid_offsets(units):
    for rows, experts, seed in ((64, 128, 1), (37, 5, 2), (1000, 16, 3), (3, 8, 4)):
        counts = np.random.default_rng(seed).multinomial(rows, np.ones(experts) / experts)
        off = [0, *np.cumsum(counts).tolist()]
        assert units(rows, 7, 33, off)[0] == sum(-(-int(c) // 8) for c in counts)


@pytest.fixture(scope="module")
def spans(tmp_path_factory):
    return _build(tmp_path_factory, "kqrows_span_probe")


@pytest.mark.parametrize("block,align", [(84, 4), (110, 2), (210, 2), (144, 16), (176, 16)])
def test_copies_stay_inside_the_tensor(spans, block, align):
    """Bulk copies take whole 16-byte units; at the ends of a tensor that begins or ends off a boundary the rest is copied by the byte."""
    for shift in range(0, 16, align):
        for rows, bpr, sb in ((1, 1, 1), (3, 5, 5), (17, 9, 4), (2, 16, 16)):
            text = f"{4096 + shift} {rows * bpr * block} {bpr * block} {sb * block}"
            r = subprocess.run([spans], input=text, capture_output=True, text=True)
            assert r.returncode == 0, (text, r.stdout)
            aligned_ends = shift == 0 and (rows * bpr * block) % 16 == 0
            assert (int(r.stdout) == 0) == aligned_ends, text
