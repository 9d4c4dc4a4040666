"""The FP64 fast path's fixed-point line solves (csrc/ati_fixed_line.h), compiled for the host, against extended precision
and the FP64 sweeps' arithmetic on the same lines.

Errors are taken point by point over many lines of a kind: the root mean square at a point of the line, the solve's over
the FP64 arithmetic's.  A unit of the solve is 2^-57 of the largest difference its group of eight rows reads, FP64 rounds
at 2^-53 of each row's values, and a group's own spread, at most a third of a bit a row on the smooth lines here, takes 2.7
bits of the four: no larger over the line and on average over its points, at most twice as large at a single one.  (1 %
for where both round one product, rough lines of the filter.)  No integer of the solve reaches 2^62.9.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tandemproject_gb300", "csrc")

# shortest lines, one group and two, ragged last groups, segment edges, many segments, the longest
LENGTHS = [13, 14, 23, 24, 29, 31, 40, 47, 48, 49, 57, 97, 121, 193, 385, 800]
OPERATORS = [(0, 0), (0, 1), (1, 0)]  # derivative, derivative of periodic lines, filter


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("line") / "fixed_line_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "fixed_line_host.cpp"), os.path.join(CSRC, "ati_fixed_tab.cpp"),
                    os.path.join(CSRC, "ati_scheme.cpp")], check=True)
    return exe


def run(program, op, length, kind, scale, lines=None, fltk=0.85):
    out = subprocess.run([program, str(op[0]), str(op[1]), str(length), str(kind), str(scale),
                          str(lines or (200 if length < 200 else 60)), "1", str(fltk)], capture_output=True, text=True)
    assert out.returncode == 0, (op, length, kind, out.returncode)
    top, mean, whole, bits = out.stdout.split()
    return float(top), float(mean), float(whole), int(bits)


@pytest.mark.parametrize("length", LENGTHS)
@pytest.mark.parametrize("op", OPERATORS)
def test_smooth_lines(program, op, length):
    """Fields of one size, also very small and large, through zero, falling by a third of a bit a row."""
    fall = min(length // 3, 40)
    kinds = [(0, 0), (0, 300), (0, -300), (1, 0)] + ([(10, fall // 2)] if op[1] else [(2, fall), (3, fall)])
    for kind, scale in kinds:
        top, mean, whole, bits = run(program, op, length, kind, scale)
        assert whole <= 1.01 and mean <= 1.01 and top <= 2 and bits <= 62, (kind, scale, top, mean, whole, bits)


@pytest.mark.parametrize("length", [40, 57, 97, 193])
@pytest.mark.parametrize("op", [(0, 0), (1, 0)])
@pytest.mark.parametrize("quiet", [10, 20, 30])
def test_layer_beside_a_small_wave(program, op, length, quiet):
    """A tanh layer and a wave 2^-10 to 2^-30 of it: the wave's part of the line is as accurate as with FP64.  The layer's
    tail falls by 0.72 bits a row, 3.1 bits a group more than the lines above: so much more at a single point."""
    top, mean, whole, bits = run(program, op, length, 4, quiet)
    assert whole <= 1.01 and mean <= 1.01 and top <= 2 * 2 ** 3.1 and bits <= 62, (top, mean, whole, bits)


@pytest.mark.parametrize("length", LENGTHS)
@pytest.mark.parametrize("op", OPERATORS)
def test_integers_stay_in_range(program, op, length):
    """Lines that drive the solve hardest: single large values, jumps, differences as large as the values, values of all
    sizes side by side, a constant."""
    for kind, scale in [(5, 20), (5, 60), (6, 0), (7, 10), (7, 200), (8, 0), (8, 5), (8, 60), (9, 20), (9, 60), (11, 0)]:
        bits = run(program, op, length, kind, scale, 60)[3]
        assert bits <= 62, (kind, scale, bits)


@pytest.mark.parametrize("length", [13, 48, 97])
def test_rough_lines(program, length):
    """Values without any smoothness, over the whole line."""
    for op in OPERATORS:
        for kind, scale in [(6, 0), (7, 10)]:
            whole = run(program, op, length, kind, scale)[2]
            assert whole <= 1.01, (op, kind, whole)


@pytest.mark.parametrize("fltk", [0.5, 0.6, 0.7, 0.8, 0.9, 0.93])
def test_filter_cut_offs(program, fltk):
    """The scales follow the filter: in range and as accurate at every cut-off that the fixed-point sweeps take."""
    for length in (13, 49, 97, 800):
        top, mean, whole, bits = run(program, (1, 0), length, 0, 0, 60, fltk)
        assert whole <= 1.01 and mean <= 1.01 and top <= 2 and bits <= 62, (length, top, mean, whole, bits)
        for kind, scale in [(6, 0), (8, 0), (9, 20)]:
            assert run(program, (1, 0), length, kind, scale, 60, fltk)[3] <= 62


@pytest.mark.parametrize("fltk", [0.97, 0.99])
def test_extreme_filters_are_left_to_the_fp64_sweeps(program, fltk):
    out = subprocess.run([program, "1", "0", "97", "0", "0", "1", "1", str(fltk)], capture_output=True)
    assert out.returncode == 3


@pytest.mark.parametrize("op,fltk", [(0, 0.85), (1, 0.5), (1, 0.6), (1, 0.7), (1, 0.85), (1, 0.9), (1, 0.93)])
def test_scales_leave_room_at_every_length(program, op, fltk):
    """The scales an operator gets: 57 to 60 bits for differences, and no value of a group's rows above 2^62.9 on lines of 13
    to 800 points, open or periodic, by the bound that holds for any line."""
    out = subprocess.run([program, "scales", str(op), str(fltk)], check=True, capture_output=True, text=True).stdout
    head, *rows = [line.split() for line in out.splitlines()]
    gbits, k, carry, spare, carry_end = map(int, head)
    assert 57 <= gbits <= 60 and 0 <= k <= 8 and 56 <= carry <= 60 and spare <= 2 and carry_end >= 56, head
    assert len(rows) == 8 * (2 - op)
    for length, per, bits in rows:
        assert float(bits) < 62.9, (length, per, bits)


@pytest.mark.parametrize("fltk", [0.3, 0.45, 0.95])
def test_scales_of_filters_that_do_not_fit(program, fltk):
    """Cut-offs below some 0.5 and above some 0.93 of the grid's limit: no scales, the FP64 sweeps filter."""
    out = subprocess.run([program, "scales", "1", str(fltk)], check=True, capture_output=True, text=True).stdout
    assert out.split()[0] == "0"
