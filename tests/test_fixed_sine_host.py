"""The quarter-wave table of the fixed-point sine: every entry is the
integer nearest to 2^62 sin(pi/2 j/1024), from the Taylor series in exact
integer arithmetic (80 guard bits, pi from Machin's formula)."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
TABLE = os.path.join(os.path.dirname(HERE), 'pyheadtail_gb300', 'csrc',
                     'phk_sine_table.inc')
ONE = 1 << 144


def _atan_inverse(n):
    total, term, k = 0, ONE // n, 0
    while term:
        total += (-1)**k * (term // (2 * k + 1))
        term //= n * n
        k += 1
    return total


def test_every_entry():
    with open(TABLE) as f:
        text = re.sub(r'//.*', '', f.read())
    got = [int(v, 16) for v in re.findall(r'0x([0-9a-f]+)ull', text)]
    assert len(got) == 1025
    half_pi = 2 * (4 * _atan_inverse(5) - _atan_inverse(239))
    for j, v in enumerate(got):
        a = half_pi * j // 1024
        total, term, k = 0, a, 1
        while term:
            total += term
            term = -term * a // ONE * a // ONE // ((k + 1) * (k + 2))
            k += 2
            if abs(term) <= 1:
                break
        assert v == (total + (1 << 81)) >> 82, j
