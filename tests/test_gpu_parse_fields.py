"""Fields at the edges of the parser's 16-byte form (at most 15 digits, one dot,
a space or the line's end after them) and just outside it, at every alignment
within a word, against the cloud-text oracle.  Doubles: equal bits."""
import random

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _field(rng, digits, dot, sign):
    s = "".join(rng.choice("0123456789") for _ in range(digits))
    if rng.random() < 0.2:
        s = "0" * (digits // 2) + s[digits // 2:]
    if dot is not None:
        s = s[:dot] + "." + s[dot:]
    return sign + s


@pytest.mark.parametrize("digits", [1, 2, 7, 8, 9, 14, 15, 16, 17, 19, 20])
@pytest.mark.parametrize("sep,tail", [(" ", ""), ("   ", " 7 x"), ("\t", "\r"), (" \v", " ")])
def test_fields(owm, ctx, digits, sep, tail):
    rng = random.Random(digits)
    lines = []
    for dot in [None] + list(range(digits + 1)):
        for sign in ("", "-", "+"):
            for pad in range(4):  # shifts the following fields by a byte each
                f = [_field(rng, digits, dot, sign), _field(rng, rng.randint(1, digits), None, ""),
                     _field(rng, digits, rng.choice([None, 0, digits]), sign)]
                lines.append(" " * pad + sep.join(f) + tail)
        lines.append(sep.join([_field(rng, digits, dot, "") + e for e in ("e2", "E-3", "")]) + tail)
    rng.shuffle(lines)
    for end in ("\n", ""):
        text = ("\n".join(lines) + end).encode()
        want = O.xyz_parse(text)
        c = ctx.cloud_parse_xyz(text)
        np.testing.assert_array_equal(c.points().view(np.uint64), want[0].view(np.uint64))
        c.close()


@pytest.mark.parametrize("bad", ["1.2.3 4 5", "1 2 3.4.", ". 1 2", "1 - 3", "12a 3 4", "1 2 +", "1 2", "--1 2 3", "1,5 2 3",
                                 "1 2 nan", "1 2 0x", "1e 2 3"])
def test_lines_like_the_oracle(owm, ctx, bad):
    text = ("1 2 3\n" * 40 + bad + "\n" + "4.5 -6 7\n" * 5).encode()
    want = O.xyz_parse(text)
    if want is None:
        with pytest.raises(owm.OwmError):
            ctx.cloud_parse_xyz(text)
    else:
        c = ctx.cloud_parse_xyz(text)
        np.testing.assert_array_equal(c.points().view(np.uint64), want[0].view(np.uint64))
        c.close()
