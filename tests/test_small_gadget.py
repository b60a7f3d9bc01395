"""The double-precision scaling of small gadgets (via_rs_b200/csrc/gadget_fp.cuh fp_scaled), restated
with exact-rational FMAs: round(r S / Q) for residues |r| <= 9/16 Q and 9 Q S < 8 2^53, at the
residues nearest a tie. No GPU needed."""
from fractions import Fraction

import pytest

ROUND = 6755399441055744.0  # 1.5 * 2^52


def fp_scaled(r, S, Q):
    return int(float(Fraction(float(r) * float(S)) * Fraction(1.0 / Q) + Fraction(ROUND)) - ROUND)


def nearest_to_ties(Q, S):
    """Residues whose r S / Q lies 1 / (2 Q) from a tie, in every representative up to 9/16 Q."""
    for t in ((Q - 1) // 2, (Q + 1) // 2):
        r = t * pow(S, -1, Q) % Q
        for x in (r, r - Q):
            if 16 * abs(x) <= 9 * Q:
                yield x


def exact(r, S, Q):
    return (2 * r * S + Q) // (2 * Q)


# Primes just below 2^35 whose rounded inverse is off by nearly half an ulp, and the preset's.
@pytest.mark.parametrize("Q", [34347294721, 34348572673, 17175674881])
def test_scaling_is_exact(Q):
    top = int(((8 << 53) / (9 * Q)) ** 0.5)
    seen = 0
    for B in range(2, top + 1):
        if 9 * Q * (B * B + 1) >= 8 << 53:
            continue
        for r in nearest_to_ties(Q, B * B):
            assert fp_scaled(r, B * B, Q) == exact(r, B * B, Q), (B, r)
            seen += 1
    assert seen > 500


def test_the_line_is_needed():
    Q, S = 34347294721, 509 * 509
    assert Q * (S + 1) < 1 << 53 and 9 * Q * S > 8 << 53
    assert any(fp_scaled(r, S, Q) != exact(r, S, Q) for r in nearest_to_ties(Q, S))
