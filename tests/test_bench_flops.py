"""The FLOP count of the CUDA-core M2L in bench.py against the blocks of the kernel's own steps, enumerated: degree
blocks of the rotations, order blocks of the z translation, coefficient pairs of the azimuth turns."""
import pytest

from bench import rotated_m2l_flops_per_pair


@pytest.mark.parametrize("p", range(1, 17))
def test_rotated_m2l_flops(p):
    lm = [(l, m) for l in range(p + 1) for m in range(-l, l + 1)]
    # a rotation about y keeps the degree and the kind (cosine, sine), a z translation the order
    rotation = sum((a[0] == b[0]) and ((a[1] < 0) == (b[1] < 0)) for a in lm for b in lm)
    shift = sum(a[1] == b[1] for a in lm for b in lm)
    turn = 2 * sum(m != 0 for _, m in lm)                # both coefficients of a pair from both
    assert rotated_m2l_flops_per_pair(p) == 3 * 2 * (2 * rotation + shift + 2 * turn)
