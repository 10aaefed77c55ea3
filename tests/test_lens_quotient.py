"""The anchor search divides a window's places by the lens model's radius from the radius's correctly rounded reciprocal r
(LensWindow::over in lizard_gb300/csrc/anchor.cu): q = RN(a r), then twice q = RN(q + r RN(a - b q)), each step one fused
multiply-add (Markstein, 1990). Checked here in exact rational arithmetic: q is the correctly rounded a / b."""
import random
from fractions import Fraction


def rn64(x):
    """A rational rounded to the nearest double, ties to even (normal range), as a Fraction."""
    if x == 0:
        return Fraction(0)
    n, d = abs(x.numerator), x.denominator
    e = n.bit_length() - d.bit_length()
    if (n << max(0, -e)) < (d << max(0, e)):
        e -= 1                                  # 2^e <= |x| < 2^(e + 1)
    ulp = Fraction(2) ** (e - 52)
    m = Fraction(n, d) / ulp
    fl = m.numerator // m.denominator
    rem = m - fl
    if rem > Fraction(1, 2) or (rem == Fraction(1, 2) and fl % 2 == 1):
        fl += 1
    return (fl if x > 0 else -fl) * ulp


def over(a, b):
    r = rn64(1 / b)
    q = rn64(a * r)
    for _ in range(2):
        q = rn64(q + r * rn64(a - b * q))
    return q


def test_rounding_is_a_doubles():
    rng = random.Random(0)
    for _ in range(500):
        a, b = rng.uniform(-1e9, 1e9), rng.uniform(1e-3, 1e9)
        assert float(rn64(Fraction(a) / Fraction(b))) == a / b


def test_quotients_are_correctly_rounded():
    rng = random.Random(1)
    one = 1 << 52
    mantissas = [one, one + 1, one + 2, 2 * one - 1, 2 * one - 2, 3 * one // 2, 3 * one // 2 + 1, 3 * one // 2 - 1]

    def mantissa():
        return rng.choice(mantissas) if rng.random() < 0.3 else rng.randrange(one, 2 * one)

    for k in range(6000):
        b = Fraction(mantissa()) * Fraction(2) ** rng.randrange(-150, 46)       # 1e-30 < b < 1e30
        if k % 3:
            a = Fraction(mantissa()) * Fraction(2) ** rng.randrange(-150, 46)
        else:                                                                   # a quotient close to halfway between doubles
            a = rn64(b * (2 * mantissa() + 1) * Fraction(2) ** rng.randrange(-60, -50))
        a = a if rng.random() < 0.5 else -a
        assert over(a, b) == rn64(a / b), (a, b)


def test_quotients_of_pixels_by_a_frames_radius():
    """The values the search meets: a float place less a double centre, over half a frame's diagonal."""
    rng = random.Random(2)
    for _ in range(3000):
        b = Fraction(rng.uniform(100.0, 9000.0))
        a = Fraction(rng.uniform(-1.0, 1.0) * 8192.0)
        assert over(a, b) == rn64(a / b)
