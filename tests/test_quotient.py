"""quotient() of csrc/quotient.h, which the float64 fluxes take in place of a division (physics.cuh), on the CPU: the
same source, compiled for the host.  Equal to a / b bit for bit over random operands of the fluxes' range, with a
divisor's own reciprocal and with the product of two (the temperature's); at zeros, infinities, NaN and overflowing
quotients, where refinable() withholds the residual, the division's value; one unit in the last place where the
quotient is subnormal.  Multiplying by the rounded reciprocal alone misses about a quarter of the values."""

import shutil
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "jax_fluid_sim_b200" / "csrc" / "quotient.h"

PROGRAM = """
#include <cfloat>
#include <cstdio>
#include <random>
#include "%s"
using namespace dgb;
static bool same(double a, double b) { return a == b || (a != a && b != b); }
int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> e(-46.0, 60.0), m(-1.0, 1.0);
  long wrong = 0, wrong2 = 0, plain = 0, kept = 0;
  const long n = 4000000;
  for (long i = 0; i < n; ++i) {
    const double b = exp2(e(g)) * (1.0 + (double)(g() >> 12) * 0x1p-52), a = m(g) * exp2(e(g)), inv = 1.0 / b;
    const double R = 287.0 * (1.0 + 0.01 * m(g)), d = b * R;
    wrong += quotient(a, b, inv) != a / b;
    wrong2 += quotient(a, d, inv * (1.0 / R)) != a / d;
    plain += product(a, inv) != a / b;
    kept += !refinable(a, b, inv);
  }
  const double as[] = {0.0, -0.0, 1.0, -3.5, 1e308, -1e308, INFINITY, -INFINITY, NAN}, bs[] = {1e-14, 1.0, 49.0, 1e300, INFINITY};
  long special = 0, tiny = 0;
  for (double a : as)
    for (double b : bs) {
      const double inv = 1.0 / b;
      special += !same(quotient(a, b, inv, refinable(a, b, inv)), a / b);
    }
  for (double a : {1e-308, -3e-310, 5e-324})
    for (double b : {49.0, 1e10}) tiny += fabs(quotient(a, b, 1.0 / b) - a / b) > 5e-324;
  printf("%%ld %%ld %%ld %%ld %%ld %%d\\n", wrong, wrong2, kept, special, tiny, plain > n / 5);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_equal_to_the_division(tmp_path):
    src = tmp_path / "q.cpp"
    src.write_text(PROGRAM % HEADER)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", str(src), "-o", str(tmp_path / "q")], check=True)
    out = subprocess.run([str(tmp_path / "q")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0", "0", "0", "1"], out
