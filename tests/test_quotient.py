"""quotient.cuh (the smoothing's division by a constant pivot) against the division, to the bit: the
pivots of the Thomas solve at several coefficients, numerators of every magnitude, zeros of both
signs, infinities and NaN.  The header is compiled for the host."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "aero2d_b200" / "csrc"

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#include "quotient.cuh"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }

template <typename T, typename U>
long run(int bits) {
  long bad = 0;
  auto check = [&](T a, T b) {
    const T v = a2d::quotient<T>(a, b, T(1) / b), t = a / b;
    if (t != t) bad += v == v;
    else bad += std::memcmp(&v, &t, sizeof(T)) != 0;
  };
  const double es[] = {0.6, 0.001, 0.05, 0.25, 1.0, 3.0, 100.0};
  for (double e : es) {
    T cp = 0;
    for (int j = 0; j < 8; ++j) {
      const T b = (j == 0 ? T(1) + T(e) : T(1) + T(2) * T(e)) - (j == 0 ? T(0) : -T(e)) * cp;
      cp = -T(e) / b;
      const U exps = U(1) << (8 * sizeof(T) - 1 - bits);   // exponent fields, subnormals and infinities among them
      for (U x = 0; x < exps; ++x)
        for (int n = 0; n < 40; ++n) {
          U u = (x << bits) | (U(rnd()) & ((U(1) << bits) - 1)) | (U(rnd() & 1) << (8 * sizeof(T) - 1));
          T a;
          std::memcpy(&a, &u, sizeof(T));
          check(a, b);
        }
      for (T a : {T(0), -T(0), std::numeric_limits<T>::infinity(), -std::numeric_limits<T>::infinity(),
                  std::numeric_limits<T>::quiet_NaN(), std::numeric_limits<T>::max(), std::numeric_limits<T>::denorm_min()})
        check(a, b);
    }
  }
  return bad;
}

int main() {
  std::printf("%ld %ld\n", run<float, uint32_t>(23), run<double, uint64_t>(52));
}
"""


def test_quotient_is_the_division(tmp_path):
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", "-x", "c++", str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0"]
