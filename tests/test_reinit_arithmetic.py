"""The reinitialization's integer-pipe shortcuts (m2cg_intfp.cuh) against the
forms that they replace, compiled for the host: bit for bit over operands of
every class, NaNs of both signs, infinities and zeros of both signs among them."""
import shutil
import subprocess

import pytest

from test_intfp import HEADER, HOST

PRELUDE = HOST.split("static uint64_t s =")[0]
RANDOM = r"""
static uint64_t s = 88172645463325252ull;
static uint64_t nx() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static const double odd[12] = {0.0, -0.0, INFINITY, -INFINITY, d64(0x7ff8000000000000ull), d64(0xfff8000000000000ull),
                               d64(0x7ff0000000000001ull), d64(0xfff0000000000123ull), 4.9e-324, -4.9e-324,
                               1.7976931348623157e308, -1.7976931348623157e308};
static double draw(double near) {
  const uint64_t r = nx();
  switch (r % 5) {
    case 0: return odd[(r >> 8) % 12];
    case 1: return d64(nx());                                              // any bits
    case 2: return near;
    case 3: return near * (1.0 + 0x1p-52 * ((int)((r >> 8) % 9) - 4));     // next to it
    default: return ((double)(nx() >> 11) * 0x1p-52 - 1.0) * 0.3;
  }
}
"""
ONE_SIDED = RANDOM + r"""
static double flip(double x, bool neg) { return d64(u64(x) ^ (neg ? 0x8000000000000000ull : 0ull)); }
static double both(double p, double m, double n, bool neg) {   // the two differences, the larger pattern or +0
  const int64_t a = (int64_t)u64(flip(p - m, neg)), b = (int64_t)u64(flip(p - n, neg)), c = a > b ? a : b;
  return d64((uint64_t)(c > 0 ? c : 0));
}
int main() {
  long bad = 0, special = 0;
  for (long i = 0; i < 20000000; i++) {
    const double p = draw(0.1), m = draw(p), n = draw(i & 1 ? p : m);
    const bool neg = nx() & 1;
    const bool sp = (int32_t)(if_special_bit(p) | if_special_bit(m) | if_special_bit(n)) < 0;
    const uint32_t sb = neg ? 0x80000000u : 0u;
    const double x = if_one_sided_any(p, m, n, sb), y = both(p, m, n, neg);
    bad += u64(x) != u64(y) || sp != !(std::isfinite(p) && std::isfinite(m) && std::isfinite(n));
    if (sp) special++;
    else bad += u64(if_one_sided(p, m, n, sb)) != u64(y);
  }
  printf("%ld %ld\n", bad, special);
}
"""


def _run(tmp_path, source):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PRELUDE.replace("HEADER", HEADER) + source)
    r = subprocess.run([cc, "-O2", "-std=c++17", "-ffp-contract=off", str(src), "-o", str(exe)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    return [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, timeout=300).stdout.split()]


def test_one_sided_difference_equals_both_differences(tmp_path):
    bad, special = _run(tmp_path, ONE_SIDED)
    assert special > 1000000
    assert bad == 0
