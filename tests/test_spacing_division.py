"""x / h in the samplers (fl_common.cuh, over): the corrected product with the
reciprocal, run on the CPU, equals the division for every cell size that the
entry points take, those included whose quotients or reciprocal leave the
range of normal floats."""
import pytest

from tests import host_source as hs

MAIN = r"""
int main() {
  unsigned s = 5;
  auto bits = [&] { s ^= s << 13; s ^= s >> 17; s ^= s << 5; return s; };
  long wrong = 0;
  auto check = [&](float x, float h) {
    const Spacing sp = make_spacing(h);
    const float got = over(x, sp), want = x / h;
    const bool ok = std::isnan(want) ? std::isnan(got) : got == want;
    if (!ok && wrong++ < 5) std::printf("%%a / %%a: %%a, not %%a\n", x, h, got, want);
  };
  std::vector<float> hs;
  for (int e = %(lo)d; e <= %(hi)d; e++)
    for (int k = 0; k < 40; k++)
      hs.push_back(std::ldexp(1.0f + (k ? bits() & 0x7fffff : 0) * 0x1p-23f, e));
  %(more)s
  for (float h : hs) {
    for (int k = 0; k < 400; k++) check(bits_as<float>(bits()), h);              // any float
    for (int k = 0; k < 400; k++) check((bits() %% 8192 + 0.5f) * h, h);         // positions
    for (int k = 0; k < 200; k++) check(std::ldexp(1.0f + (bits() & 0x7fffff) * 0x1p-23f, -66 + (int)(bits() %% 135)), h);
    for (float x : {0.0f, -0.0f, INFINITY, -INFINITY, NAN, FLT_MIN, 0x1p-149f, FLT_MAX, -FLT_MAX, 0x1p-63f, 0x1p65f,
                    std::nextafterf(0x1p-63f, 0.0f), std::nextafterf(0x1p65f, 0.0f)})
      check(x, h);
  }
  std::printf("%%ld\n", wrong);
}
"""


@pytest.mark.parametrize("lo,hi,more", [
    (-30, 12, ""),
    (-126, 127, "for (float h : {INFINITY, 0.0f, FLT_MAX, 0x1p127f, FLT_MIN}) hs.push_back(h);"),
    (-148, -127, "for (float h : {0x1p-149f, 3 * 0x1p-149f}) hs.push_back(h);"),
])
def test_the_corrected_product_is_the_quotient(tmp_path, lo, hi, more):
    common = hs.source("fl_common.cuh")
    code = hs.between(common, "struct Spacing {", "struct AxisF")
    out = hs.run(tmp_path, code + MAIN % {"lo": lo, "hi": hi, "more": more}).splitlines()
    assert out == ["0"], out
