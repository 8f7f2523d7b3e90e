"""The advection kernels that start while their predecessor drains
(fl_common.cuh, dep_wait), run on the CPU: what the predecessor writes is read
behind the wait and never by a read-only load, which is defined only for memory
that nobody writes while the kernel lives. Until a thread's wait the
predecessor's results hold NaN here; read-only loads are checked by address."""
import re

import pytest

from tests import host_source as hs

HARNESS = r"""
struct I3 { int x, y, z; };
I3 threadIdx, blockIdx, blockDim;
struct Range { const float* p; long n; };
std::vector<Range> fresh;  // what the launch before writes
long readonly_loads = 0, readonly_fresh = 0;
template <class T> T __ldg(const T* p) {
  readonly_loads++;
  for (const Range& r : fresh) readonly_fresh += (const void*)p >= r.p && (const void*)p < r.p + r.n;
  return *p;
}
std::vector<std::vector<float>> value;  // the fresh buffers' contents once it has ended
void dep_wait() { for (size_t k = 0; k < fresh.size(); k++) std::memcpy((void*)fresh[k].p, value[k].data(), 4 * fresh[k].n); }
void dep_trigger() {}
void poison() { for (const Range& r : fresh) std::fill((float*)r.p, (float*)r.p + r.n, NAN); }
#include <functional>
float uniform() { static unsigned s = 1; s = s * 1664525u + 1013904223u; return (float)(s >> 8) / 8388608.0f - 1.0f; }
"""

MAIN = r"""
using namespace fl;
int main() {
  const int nx = 13, ny = 9, D = 2, dnx = nx * D, dny = ny * D;
  const float h = %(h)s;
  const long nu = (nx + 1) * ny, nv = nx * (ny + 1), nd = 3L * dnx * dny;
  auto field = [](long n) { std::vector<float> f(n); for (float& x : f) x = uniform(); return f; };
  std::vector<float> u = field(nu), v = field(nv), q = field(nd), uh = field(nu), vh = field(nv), qh = field(nd);
  std::vector<float> uo(nu), vo(nv), qo(nd);
  std::vector<uint8_t> label(nx * ny, FLUID);
  label[3 + 4 * nx] = label[4 + 4 * nx] = SOLID;
  StepScalars sc{};
  sc.dt = 1.7f * h;
  for (float& k : sc.keep) k = 0.9f;
  const Spacing H = make_spacing(h), DH = make_spacing(h / D);
  // one thread at a time, with and without the predecessor's results before its wait
  auto run = [&](const char* what, int gx, int gy, std::vector<Range> before, std::vector<std::vector<float>*> out,
                 std::function<void()> body) {
    fresh = before;
    value.clear();
    for (const Range& r : fresh) value.emplace_back(r.p, r.p + r.n);
    readonly_loads = readonly_fresh = 0;
    std::vector<std::vector<float>> kept[2], start;
    for (auto* o : out) start.push_back(*o);
    for (int poisoned = 0; poisoned < 2; poisoned++)
      for (int j = 0; j < gy; j++)
        for (int i = 0; i < gx; i++) {
          for (size_t k = 0; k < out.size(); k++) std::copy(start[k].begin(), start[k].end(), out[k]->begin());
          dep_wait();
          if (poisoned) poison();
          blockIdx = {i, j, 0}, blockDim = {1, 1, 1}, threadIdx = {0, 0, 0};
          body();
          for (auto* o : out) kept[poisoned].push_back(*o);
        }
    bool same = kept[0].size() == kept[1].size();
    for (size_t k = 0; same && k < kept[0].size(); k++)
      same = std::memcmp(kept[0][k].data(), kept[1][k].data(), 4 * kept[0][k].size()) == 0;
    std::printf("%%s %%d %%ld %%ld\n", what, (int)same, readonly_loads, readonly_fresh);
    dep_wait();
  };
  auto vel = [&](auto mode, float* ou, float* ov, float* au, float* av) {
    constexpr int M = decltype(mode)::value;
    k_advect_velocity<M>(nx, ny, H, u.data(), v.data(), uh.data(), vh.data(), ou, ov, label.data(), &sc, au, av);
  };
  using M0 = std::integral_constant<int, 0>;
  using M1 = std::integral_constant<int, 1>;
  auto each = [&](int gx, int gy, auto f) {
    for (int j = 0; j < gy; j++)
      for (int i = 0; i < gx; i++) { blockIdx = {i, j, 0}, blockDim = {1, 1, 1}, threadIdx = {0, 0, 0}; f(); }
  };
  // the velocity's correction behind its forward pass
  each(nx + 1, ny + 1, [&] { vel(M0{}, uh.data(), vh.data(), uo.data(), vo.data()); });
  run("velocity correction", nx + 1, ny + 1, {{uh.data(), nu}, {vh.data(), nv}, {uo.data(), nu}, {vo.data(), nv}},
      {&uo, &vo}, [&] { vel(M1{}, uo.data(), vo.data(), nullptr, nullptr); });
  // the dye's forward pass behind the projection, which writes u and v
  auto dye0 = [&] {
    k_advect_dye<0, false>(nx, ny, H, dnx, dny, DH, u.data(), v.data(), q.data(), nullptr, qh.data(), label.data(), &sc,
                           nullptr, 0, 0, 0, 0, qo.data());
  };
  run("dye", dnx, dny, {{u.data(), nu}, {v.data(), nv}}, {&qh}, dye0);
  // its correction behind the forward pass
  each(dnx, dny, dye0);
  run("dye correction", dnx, dny, {{qh.data(), nd}, {qo.data(), nd}}, {&qo}, [&] {
    k_advect_dye<1, true>(nx, ny, H, dnx, dny, DH, u.data(), v.data(), q.data(), qh.data(), qo.data(), label.data(), &sc,
                          nullptr, 0, 0, 0, 0, nullptr);
  });
}
"""


@pytest.mark.parametrize("h", ["0.0625f", "0.07f"])
def test_a_predecessors_results_are_read_behind_the_wait_by_ordinary_loads(tmp_path, h):
    common, advect = hs.source("fl_common.cuh"), hs.source("fl_advect.cu")
    scalars = hs.block(common, "struct StepScalars")
    sampling = hs.between(common, "struct Spacing {", "// Programmatic dependent launch")
    for name, test in (("min_nan", "a != a || a < b"), ("max_nan", "a != a || b < a")):
        fn = hs.block(sampling, "__device__ __forceinline__ float %s(" % name)
        sampling = sampling.replace(fn, "inline float %s(float a, float b) { return %s ? a : b; }" % (name, test))
    kernels = hs.between(advect, "// advect.ts:41-55", "void launch_advect_velocity(")
    code = HARNESS + "namespace fl {\n" + hs.between(common, "constexpr uint8_t FLUID", "// Per-cell stencil code")
    code += scalars + "\n" + sampling + kernels + "}\n" + MAIN % {"h": h}
    assert not re.search(r"\basm\b", code)
    lines = hs.run(tmp_path, code).splitlines()
    assert len(lines) == 3
    for line in lines:
        what, same, loads, of_fresh = re.fullmatch(r"([a-z ]+) (\d) (\d+) (\d+)", line).groups()
        assert same == "1", "%s: a result of the launch before is read ahead of the wait" % what
        assert int(loads) > 0 and of_fresh == "0", "%s: %s read-only loads of what the launch before writes" % (what, of_fresh)
