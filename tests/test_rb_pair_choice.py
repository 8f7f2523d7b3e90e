"""The red-black pairs a launch and their region shape (fl_multigrid.cu,
rb_launch_pairs and rb_shape), run on the CPU: every span that a solve can ask
for, none included, on devices of several sizes."""
from tests import host_source as hs

MAIN = r"""
int main() {
  for (int sms : {38, 76, 152})
    for (int span = -1; span <= 70; span++)
      for (int n : {2, 40, 128, 320, 517, 1024, 2048}) {
        const int ny = n * 3 / 4 + 1, p = rb_launch_pairs(n, ny, span, sms);
        const RbShape s = rb_shape(n, ny, p, sms);
        const int tx = 64 - 4 * p, ty = s.nw * s.rw - 4 * p;
        std::printf("%d %d %d %d %d %d\n", sms, span, n, p, s.rw, (n + tx - 1) / tx * ((ny + ty - 1) / ty));
      }
}
"""


def test_every_span_has_a_choice(tmp_path):
    text = hs.source("fl_multigrid.cu")
    code = hs.block(text, "struct RbShape") + hs.block(text, "static RbShape rb_shape(") + hs.block(text, "int rb_launch_pairs(")
    rows = [tuple(map(int, line.split())) for line in hs.run(tmp_path, code + MAIN).splitlines()]
    assert len(rows) == 3 * 72 * 7
    for sms, span, n, pairs, rw, regions in rows:
        assert 1 <= pairs <= max(1, min(10, span)), (span, n, pairs)
        # the 16-warp shapes: one or two regions an SM, counted on the device there is
        assert rw == 8 or regions <= 2 * sms, (sms, span, n, pairs, rw, regions)
