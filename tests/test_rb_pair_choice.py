"""The red-black pairs a launch (fl_multigrid.cu, rb_launch_pairs), run on the
CPU: every span that a solve can ask for, none included."""
from tests import host_source as hs

MAIN = r"""
int main() {
  for (int span = -1; span <= 70; span++)
    for (int n : {2, 40, 128, 320, 517, 1024, 2048})
      std::printf("%d %d %d\n", span, n, rb_launch_pairs(n, n * 3 / 4 + 1, span));
}
"""


def test_every_span_has_a_choice(tmp_path):
    text = hs.source("fl_multigrid.cu")
    code = hs.block(text, "struct RbShape") + hs.block(text, "static RbShape rb_shape(") + hs.block(text, "int rb_launch_pairs(")
    rows = [tuple(map(int, line.split())) for line in hs.run(tmp_path, code + MAIN).splitlines()]
    assert len(rows) == 72 * 7
    for span, n, pairs in rows:
        assert 1 <= pairs <= max(1, min(10, span)), (span, n, pairs)
