"""CPU check of the POST smoother's prolongation columns, restated from
csrc/fl_multigrid.cu (smooth_tile): a lane's columns col = bx T - H + 2 lane
(even) and col + 1 read the coarse columns m - 1, m, m + 1 with m = col / 2,
column col leaning on m - 1 and column col + 1 on m + 1. A lane loads
clamp(m); m - 1 and m + 1 come from the lanes beside it, and the first and last
lane load theirs. For a cell inside the grid that must be its own (I, I2) of
pressureMultigrid.ts's prolongation, and every column read must lie inside the
coarse level; rows alike."""
from tests.test_index_maps import coarse, own_columns


def clamp(v, n):
    return min(max(v, 0), n - 1)


def test_a_lanes_columns_read_their_own_coarse_columns():
    checked = 0
    for pairs in range(0, 5):
        for halo in {2 * pairs, 2 * pairs + 2}:
            for side in (32, 64):  # rows of the two shapes; columns are always 64
                T = side - 2 * halo
                if T <= 0:
                    continue
                assert halo % 2 == 0 and T % 2 == 0
                lanes = side // 2
                for n in list(range(2, 80)) + [127, 128, 129, 511, 512, 513, 1024]:
                    cn = coarse(n)
                    for b in range(-(-n // T)):
                        first = b * T - halo
                        loaded = [clamp((first >> 1) + k, cn) for k in range(lanes)]
                        for k in range(lanes):
                            col = first + 2 * k
                            m = col >> 1
                            left = clamp(m - 1, cn) if k == 0 else loaded[k - 1]
                            right = clamp(m + 1, cn) if k == lanes - 1 else loaded[k + 1]
                            assert 0 <= min(loaded[k], left, right) and max(loaded[k], left, right) < cn
                            for cell, mine in ((col, (loaded[k], left)), (col + 1, (loaded[k], right))):
                                if 0 <= cell < n:
                                    assert own_columns(cell, cn) == mine, (pairs, side, n, b, k, cell)
                                    checked += 1
    assert checked > 100000
