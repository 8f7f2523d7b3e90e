// Red-black SOR and the geometric-multigrid V-cycle (src/core/
// pressureRedBlack.ts:32-113, pressureMultigrid.ts:47-320; WGSL twins
// src/gpu/redBlack.wgsl and src/gpu/multigrid.wgsl).
//
// GB300 shape of the V-cycle:
//   * Fine levels: ONE launch per level on the way down and one on the way up.
//     Each CTA loads its tile plus a halo into registers and runs all of
//     the level's red-black half-sweeps there (temporal blocking: half-sweep s
//     is valid on the region shrunk by s+1 cells, so a halo of 2*pairs+1
//     leaves the tile and a one-cell ring valid after the last sweep). The
//     down kernel then forms the residual and restricts it to the coarse rhs;
//     the up kernel first adds the prolonged coarse correction. Every cell
//     sees exactly the operations, in exactly the order, of the reference's
//     sequence of separate passes, so the result is identical to it.
//     x is double-buffered per level: a tile reads its halo's pre-sweep values
//     while neighbouring tiles write.
//   * Coarse levels (from the first level with <= coarse_cells cells): ONE
//     single-CTA launch runs the rest of the V-cycle entirely in shared
//     memory, including the coarsest-level sweeps.
//   * Labels become one byte per cell of stencil links (fl_common.cuh), built
//     per level when labels change (pressureMultigrid.ts:302-310 rebuilt them
//     every solve; stepGpu.ts:498 only on change, as here).
#include <cfloat>
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>

#include "fl_internal.h"

namespace fl {

constexpr int MODE_PLAIN = 0, MODE_PRE = 1, MODE_POST = 2;
constexpr int MAX_LEVELS = 24;

// ------------------------------------------------------------ label codes

// The stencil code of cell (i, j) of a level.
__device__ __forceinline__ unsigned cell_code(const uint8_t* label, int nx, int ny, int i, int j) {
  const int k = i + j * nx;
  unsigned c = label[k] & 3u;
  if (i + 1 < nx && label[k + 1] != SOLID) c |= LINK_XP;
  if (i > 0 && label[k - 1] != SOLID) c |= LINK_XM;
  if (j + 1 < ny && label[k + nx] != SOLID) c |= LINK_YP;
  if (j > 0 && label[k - nx] != SOLID) c |= LINK_YM;
  return c;
}

// pressureMultigrid.ts:92-110 (multigrid.wgsl:259-286): the coarse label of
// the 2 x 2 cells from (i, j) on (even), Air > Fluid > Solid.
__device__ __forceinline__ uint8_t coarse_label(const uint8_t* label, int nx, int ny, int i, int j) {
  bool air = false, fluid = false;
  for (int dj = 0; dj < 2; dj++)
    for (int di = 0; di < 2; di++) {
      if (i + di >= nx || j + dj >= ny) continue;
      const uint8_t l = label[i + di + (j + dj) * nx];
      air = air || l == AIR;
      fluid = fluid || l == FLUID;
    }
  return air ? AIR : (fluid ? FLUID : SOLID);
}

// A level's stencil codes and, where `coarse` is set, the next level's labels.
// only_if (when set): the kernel does nothing unless *only_if is nonzero
__global__ void k_build_codes(int nx, int ny, const uint8_t* __restrict__ label, uint8_t* __restrict__ code,
                              uint8_t* __restrict__ coarse, const int* only_if) {
  if (only_if != nullptr && *only_if == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  code[i + j * nx] = (uint8_t)cell_code(label, nx, ny, i, j);  // 32-bit offsets: a level holds fewer than 2^31 cells
  if (coarse != nullptr && ((i | j) & 1) == 0)
    coarse[(i >> 1) + (j >> 1) * ((nx + 1) / 2)] = coarse_label(label, nx, ny, i, j);
}

// The uploaded labels against the current ones: copies the cells that
// differ and raises *flag if there were any (16 bytes per thread step; the
// buffers come from cudaMalloc, so the 16-byte body is aligned).
__global__ void __launch_bounds__(256) k_label_sync(const uint8_t* __restrict__ in, uint8_t* __restrict__ cur, long n,
                                                    int* flag) {
  bool changed = false;
  const long stride = (long)gridDim.x * blockDim.x;
  const long t0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const uint4* in4 = reinterpret_cast<const uint4*>(in);
  uint4* cur4 = reinterpret_cast<uint4*>(cur);
  for (long k = t0; k < n / 16; k += stride) {
    const uint4 a = in4[k], b = cur4[k];
    if (a.x != b.x || a.y != b.y || a.z != b.z || a.w != b.w) {
      cur4[k] = a;
      changed = true;
    }
  }
  for (long k = 16 * (n / 16) + t0; k < n; k += stride)
    if (in[k] != cur[k]) {
      cur[k] = in[k];
      changed = true;
    }
  if (__syncthreads_or(changed) && threadIdx.x == 0) atomicOr(flag, 1);
}

__global__ void k_label_cond(int* flag, cudaGraphConditionalHandle h) {
  cudaGraphSetConditional(h, *flag != 0 ? 1u : 0u);
  *flag = 0;
}

void launch_label_sync(cudaStream_t s, const uint8_t* in, uint8_t* cur, long n, int* flag) {
  const long blocks = std::min(std::max(1L, (n / 16 + 255) / 256), 152L * 4);
  k_label_sync<<<(unsigned)blocks, 256, 0, s>>>(in, cur, n, flag);
}

void launch_label_cond(cudaStream_t s, int* flag, cudaGraphConditionalHandle h) { k_label_cond<<<1, 1, 0, s>>>(flag, h); }

struct SmoothArgs {
  int nx, ny;
  const float* xin;
  float* xout;
  const float* b;
  const uint8_t* code;
  float scale, omega;
  const float* scale_dev;  // PLAIN: when set, the scale is read here (the step's scalars)
  float* bc;  // PRE: coarse rhs target
  int cnx, cny;
  const float* ec;  // POST: coarse correction
  StepAccum* acc;   // POST: residual norm accumulation (may be null)
  int x_is_zero;    // PRE on a coarse level: x starts at zero (pressureMultigrid.ts:175)
  int pairs, halo;  // sweep pairs, and the region's halo (smooth_halo)
};

// s / count for rc = (RN(1 / count), -count), count 1..4, without a branch or
// a test of the count: the correctly rounded quotient formed with two FMAs
// (the correction step for a divisor known in advance: Markstein; Brisebarre,
// Muller and Raina, IEEE Trans. Computers 2004): q0 = RN(s * RN(1 / count)),
// r = s - count q0 (exact), q = RN(q0 + r * RN(1 / count)). For 1, 2 and 4 q0
// is the quotient, r is 0 and the second step changes nothing. An infinite s
// has a NaN remainder, which fmaxf turns into a finite number: the quotient
// then stays infinite. Equals IEEE division for every float (for 3 checked
// exhaustively) but for the sign of a zero.
__device__ __forceinline__ float over_links(float s, float2 rc) {
  const float q0 = __fmul_rn(s, rc.x);
  const float r = fmaxf(__fmaf_rn(rc.y, q0, s), -3.402823466e+38f);
  return __fmaf_rn(r, rc.x, q0);
}

// over_links' factors of a cell with this code: (0, 0) unless it is fluid
// with a link, which the sweeps update (pressureRedBlack.ts:52-66).
__device__ __forceinline__ float2 link_factors(int code) {
  const int cnt = code_count((uint8_t)code);
  const bool on = (code & 3) == FLUID && cnt > 0;
  return make_float2(on ? 1.0f / (float)cnt : 0.0f, on ? -(float)cnt : 0.0f);
}

// Temporally blocked red-black smoother. One CTA of NW warps owns a region of
// 64 columns x NW * RW rows: its tile plus a halo of H cells all round (H
// even). Lane l of a warp owns the columns 2l and 2l + 1 of the warp's RW
// rows, value and rhs in registers for the whole launch. A cell's vertical
// neighbours are then the same lane's registers, one horizontal neighbour is
// the lane's other column and the other one shuffle away; only the first and
// last row of each warp go through shared memory, one value a lane and
// half-sweep (edge[c]: colour c's cells of those rows, written by the
// half-sweeps of colour c and read by those of the other colour, so one
// barrier a half-sweep orders both). The region starts at even coordinates:
// the colour-c cell of row r is column (c + r) & 1 of the pair in every lane,
// known at compile time, and the 2 x 2 children of a coarse cell belong to
// one lane.
//
// Every half-sweep updates every updatable cell of its colour. Half-sweep s
// is correct on the region shrunk by s + 1 cells (beyond the region's border
// a cell sees some finite value), so a halo of 2 pairs leaves the tile with
// exactly the values that the sequential sweeps produce, and 2 pairs + 1 a
// ring around it for the residual (rounded up to even). From x = 0 the first
// half-sweep sees nothing but zeros, inside the region and beyond: it is
// correct everywhere, and 2 pairs serve the residual too (smooth_halo).
//
// Bound by instruction issue and, where a level has few regions, by the
// latency of one region (load, 2 pairs half-sweeps of ~150 to 250 cycles,
// residual). Launches chained in a graph, with x in shared memory -> in
// registers: V(3,3) PRE from zero / POST at 2048^2 44.3 / 45.8 -> 14.8 / 17.4
// us, 1024^2 12.0 / 12.5 -> 5.8 / 6.2, 256^2 3.4 / 3.5 -> 2.6 / 3.1; four SOR
// pairs at 1024^2 with obstacles 16.6 -> 8.9.
//
// The shapes: 8 warps of 8 rows (a 64 x 64 region) spend the fewest
// instructions a cell; 16 warps of 2 rows (64 x 32) have the shortest chain
// of updates a warp, for levels whose 64 x 64 regions would leave SMs idle or
// give a few of them a second one (fewer than smooth_small: 176 on 152 SMs).
// PRE in the large and the small regions: 512^2 (100 regions) 4.2 against 3.2
// us, 640^2 (169) 4.9 against 4.2, 704^2 (196) 4.9 against 4.9, 1024^2 (400) 6.1
// against 7.7; POST at 704^2 5.4 against 5.8. 8 x 4 and 16 x 4 lay between.
static long smooth_small(int sms) { return 22L * sms / 19; }

template <int NW, int RW>
struct SmoothShared {
  float edge[2][NW + 2][2][32];        // [colour][warp + 1][first / last row][lane]; beyond the region: 0
  float2 rc[2 * RW][32 * NW];          // (RN(1 / count), -count) of a cell's links, (0, 0) where it is not updated
  float2 lut[64];                      // that pair for each code
};

// One region of the smoother, region (bx, by) of the level; called by one
// whole block (every thread, in step).
template <int MODE, int NW, int RW>
__device__ __forceinline__ void smooth_tile(const SmoothArgs& a, int bx, int by, SmoothShared<NW, RW>& sh) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nx = a.nx, ny = a.ny, H = a.halo;
  const int TX = 64 - 2 * H, TY = RW * NW - 2 * H;
  const int col = bx * TX - H + 2 * lane;      // even
  const int row = by * TY - H + RW * w;        // even
  // rows of an even width start at multiples of 8 bytes, so a lane's pair is
  // one 8-byte access (the levels' buffers come from cudaMalloc)
  const bool pair = (nx & 1) == 0;
  constexpr unsigned OUTSIDE2 = CODE_OUTSIDE | (unsigned)CODE_OUTSIDE << 8;
  constexpr unsigned FULL2 = 0x3c3cu;  // two fluid cells with four links each

  float x[RW][2], b[RW][2];
  unsigned cd[RW];  // the two cells' codes
  auto load_codes = [&](int r) {
    const int gj = row + r, k = col + gj * nx;  // 32-bit offsets: a level holds fewer than 2^31 cells
    cd[r] = OUTSIDE2;
    if ((unsigned)gj >= (unsigned)ny) return;
    if (pair) {
      if ((unsigned)col < (unsigned)nx) cd[r] = *reinterpret_cast<const unsigned short*>(a.code + k);
    } else {
#pragma unroll
      for (int o = 0; o < 2; o++)
        if ((unsigned)(col + o) < (unsigned)nx)
          cd[r] = (cd[r] & (o ? 0x00ffu : 0xff00u)) | (unsigned)a.code[k + o] << (8 * o);
    }
  };
  auto load_row = [&](const float* f, float* v, int gj) {
    const int k = col + gj * nx;
    v[0] = v[1] = 0.0f;
    if ((unsigned)gj >= (unsigned)ny) return;
    if (pair) {
      if ((unsigned)col < (unsigned)nx) {
        const float2 q = *reinterpret_cast<const float2*>(f + k);
        v[0] = q.x;
        v[1] = q.y;
      }
    } else {
#pragma unroll
      for (int o = 0; o < 2; o++)
        if ((unsigned)(col + o) < (unsigned)nx) v[o] = f[k + o];
    }
  };
  auto load_b = [&](int r) { load_row(a.b, b[r], row + r); };
  auto load_x = [&](int r) {
    x[r][0] = x[r][1] = 0.0f;
    if (!a.x_is_zero) load_row(a.xin, x[r], row + r);
  };
  // Before dep_wait: the codes (built long before), and on the way up b and x,
  // which this level's PRE launch and the finer one's wrote; only the coarse
  // correction comes from the launch before. On the way down b does. Of a row
  // of SOR launches (the first is an ordinary one) only x does.
#pragma unroll
  for (int r = 0; r < RW; r++) load_codes(r);
  if (MODE != MODE_PRE) {
#pragma unroll
    for (int r = 0; r < RW; r++) load_b(r);
  }
  if (MODE == MODE_POST) {
#pragma unroll
    for (int r = 0; r < RW; r++) load_x(r);
  }
  const float scale = MODE == MODE_PLAIN && a.scale_dev ? *a.scale_dev : a.scale;
  if (tid < 64) sh.lut[tid] = link_factors(tid);
  if (w == 0) {
    sh.edge[0][0][1][lane] = sh.edge[1][0][1][lane] = 0.0f;
    sh.edge[0][NW + 1][0][lane] = sh.edge[1][NW + 1][0][lane] = 0.0f;
  }
  dep_wait();
  dep_trigger();
  if (MODE == MODE_PRE) {
#pragma unroll
    for (int r = 0; r < RW; r++) load_b(r);
  }
  if (MODE != MODE_POST) {
#pragma unroll
    for (int r = 0; r < RW; r++) load_x(r);
  }
  if constexpr (MODE == MODE_POST) {
    // pressureMultigrid.ts:192-207 — a fluid cell's x += 9/16, 3/16, 3/16,
    // 1/16 of e at coarse columns (I, I2) and rows (J, J2), I = i >> 1, I2 =
    // I + 1 (odd i) or I - 1 (even i), clamped. The pair of columns 2m, 2m+1
    // reads coarse columns m-1, m, m+1: each lane loads its m, the others
    // come by shuffle (the first and last lane load theirs). The 8 rows read
    // 6 coarse rows. The clamps change nothing for a cell in the grid.
    const int m = col >> 1, J0 = row >> 1;
    const int cm = min(max(m, 0), a.cnx - 1);
    const int ce = min(max(lane == 0 ? m - 1 : m + 1, 0), a.cnx - 1);
    const bool end = lane == 0 || lane == 31;
    float eL[RW / 2 + 2], eM[RW / 2 + 2], eR[RW / 2 + 2];  // coarse rows J0 - 1 .. J0 + RW / 2
#pragma unroll
    for (int q = 0; q < RW / 2 + 2; q++) {
      const float* e = a.ec + min(max(J0 - 1 + q, 0), a.cny - 1) * a.cnx;
      eM[q] = e[cm];
      eL[q] = end ? e[ce] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < RW / 2 + 2; q++) {
      const float l = __shfl_up_sync(0xffffffffu, eM[q], 1), r = __shfl_down_sync(0xffffffffu, eM[q], 1);
      eR[q] = lane == 31 ? eL[q] : r;
      eL[q] = lane == 0 ? eL[q] : l;
    }
#pragma unroll
    for (int r = 0; r < RW; r++) {
      const int q = 1 + r / 2, f = (r & 1) ? q + 1 : q - 1;  // an even row leans on the coarse row below, an odd one above
      const float p0 = 0.5625f * eM[q] + 0.1875f * (eL[q] + eM[f]) + 0.0625f * eL[f];
      const float p1 = 0.5625f * eM[q] + 0.1875f * (eR[q] + eM[f]) + 0.0625f * eR[f];
      const float x0 = x[r][0] + p0, x1 = x[r][1] + p1;
      x[r][0] = (cd[r] & 3u) == FLUID ? x0 : x[r][0];
      x[r][1] = (cd[r] & 0x300u) == 0u ? x1 : x[r][1];
    }
  }

  __syncthreads();

  // the warp's form: every cell fluid with four links, or not (then its
  // cells' link counts go to shared memory, and the update has no branches:
  // a lane-divergent one in each of its cells cost ~100 cycles an update)
  unsigned odd = 0u;
#pragma unroll
  for (int r = 0; r < RW; r++) odd |= cd[r] ^ FULL2;
  const bool full = __all_sync(0xffffffffu, odd == 0u);
  if (!full) {
#pragma unroll
    for (int r = 0; r < RW; r++)
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const unsigned c = cd[r] >> (8 * o) & 0x3fu;
        sh.rc[2 * r + o][tid] = sh.lut[c];
        // Solid cells (and cells outside the grid) are exactly the
        // neighbours no link points to: they hold +0.0, so that a sum adds
        // all four neighbours without a test (x + 0.0 is x, but for the sign
        // of an exact zero). A solid cell's own value is written back from xin.
        x[r][o] = (c & 3u) == SOLID ? 0.0f : x[r][o];
      }
  }
  if constexpr (MODE == MODE_PLAIN) {
#pragma unroll
    for (int r = 0; r < RW; r++) {
      b[r][0] = scale * b[r][0];
      b[r][1] = scale * b[r][1];
    }
  }
  // colour c in the warp's first row (even) is column c, in its last (odd) column 1 - c
  auto publish = [&](int c) {
    sh.edge[c][w + 1][0][lane] = x[0][c];
    sh.edge[c][w + 1][1][lane] = x[RW - 1][1 - c];
  };
  publish(0);
  publish(1);
  __syncthreads();

  const float omega = a.omega, keep = 1.0f - omega;
  // With omega = 1 (the multigrid's relaxation) the blend (1 - omega) x +
  // omega pGS is pGS for every finite x, up to the sign of an exact zero
  // (0 x + (-0) is +0), which compares equal: the sweeps then skip it.
  auto half_sweep = [&](auto unit, auto colour) {
    constexpr bool UNIT = decltype(unit)::value;
    constexpr int c = decltype(colour)::value;
    const float above = sh.edge[1 - c][w + 2][0][lane], below = sh.edge[1 - c][w][1][lane];
    // pressureRedBlack.ts:52-66, sum order +x, -x, +y, -y
    auto rhs = [&](int r, int o) {
      const float own = x[r][1 - o];
      const float far = o == 0 ? __shfl_up_sync(0xffffffffu, own, 1) : __shfl_down_sync(0xffffffffu, own, 1);
      float sum = o == 0 ? own + far : far + own;
      sum += r < RW - 1 ? x[r + 1][o] : above;
      sum += r > 0 ? x[r - 1][o] : below;
      // the multigrid's scale is -1: sum - (-1) b
      return MODE == MODE_PLAIN ? sum - b[r][o] : sum + b[r][o];
    };
    if (full) {
#pragma unroll
      for (int r = 0; r < RW; r++) {
        const int o = (c + r) & 1;
        const float pgs = rhs(r, o) * 0.25f;
        x[r][o] = UNIT ? pgs : keep * x[r][o] + omega * pgs;
      }
    } else {
#pragma unroll
      for (int r = 0; r < RW; r++) {
        const int o = (c + r) & 1;
        const float2 rc = sh.rc[2 * r + o][tid];
        const float pgs = over_links(rhs(r, o), rc);
        const float nv = UNIT ? pgs : keep * x[r][o] + omega * pgs;
        x[r][o] = rc.x != 0.0f ? nv : x[r][o];
      }
    }
    publish(c);
    __syncthreads();
  };
  auto sweeps = [&](auto unit) {
#pragma unroll 1
    for (int k = 0; k < a.pairs; k++) {
      half_sweep(unit, std::integral_constant<int, 0>{});
      half_sweep(unit, std::integral_constant<int, 1>{});
    }
  };
  if (omega == 1.0f)
    sweeps(std::true_type{});
  else
    sweeps(std::false_type{});

  // the tile's cells of this thread: all columns of the pair, rows lo..hi-1
  const bool mine = lane >= H / 2 && lane < 32 - H / 2;
  const int lo = max(H - RW * w, 0), hi = min(min(RW * NW - H - RW * w, RW), ny - row);

  if (MODE == MODE_PRE || (MODE == MODE_POST && a.acc != nullptr)) {
    // r = b - (count*x - sum), 0 off-fluid (pressureMultigrid.ts:117-151), as
    // b + (-count*x + sum): every operation the negation of the same rounding
    double rsq = 0.0;
    unsigned long long rn = 0;
    auto residuals = [&](auto four) {
      constexpr bool FOUR = decltype(four)::value;
      [[maybe_unused]] float even = 0.0f;  // the even row's two residuals, summed
#pragma unroll
      for (int r = 0; r < RW; r++) {
        float res[2];
        const float left = __shfl_up_sync(0xffffffffu, x[r][1], 1), right = __shfl_down_sync(0xffffffffu, x[r][0], 1);
#pragma unroll
        for (int o = 0; o < 2; o++) {
          float sum = o == 0 ? x[r][1] + left : right + x[r][0];
          sum += r < RW - 1 ? x[r + 1][o] : sh.edge[o][w + 2][0][lane];
          sum += r > 0 ? x[r - 1][o] : sh.edge[1 - o][w][1][lane];
          const float n = FOUR ? -4.0f : sh.rc[2 * r + o][tid].y;
          const float v = b[r][o] + (n * x[r][o] + sum);
          res[o] = FOUR || n != 0.0f ? v : 0.0f;
          if (MODE == MODE_POST && (FOUR || n != 0.0f) && mine && r >= lo && r < hi) {
            const double d = f2d_exact(res[o]);
            rsq = fma(d, d, rsq);
            rn += 1;
          }
        }
        if constexpr (MODE == MODE_PRE) {
          // pressureMultigrid.ts:156-178: coarse b = sum of the children's
          // residuals (a child outside the grid is 0)
          if ((r & 1) == 0) {
            even = res[0] + res[1];
          } else {
            const float sum = (even + res[0]) + res[1];
            const int I = col >> 1, J = (row + r) >> 1;
            if (mine && r >= lo && r - 1 < hi && I < a.cnx) a.bc[I + J * a.cnx] = sum;
          }
        }
      }
    };
    if (full)
      residuals(std::true_type{});
    else
      residuals(std::false_type{});
    if constexpr (MODE == MODE_POST) {
      __shared__ double red[32];
      __shared__ unsigned long long redn[32];
      const double bsum = block_sum(rsq, red);
      const unsigned long long bn = block_sum_u64(rn, redn);
      if (tid == 0) {
        atomicAdd(&a.acc->res_sq, bsum);
        atomicAdd(&a.acc->n_res, bn);
      }
    }
  }

  if (a.xout == nullptr || !mine) return;
#pragma unroll
  for (int r = 0; r < RW; r++) {
    if (r < lo || r >= hi) continue;
    const int k = col + (row + r) * nx;
    if (!full && !a.x_is_zero) {
#pragma unroll
      for (int o = 0; o < 2; o++)
        if ((cd[r] >> (8 * o) & 3u) == SOLID && col + o < nx) x[r][o] = a.xin[k + o];
    }
    if (pair) {
      if (col < nx) *reinterpret_cast<float2*>(a.xout + k) = make_float2(x[r][0], x[r][1]);
    } else {
      if (col < nx) a.xout[k] = x[r][0];
      if (col + 1 < nx) a.xout[k + 1] = x[r][1];
    }
  }
}

// The halo (even) that leaves the tile correct: see smooth_tile.
__host__ __device__ static int smooth_halo(int mode, int pairs, bool x_is_zero, bool residual) {
  if (mode == MODE_PRE && x_is_zero) return 2 * pairs;
  return mode == MODE_PRE || residual ? 2 * pairs + 2 : 2 * pairs;
}

template <int MODE, int NW, int RW>
__global__ void __launch_bounds__(32 * NW, RW == 8 ? 24 / NW : 32 / NW) k_smooth(SmoothArgs a) {
  __shared__ SmoothShared<NW, RW> sh;
  smooth_tile<MODE, NW, RW>(a, blockIdx.x, blockIdx.y, sh);
}

// ----------------------------------------------------- single-CTA coarse tail

// The coarsest levels (both sides <= fl_params.mg_tail_side, at most 64) run
// in ONE CTA. Each level lies in a square frame of a power-of-two side F (the
// tail's first level in the smallest frame that holds it, the next in half of
// that, and so on; cells beyond the level are coded outside), so that every
// index is known at compile time. A lane owns a pair of columns (2i, 2i + 1)
// of one row: one cell of each colour. A row takes F / 2 lanes, a warp 64 / F
// rows, and the frame's first F^2 / 64 warps (at most 32; at F = 64 each of
// them has two row groups) take part in a level's phases, synchronising on the
// frame's own named barrier. A pair's index in its frame, row * F / 2 + i, is
// then the thread's index (+ 1024 in its second row group).
//
// The CTA is one chain of dependent phases, so their latency is all that
// counts. A level's values, rhs and codes stay in its owners' registers from
// the pre-smoothing to the post-smoothing. In a half-sweep a cell's one
// horizontal neighbour is the lane's other value, the other one shuffle away,
// the vertical ones two shared-memory loads, or two shuffles in a frame that
// one warp holds, which then needs no shared memory and no barrier. An
// unlinked neighbour is masked to +0.0 (which leaves a sum's bits unchanged
// but for the sign of an exact zero), and over_links divides without a branch.
// The fine level's owners write their residuals by column into an exchange
// buffer, from which the coarse level's owners sum them (two 16-byte loads a
// pair); the coarse level's result comes back through its own.
//
// Coarser levels are owned by a subset of the finer level's warps, so the
// barrier that ends a phase on a level also orders it before every
// coarser-level phase.
//
// Measured, 32^2 to 8^2 with V(3,3) and 16 coarsest pairs, launches chained in
// a graph: 6.0 us, against 16.1 with the values, codes and geometry in shared
// memory and fetched again in every phase. From 64^2 on: 13.3 us, hardly less
// than with the 64^2 level's own two launches (14.1), and 1024^2 V-cycles 45.0
// against 45.6: the tail stays at 32^2.
constexpr int TAIL_LEVELS = 7;  // at most 64 a side

struct CoarseArgs {
  int nx, ny, nlev;       // of the tail's first level; levels
  int frame;              // its frame's side
  const uint16_t* codes;  // every frame's codes (k_tail_codes)
  const float* b_top;
  float* x_top;
  int x_is_zero;
  int pre, post, coarse_sweeps;
  float omega;
  StepAccum* acc;
};

// Default first level of the single-CTA tail (fl_params.mg_tail_side = 0):
// levels with both sides <= 32.
constexpr int TAIL_SIDE_DEFAULT = 32;

template <int F>
struct Frame {
  static constexpr int LPR = F > 1 ? F / 2 : 1;                       // lanes a row
  static constexpr int PAIRS = F * LPR;
  static constexpr int NP = PAIRS < 32 ? 32 : PAIRS;                  // with the warp's idle lanes
  static constexpr int WARPS = NP > 1024 ? 32 : NP / 32;
  static constexpr int SLOTS = NP > 1024 ? 2 : 1;
  static constexpr bool ONE = WARPS == 1;
  static constexpr int BAR = F == 64 ? 1 : F == 32 ? 2 : 3;           // named barrier (64, 32 and 16)
  // shared memory, in floats: the frames one after the other, smallest first;
  // the exchange buffer (a float2 a pair, by column), then the values by
  // colour, a row of lanes before and after each
  static constexpr int OFF = Frame<F / 2>::OFF + Frame<F / 2>::FLOATS;
  static constexpr int FLOATS = 2 * NP + (ONE ? 0 : 2 * (NP + 2 * LPR));
  static constexpr int CODES = Frame<F / 2>::CODES + Frame<F / 2>::NP;  // offset of the frame's codes
};
template <>
struct Frame<0> {
  static constexpr int NP = 0, OFF = 0, FLOATS = 0, CODES = 0;
};
constexpr int TAIL_CODES = Frame<64>::CODES + Frame<64>::NP;

// What a lane keeps of one pair, by colour.
struct TailPair {
  float x[2], b[2];
  unsigned code;  // byte c: colour c's
};

__device__ __forceinline__ float masked(float v, int m) { return __int_as_float(__float_as_int(v) & m); }

template <int F>
struct TailLevel {
  using G = Frame<F>;
  float2* r;       // exchange buffer
  float* v[2];     // values by colour
  int tid, lane;
  TailPair q[G::SLOTS];

  __device__ __forceinline__ TailLevel(float* smem, int tid_) : tid(tid_), lane(tid_ & 31) {
    r = reinterpret_cast<float2*>(smem + G::OFF);
    v[0] = smem + G::OFF + 2 * G::NP + G::LPR;
    v[1] = v[0] + G::NP + 2 * G::LPR;
  }
  __device__ __forceinline__ int pair(int s) const { return tid + 1024 * s; }
  __device__ __forceinline__ int row(int s) const { return pair(s) / G::LPR; }
  __device__ __forceinline__ void bar() const {
    if (G::ONE)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"n"(G::BAR), "n"(32 * G::WARPS) : "memory");
  }
  // the neighbour sum of pair s's colour-c cell, order +x, -x, +y, -y (the
  // first two commute)
  __device__ __forceinline__ float sum(int s, int c) const {
    const unsigned k = q[s].code >> (8 * c);
    const int o = (c + row(s)) & 1;  // the pair's column of colour c
    const int xp = -(int)(k >> 2 & 1u), xm = -(int)(k >> 3 & 1u);
    const float own = q[s].x[1 - c];
    const float far = __shfl_sync(0xffffffffu, own, lane + (o ? 1 : -1));
    float up, dn;
    if constexpr (G::ONE) {
      up = __shfl_sync(0xffffffffu, own, lane + G::LPR);
      dn = __shfl_sync(0xffffffffu, own, lane - G::LPR);
    } else {
      up = v[1 - c][pair(s) + G::LPR];
      dn = v[1 - c][pair(s) - G::LPR];
    }
    return ((masked(own, o ? xm : xp) + masked(far, o ? xp : xm)) + masked(up, -(int)(k >> 4 & 1u))) +
           masked(dn, -(int)(k >> 5 & 1u));
  }
  __device__ __forceinline__ void publish(int s, int c) const {
    if constexpr (!G::ONE) v[c][pair(s)] = q[s].x[c];
  }
  __device__ __forceinline__ void publish_all() const {
#pragma unroll
    for (int s = 0; s < G::SLOTS; s++) publish(s, 0), publish(s, 1);
    bar();
  }
  __device__ __forceinline__ void exchange(int s, float c0, float c1) const {
    r[pair(s)] = (row(s) & 1) ? make_float2(c1, c0) : make_float2(c0, c1);  // odd rows: colour 0 is column 1
  }
  __device__ __forceinline__ float2 factors(const float2* lut, int s, int c) const {
    return lut[q[s].code >> (8 * c) & 0x3fu];
  }
  // r = b - (count*x - sum), 0 where the cell is not updated (pressureMultigrid.ts:117-151)
  __device__ __forceinline__ float residual(const float2* lut, int s, int c) const {
    const float2 rc = factors(lut, s, c);
    const float res = q[s].b[c] + (rc.y * q[s].x[c] + sum(s, c));
    return rc.x != 0.0f ? res : 0.0f;
  }
  // `pairs` red-black sweep pairs; from_zero: the values are 0 and not yet
  // published, so the first half-sweep has no neighbours to add.
  __device__ __forceinline__ void sweeps(const float2* lut, int pairs, float omega, bool from_zero) {
    float2 rc[G::SLOTS][2];
#pragma unroll
    for (int s = 0; s < G::SLOTS; s++)
#pragma unroll
      for (int c = 0; c < 2; c++) rc[s][c] = factors(lut, s, c);
    const float keep = 1.0f - omega;
    auto run = [&](auto unit) {
      constexpr bool UNIT = decltype(unit)::value;  // omega = 1: pGS itself (see smooth_tile)
#pragma unroll 1
      for (int k = 0; k < pairs; k++) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
#pragma unroll
          for (int s = 0; s < G::SLOTS; s++) {
            float t = q[s].b[c];
            if (c == 1 || k > 0 || !from_zero) t = sum(s, c) + t;
            const float pgs = over_links(t, rc[s][c]);
            const float nv = UNIT ? pgs : keep * q[s].x[c] + omega * pgs;
            q[s].x[c] = rc[s][c].x != 0.0f ? nv : q[s].x[c];
            publish(s, c);
          }
          if (!G::ONE) bar();
        }
      }
    };
    if (omega == 1.0f)
      run(std::true_type{});
    else
      run(std::false_type{});
  }
};

// The V-cycle from frame F down (frames larger than the tail's first one pass
// the call on); rsq, rn: the residual norm of the first level when a.acc asks
// for it.
template <int F>
__device__ __forceinline__ void tail_frame(const CoarseArgs& a, float* smem, const float2* lut, const unsigned* code,
                                           int tid, double& rsq, unsigned long long& rn) {
  using G = Frame<F>;
  if (F > a.frame) {
    if constexpr (F > 1) tail_frame<F / 2>(a, smem, lut, code, tid, rsq, rn);
    return;
  }
  if (tid >= 32 * G::WARPS) return;
  TailLevel<F> L(smem, tid);
  const int depth = __popc(a.frame - 1) - __popc(F - 1);  // the level below the tail's first
  const bool last = depth == a.nlev - 1, top = depth == 0;
  const int nx = ((a.nx - 1) >> depth) + 1, ny = ((a.ny - 1) >> depth) + 1;
  constexpr int LOG = F == 64 ? 6 : F == 32 ? 5 : F == 16 ? 4 : F == 8 ? 3 : F == 4 ? 2 : F == 2 ? 1 : 0;
#pragma unroll
  for (int s = 0; s < G::SLOTS; s++) {
    TailPair& q = L.q[s];
    q.code = code[s == 1 ? 7 : LOG];
    q.x[0] = q.x[1] = 0.0f;
    float2 b = make_float2(0.0f, 0.0f);  // by column
    const int j = L.row(s), i = 2 * (L.pair(s) & (G::LPR - 1));
    if (top) {
      if (j < ny && i < nx) {
        const int k = i + j * nx;
        b.x = a.b_top[k];
        if (i + 1 < nx) b.y = a.b_top[k + 1];
        if (!a.x_is_zero) {
          const float x0 = a.x_top[k], x1 = i + 1 < nx ? a.x_top[k + 1] : 0.0f;
          q.x[0] = (j & 1) ? x1 : x0;
          q.x[1] = (j & 1) ? x0 : x1;
        }
      }
    } else if (F < 64 && L.pair(s) < G::PAIRS) {
      // the coarse rhs: the sum of the children's residuals
      // (pressureMultigrid.ts:156-178; those outside the level are 0)
      constexpr int FF = F < 64 ? 2 * F : 64;
      const float2* f = reinterpret_cast<const float2*>(smem + Frame<FF>::OFF) + 2 * j * Frame<FF>::LPR + i;
      const float2 lo = f[0], hi = f[Frame<FF>::LPR];
      b.x = ((lo.x + lo.y) + hi.x) + hi.y;
      if (F > 1) {
        const float2 lo2 = f[1], hi2 = f[Frame<FF>::LPR + 1];
        b.y = ((lo2.x + lo2.y) + hi2.x) + hi2.y;
      }
    }
    q.b[0] = (j & 1) ? b.y : b.x;
    q.b[1] = (j & 1) ? b.x : b.y;
  }
  const int sweeps = last ? a.coarse_sweeps : a.pre;
  const bool from_zero = !top || a.x_is_zero;
  if (!from_zero || sweeps == 0) L.publish_all();
  L.sweeps(lut, sweeps, a.omega, from_zero);
  if constexpr (F > 1) {
    if (!last) {
#pragma unroll
      for (int s = 0; s < G::SLOTS; s++) L.exchange(s, L.residual(lut, s, 0), L.residual(lut, s, 1));
      L.bar();
      tail_frame<F / 2>(a, smem, lut, code, tid, rsq, rn);
      L.bar();  // the coarse level's owners are done with it
      // prolongation (9/16, 3/16, 3/16, 1/16, pressureMultigrid.ts:192-207)
      const float* e = smem + Frame<F / 2>::OFF;
      constexpr int ES = 2 * Frame<F / 2>::LPR;
      const int cx = (nx + 1) / 2 - 1, cy = (ny + 1) / 2 - 1;
#pragma unroll
      for (int s = 0; s < G::SLOTS; s++) {
        TailPair& q = L.q[s];
        const int j = L.row(s), I = min(L.pair(s) & (G::LPR - 1), cx);
        const int J = min(j >> 1, cy), J2 = (j & 1) ? min(J + 1, cy) : max(J - 1, 0);
        const int left = max(I - 1, 0), right = min(I + 1, cx);
        const float m1 = e[J * ES + I], l1 = e[J * ES + left], r1 = e[J * ES + right];
        const float m2 = e[J2 * ES + I], l2 = e[J2 * ES + left], r2 = e[J2 * ES + right];
        const float add0 = 0.5625f * m1 + 0.1875f * (l1 + m2) + 0.0625f * l2;
        const float add1 = 0.5625f * m1 + 0.1875f * (r1 + m2) + 0.0625f * r2;
        const float x0 = q.x[0] + ((j & 1) ? add1 : add0), x1 = q.x[1] + ((j & 1) ? add0 : add1);
        q.x[0] = (q.code & 3u) == FLUID ? x0 : q.x[0];
        q.x[1] = (q.code >> 8 & 3u) == FLUID ? x1 : q.x[1];
      }
      if (!G::ONE || a.post == 0) L.publish_all();
      L.sweeps(lut, a.post, a.omega, false);
    }
  }
  if (!top) {
#pragma unroll
    for (int s = 0; s < G::SLOTS; s++) L.exchange(s, L.q[s].x[0], L.q[s].x[1]);
    return;
  }
#pragma unroll
  for (int s = 0; s < G::SLOTS; s++) {
    const TailPair& q = L.q[s];
    if (a.acc != nullptr)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const double d = f2d_exact(L.residual(lut, s, c));  // 0 where not counted
        rsq = fma(d, d, rsq);
        rn += L.factors(lut, s, c).x != 0.0f;
      }
    const int j = L.row(s), i = 2 * (L.pair(s) & (G::LPR - 1));
    if (j < ny && i < nx) a.x_top[i + j * nx] = (j & 1) ? q.x[1] : q.x[0];
    if (j < ny && i + 1 < nx) a.x_top[i + 1 + j * nx] = (j & 1) ? q.x[0] : q.x[1];
  }
}

// The whole tail, run by one block of at least the first frame's warps (and
// 64 threads).
template <int TOP>
struct TailShared {
  float f[Frame<TOP>::OFF + Frame<TOP>::FLOATS];
  float2 lut[64];  // code -> (RN(1 / count), -count)
};

template <int TOP>
__device__ __forceinline__ void mg_coarse_body(const CoarseArgs& a, TailShared<TOP>& sh) {
  const int tid = threadIdx.x;
  // the codes of the thread's pair of every frame it has one in (7: its second of frame 64)
  unsigned code[8];
  auto load = [&](int q, int at, int np, int p) { code[q] = p < np ? __ldg(a.codes + at + p) : 0u; };
  load(0, Frame<1>::CODES, Frame<1>::NP, tid);
  load(1, Frame<2>::CODES, Frame<2>::NP, tid);
  load(2, Frame<4>::CODES, Frame<4>::NP, tid);
  load(3, Frame<8>::CODES, Frame<8>::NP, tid);
  load(4, Frame<16>::CODES, Frame<16>::NP, tid);
  load(5, Frame<32>::CODES, Frame<32>::NP, tid);
  if (TOP == 64) {
    load(6, Frame<64>::CODES, Frame<64>::NP, tid);
    load(7, Frame<64>::CODES, Frame<64>::NP, tid + 1024);
  }
  if (tid < 64) sh.lut[tid] = link_factors(tid);
  __syncthreads();
  dep_wait();
  dep_trigger();
  double rsq = 0.0;
  unsigned long long rn = 0;
  tail_frame<TOP>(a, sh.f, sh.lut, code, tid, rsq, rn);
  if (a.acc != nullptr) {
    __shared__ double red[32];
    __shared__ unsigned long long redn[32];
    const double bsum = block_sum(rsq, red);
    const unsigned long long bn = block_sum_u64(rn, redn);
    if (tid == 0) {
      atomicAdd(&a.acc->res_sq, bsum);
      atomicAdd(&a.acc->n_res, bn);
    }
  }
}

// TOP 32: first levels of at most 32 a side, with twice the registers a thread
template <int TOP>
__global__ void __launch_bounds__(TOP == 64 ? 1024 : 512, 1) k_mg_coarse(CoarseArgs a) {
  __shared__ TailShared<TOP> sh;
  mg_coarse_body<TOP>(a, sh);
}

// The labels and codes of every level of the tail in one launch of one CTA:
// from the first level's labels down, each level's codes, the next level's
// labels, and the level's codes in its frame (the layout of Frame<F>::CODES; a
// pair's low byte is its cell of colour 0; cells beyond the level are outside).
struct TailLabels {
  int nx, ny, nlev, frame;
  uint8_t* label[TAIL_LEVELS];
  uint8_t* code[TAIL_LEVELS];
  uint16_t* out;
};

template <int F>
__device__ __forceinline__ void tail_codes(const TailLabels& a, int l, int nx, int ny) {
  using G = Frame<F>;
  if (F == a.frame >> l) {
    const uint8_t* label = a.label[l];
    for (int p = threadIdx.x; p < G::NP; p += blockDim.x) {
      const int j = p / G::LPR, i = 2 * (p & (G::LPR - 1));
      unsigned c[2] = {CODE_OUTSIDE, CODE_OUTSIDE};
      if (p < G::PAIRS && j < ny) {
#pragma unroll
        for (int o = 0; o < 2; o++)
          if (i + o < nx) {
            c[o] = cell_code(label, nx, ny, i + o, j);
            a.code[l][i + o + j * nx] = (uint8_t)c[o];
          }
        if (l + 1 < a.nlev && i < nx && (j & 1) == 0)
          a.label[l + 1][i / 2 + j / 2 * ((nx + 1) / 2)] = coarse_label(label, nx, ny, i, j);
      }
      a.out[G::CODES + p] = (uint16_t)((j & 1) ? (c[1] | c[0] << 8) : (c[0] | c[1] << 8));
    }
    __syncthreads();
    if (++l == a.nlev) return;
    nx = (nx + 1) / 2;
    ny = (ny + 1) / 2;
  }
  if constexpr (F > 1) tail_codes<F / 2>(a, l, nx, ny);
}

__global__ void __launch_bounds__(1024) k_tail_labels(TailLabels a, const int* only_if) {
  if (only_if != nullptr && *only_if == 0) return;
  tail_codes<64>(a, 0, a.nx, a.ny);
}

// ----------------------------------------------------- the defect-correction pass
//
// p' = p + e (when `update`), r = b - (count*p' - sum) in extended precision
// with the neighbour sum in the order +x, -x, +y, -y, r32 = float(r), and the
// squared norm of r accumulated: the finest level's part of a defect-
// correction cycle (iterative refinement, solveMixed), in float64 or in
// double-float pairs. A warp owns the interior columns of its lanes (the
// first and last lane hold the halo) and its rows (defect_rows); every load of
// its first rows is issued before any arithmetic, all but e's before the launch
// waits for the smoother that writes e (e is not restrict: its loads must not
// move above that wait). Each p' is formed once a warp and handed to its
// neighbours in registers (the rows above and below) and by shuffles (left and
// right).
constexpr int DEFECT_WARPS = 4;
// Columns a block owns.
__host__ __device__ constexpr int defect_cols(bool df) { return df ? 60 : 30; }

// Sums the block's norm in its first thread and adds it to the accumulators:
// a warp's lanes by shuffles, then the first thread over the warps (a second
// tree over 32 lanes for 4 values cost as much as the first).
// n: the warp's count, the same in every lane.
template <class T, class Add, class Wide>
__device__ __forceinline__ void defect_norm(T v, int n, Add add, Wide wide, StepAccum* acc) {
  __shared__ T part[DEFECT_WARPS];
  __shared__ int parts[DEFECT_WARPS];
  for (int o = 16; o > 0; o >>= 1) v = add(v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    part[w] = v;
    parts[w] = n;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = wide(part[0]);
    int m = parts[0];
    for (int k = 1; k < DEFECT_WARPS; k++) {
      s += wide(part[k]);
      m += parts[k];
    }
    atomicAdd(&acc->res_sq, s);
    atomicAdd(&acc->n_res, (unsigned long long)m);
  }
}

// The float64 pass. GB300 issues float64 arithmetic at about 2 lanes per
// clock per SM (32-bit integer adds: ~100), so this pass is bound by its
// float64 instructions, not by memory, and spends them only where the result
// needs them: the exact float -> double widenings, b + b_lo, the first
// addition to 0.0, the products by 2 and 4 and the rounding of r to float run
// on the integer pipe with identical results (fl_common.cuh), with their rare
// cases out of line and their bit casts opaque, so that the compiler neither
// predicates nor re-forms float64 instructions into every cell.
// One block's rows of the pass: block (bx, by) of its grid.
template <bool UPDATE, int RW>
__device__ __forceinline__ void update_resid64_tile(int nx, int ny, double* __restrict__ p64a,
                                                    double* __restrict__ p64b, const SolveCtl* ctl,
                                                    const float* e, const float* __restrict__ b,
                                                    const float* __restrict__ b_lo,
                                                    const uint8_t* __restrict__ code, float* __restrict__ r32,
                                                    StepAccum* acc, int bx, int by) {
  const int par = ctl->par;
  const double* p_in = par ? p64b : p64a;
  double* p_out = par ? p64a : p64b;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gx = bx * 30 - 1 + lane;
  const int y0 = (by * DEFECT_WARPS + w) * RW;
  const bool col = gx >= 0 && gx < nx;
  const bool own = col && lane != 0 && lane != 31;

  // rows y0-1 .. y0+RW of p and e, rows y0 .. y0+RW-1 of the rest; zero /
  // outside where the grid ends. 32-bit offsets: a grid holds fewer than 2^31 cells
  double P[RW + 2];
  float E[RW + 2], B[RW], BL[RW];
  uint8_t C[RW];
#pragma unroll
  for (int r = 0; r < RW + 2; r++) {
    const int y = y0 - 1 + r;
    P[r] = col && (unsigned)y < (unsigned)ny ? p_in[gx + y * nx] : 0.0;
  }
#pragma unroll
  for (int r = 0; r < RW; r++) {
    const int y = y0 + r;
    const bool in = own && y < ny;
    B[r] = in ? b[gx + y * nx] : 0.0f;
    BL[r] = in ? b_lo[gx + y * nx] : 0.0f;
    C[r] = in ? code[gx + y * nx] : (uint8_t)CODE_OUTSIDE;
  }
  dep_wait();
  if (UPDATE) {
#pragma unroll
    for (int r = 0; r < RW + 2; r++) {
      const int y = y0 - 1 + r;
      E[r] = col && (unsigned)y < (unsigned)ny ? e[gx + y * nx] : 0.0f;
    }
#pragma unroll
    for (int r = 0; r < RW + 2; r++) P[r] = P[r] + f2d_exact(E[r]);
  }

  double sq = 0.0;
  int n = 0;
#pragma unroll
  for (int t = 0; t < RW; t++) {
    const int gy = y0 + t;
    const double pc = P[t + 1];
    const double left = __shfl_up_sync(0xffffffffu, pc, 1);
    const double right = __shfl_down_sync(0xffffffffu, pc, 1);
    const uint8_t c = C[t];
    const int cnt = code_count(c);
    const bool on = (c & 3u) == FLUID && cnt > 0;
    n += __popc(__ballot_sync(0xffffffffu, on));
    if (own && gy < ny) {
      const int k = gx + gy * nx;
      if (UPDATE) p_out[k] = pc;
      float r = 0.0f;
      if (on) {
        // the first linked term enters as 0.0 + term
        double sum;
        bool first = true;
        if (c & LINK_XP) {
          sum = zero_plus(right);
          first = false;
        }
        if (c & LINK_XM) {
          sum = first ? zero_plus(left) : sum + left;
          first = false;
        }
        if (c & LINK_YP) {
          sum = first ? zero_plus(P[t + 2]) : sum + P[t + 2];
          first = false;
        }
        if (c & LINK_YM) sum = first ? zero_plus(P[t]) : sum + P[t];
        const double cp = cnt == 4 ? scale_pow2(pc, 2)
                          : cnt == 2 ? scale_pow2(pc, 1)
                          : cnt == 1 ? pc
                                     : dmul_slow(pc, 3.0);
        const double rd = sum_exact(B[t], BL[t]) - (cp - sum);
        r = d2f_rn(rd);
        sq = fma(rd, rd, sq);
      }
      r32[k] = r;
    }
  }
  defect_norm(
      sq, n, [](double a, int o) { return a + __shfl_down_sync(0xffffffffu, a, o); },
      [](double a) { return a; }, acc);
}

// The same pass with the double-float pressure (fl_params.mixed = 2): p' =
// p + e per cell (df_add_f), then r in double-float arithmetic, the neighbour
// sum starting from the first linked neighbour, r32 = the pair rounded to
// float. All of it is float32 arithmetic (~100 operations per cell), which
// bounds it. A lane owns a pair of columns (16-byte loads of p where the rows
// allow it), so half of the horizontal neighbours are its own. A warp walks
// its rows two at a time, the next two loaded before the arithmetic (unrolled
// over 8 rows, the code outgrew the instruction cache: 2.6 of 8.9 stall cycles
// an instruction). The residual norm sums r32^2: each
// square is an exact pair (the product and its FMA error), accumulated as a
// double-float and widened to double once a warp.
template <bool UPDATE>
__device__ __forceinline__ void update_resid_df_tile(int nx, int ny, float2* __restrict__ p2a,
                                                     float2* __restrict__ p2b, const SolveCtl* ctl,
                                                     const float* e, const float* __restrict__ b,
                                                     const float* __restrict__ b_lo,
                                                     const uint8_t* __restrict__ code, float* __restrict__ r32,
                                                     StepAccum* acc, int bx, int by, int rows) {
  const int par = ctl->par;
  const float2* p_in = par ? p2b : p2a;
  float2* p_out = par ? p2a : p2b;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int gx = bx * 60 - 2 + 2 * lane;  // even: the lane's first column
  const int y0 = (by * DEFECT_WARPS + w) * rows, y1 = min(y0 + rows, ny);
  const bool pair = (nx & 1) == 0;  // rows start at multiples of 16 bytes of p: the lane's columns are in or out together
  const bool in0 = (unsigned)gx < (unsigned)nx, in1 = (unsigned)(gx + 1) < (unsigned)nx;
  const bool mine = lane != 0 && lane != 31;
  constexpr unsigned OUTSIDE2 = CODE_OUTSIDE | (unsigned)CODE_OUTSIDE << 8;
  // a neighbour where the link bit is set, else 0, which leaves a sum as it is
  // (pairs are normalised): no lane-divergent branches
  auto linked = [](float2 v, unsigned bit) {
    const int m = -(int)(bit & 1u);
    return make_float2(masked(v.x, m), masked(v.y, m));
  };

  // row y of the lane's pair (0 / outside beyond the grid); 32-bit offsets: a
  // grid holds fewer than 2^31 cells
  auto load2 = [&](const float* f, int y, bool ok) {
    float2 v = make_float2(0.0f, 0.0f);
    const int k = gx + y * nx;
    if (pair) {
      if (ok && in0) v = *reinterpret_cast<const float2*>(f + k);
    } else {
      if (ok && in0) v.x = f[k];
      if (ok && in1) v.y = f[k + 1];
    }
    return v;
  };
  auto load_p = [&](int y, float2* v) {
    const int k = gx + y * nx;
    const bool ok = (unsigned)y < (unsigned)ny;
    v[0] = v[1] = make_float2(0.0f, 0.0f);
    if (pair) {
      if (ok && in0) {
        const float4 q = *reinterpret_cast<const float4*>(p_in + k);
        v[0] = make_float2(q.x, q.y);
        v[1] = make_float2(q.z, q.w);
      }
    } else {
      if (ok && in0) v[0] = p_in[k];
      if (ok && in1) v[1] = p_in[k + 1];
    }
  };
  auto load_code = [&](int y, bool ok) {
    const int k = gx + y * nx;
    unsigned c = OUTSIDE2;
    if (pair) {
      if (ok && in0) c = *reinterpret_cast<const unsigned short*>(code + k);
    } else {
      if (ok && in0) c = (c & 0xff00u) | code[k];
      if (ok && in1) c = (c & 0x00ffu) | (unsigned)code[k + 1] << 8;
    }
    return c;
  };
  auto form = [](float2* v, float2 x) {
    if (UPDATE) {
      v[0] = df_add_f(v[0], x.x);
      v[1] = df_add_f(v[1], x.y);
    }
  };

  float2 P[4][2], N[2][2];  // rows y-1 .. y+2 of p', and the raw rows y+3, y+4
  float2 E[2], B[2], BL[2];
  unsigned C[2];
#pragma unroll
  for (int r = 0; r < 4; r++) load_p(y0 - 1 + r, P[r]);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const bool ok = mine && y0 + r < y1;
    B[r] = load2(b, y0 + r, ok);
    BL[r] = load2(b_lo, y0 + r, ok);
    C[r] = load_code(y0 + r, ok);
  }
  dep_wait();
  if (UPDATE) {
    float2 e0[4];
#pragma unroll
    for (int r = 0; r < 4; r++) e0[r] = load2(e, y0 - 1 + r, (unsigned)(y0 - 1 + r) < (unsigned)ny);
#pragma unroll
    for (int r = 0; r < 4; r++) form(P[r], e0[r]);
  }

  float2 sq = make_float2(0.0f, 0.0f);
  int n = 0;
#pragma unroll 1
  for (int y = y0; y < y1; y += 2) {
    const bool more = y + 2 < y1;  // the same for the whole warp
    float2 B1[2], BL1[2];
    unsigned C1[2];
    if (more) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const bool ok = mine && y + 2 + r < y1;
        load_p(y + 3 + r, N[r]);
        if (UPDATE) E[r] = load2(e, y + 3 + r, y + 3 + r < ny);
        B1[r] = load2(b, y + 2 + r, ok);
        BL1[r] = load2(b_lo, y + 2 + r, ok);
        C1[r] = load_code(y + 2 + r, ok);
      }
    }
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const float2 p0 = P[t + 1][0], p1 = P[t + 1][1];
      const float2 left = make_float2(__shfl_up_sync(0xffffffffu, p1.x, 1), __shfl_up_sync(0xffffffffu, p1.y, 1));
      const float2 right =
          make_float2(__shfl_down_sync(0xffffffffu, p0.x, 1), __shfl_down_sync(0xffffffffu, p0.y, 1));
      float res[2];
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const float2 pc = o ? p1 : p0, xp = o ? right : p1, xm = o ? p0 : left, yp = P[t + 2][o], ym = P[t][o];
        const unsigned c = C[t] >> (8 * o) & 0xffu;
        const int cnt = code_count((uint8_t)c);
        const bool on = (c & 3u) == FLUID && cnt > 0;
        n += __popc(__ballot_sync(0xffffffffu, on));
        const float2 sum = df_add(df_add(df_add(linked(xp, c >> 2), linked(xm, c >> 3)), linked(yp, c >> 4)),
                                  linked(ym, c >> 5));
        const float2 d = df_add(df_mul_count(pc, (float)cnt), df_neg(sum));
        // (b + b_lo) - d: b_lo (the rhs's rounding error) joins the low parts
        const float2 s = df_two_sum(o ? B[t].y : B[t].x, -d.x);
        const float r = __fadd_rn(s.x, __fadd_rn(s.y, __fsub_rn(o ? BL[t].y : BL[t].x, d.y)));
        res[o] = on ? r : 0.0f;
        const float q = __fmul_rn(res[o], res[o]);
        sq = df_add(sq, make_float2(q, __fmaf_rn(res[o], res[o], -q)));
      }
      const int gy = y + t, k = gx + gy * nx;
      if (mine && gy < y1) {
        if (pair) {
          if (in0) {
            if (UPDATE) *reinterpret_cast<float4*>(p_out + k) = make_float4(p0.x, p0.y, p1.x, p1.y);
            *reinterpret_cast<float2*>(r32 + k) = make_float2(res[0], res[1]);
          }
        } else {
          if (in0) {
            if (UPDATE) p_out[k] = p0;
            r32[k] = res[0];
          }
          if (in1) {
            if (UPDATE) p_out[k + 1] = p1;
            r32[k + 1] = res[1];
          }
        }
      }
    }
    if (more) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        form(N[r], E[r]);
        P[r][0] = P[r + 2][0], P[r][1] = P[r + 2][1];
        P[r + 2][0] = N[r][0], P[r + 2][1] = N[r][1];
        B[r] = B1[r];
        BL[r] = BL1[r];
        C[r] = C1[r];
      }
    }
  }
  defect_norm(
      sq, n,
      [](float2 a, int o) {
        return df_add(a, make_float2(__shfl_down_sync(0xffffffffu, a.x, o), __shfl_down_sync(0xffffffffu, a.y, o)));
      },
      [](float2 a) { return df_to_double(a); }, acc);
}

__device__ __forceinline__ double acc_rms(double sq, unsigned long long n) { return n ? sqrt(sq / (double)n) : 0.0; }

// Before the cycle loop (pressureMultigrid.ts:294-300, solveMixed): the rhs
// RMS; a vanishing rhs means p = 0 and no cycle; the float64 path also tests
// its initial residual, so a converged warm start costs no cycle.
__device__ int solve_begin_sums(StepAccum* acc, SolveCtl* ctl, double res_sq, unsigned long long n_res) {
  const double b_rms = acc_rms(acc->b_sq, acc->n_fluid);
  ctl->b_rms = b_rms;
  ctl->cycles = 0;
  ctl->zero_p = b_rms == 0.0;
  ctl->nonfinite = !isfinite(b_rms);
  int cont = 0;
  if (ctl->zero_p) {
    ctl->rel = 0.0;
  } else if (ctl->nonfinite) {
    ctl->rel = -1.0;
  } else if (ctl->mode == SOLVE_MIXED) {
    const double rel = acc_rms(res_sq, n_res) / b_rms;
    ctl->rel = rel;
    cont = ctl->max_cycles > 0 && !(rel <= ctl->tol);
  } else {
    ctl->rel = -1.0;
    cont = ctl->max_cycles > 0;
  }
  ctl->rel0 = ctl->rel;
  acc->res_sq = 0.0;
  acc->n_res = 0ull;
  ctl->cont = cont;
  return cont;
}

__device__ int solve_begin(StepAccum* acc, SolveCtl* ctl) { return solve_begin_sums(acc, ctl, acc->res_sq, acc->n_res); }

__global__ void k_solve_begin(StepAccum* acc, SolveCtl* ctl, int use_cond, cudaGraphConditionalHandle h) {
  const int cont = solve_begin(acc, ctl);
  if (use_cond) cudaGraphSetConditional(h, cont);
}

// After each cycle: count it, evaluate the relative residual the cycle's
// last kernel accumulated, and decide on another (pressureMultigrid.ts:
// 314-317 for float32, solveMixed for float64 defect correction).
__device__ int solve_check_sums(StepAccum* acc, SolveCtl* ctl, double res_sq, unsigned long long n_res) {
  ctl->cycles += 1;
  if (ctl->mode == SOLVE_MIXED) ctl->par = 1 - ctl->par;
  const double rel = acc_rms(res_sq, n_res) / ctl->b_rms;
  ctl->rel = rel;
  int cont = ctl->cycles < ctl->max_cycles;
  if (!isfinite(rel)) {
    ctl->nonfinite = 1;
    cont = 0;
  } else if (ctl->mode == SOLVE_MIXED) {
    cont = cont && !(rel <= ctl->tol);
  } else if (ctl->tol > 0) {
    cont = cont && !(rel <= ctl->tol);
  }
  acc->res_sq = 0.0;
  acc->n_res = 0ull;
  ctl->cont = cont;
  return cont;
}

__device__ int solve_check(StepAccum* acc, SolveCtl* ctl) { return solve_check_sums(acc, ctl, acc->res_sq, acc->n_res); }

// The begin test (test 1) or the cycle test (test 2) run by the last block
// of the defect pass that accumulated the residual, instead of a one-thread
// launch after it. Each block's thread 0 has added its sums (the tile's
// last statement) before it counts itself done; the last block reads the
// totals from L2 once every block has counted, and resets the counter.
__device__ __noinline__ void defect_pass_test_last(StepAccum* acc, SolveCtl* ctl, int test, int use_cond,
                                                   cudaGraphConditionalHandle h) {
  __threadfence();
  acc->test_done = 0u;
  const double sq = __ldcg(&acc->res_sq);
  const unsigned long long n = __ldcg(&acc->n_res);
  const int cont = test == 1 ? solve_begin_sums(acc, ctl, sq, n) : solve_check_sums(acc, ctl, sq, n);
  if (use_cond) cudaGraphSetConditional(h, cont);
}

__device__ __forceinline__ void defect_pass_test(StepAccum* acc, SolveCtl* ctl, int test, int use_cond,
                                                 cudaGraphConditionalHandle h) {
  // only the first thread, which added the block's sums, takes part: the
  // block's other threads are done
  if (test == 0 || threadIdx.x != 0) return;
  __threadfence();
  const unsigned int done = atomicAdd(&acc->test_done, 1u);
  if (done != gridDim.x * gridDim.y - 1) return;
  // out of line: the tests' float64 arithmetic stays out of the pass's
  // register budget (64 registers for 8 blocks per SM)
  defect_pass_test_last(acc, ctl, test, use_cond, h);
}

__global__ void k_solve_check(StepAccum* acc, SolveCtl* ctl, int use_cond, cudaGraphConditionalHandle h) {
  const int cont = solve_check(acc, ctl);
  if (use_cond) cudaGraphSetConditional(h, cont);
}

// After the loop: when the rhs vanished the answer is p = 0 (float32 field
// or the current float64 buffer).
__global__ void k_zero_if(const SolveCtl* __restrict__ ctl, float* __restrict__ p32, double* __restrict__ p64a,
                          double* __restrict__ p64b, long n) {
  dep_trigger();  // an ordinary launch: what precedes it is complete
  if (!ctl->zero_p) return;
  double* p64 = p64a ? (ctl->par ? p64b : p64a) : nullptr;
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
    if (p32) p32[k] = 0.0f;
    if (p64) p64[k] = 0.0;
  }
}

// Remaining divergence of the red-black solver's stopping test (pressure.ts:
// 127-167): neighbour sum in the lexicographic order +x, +y, -x, -y, the
// residual formed in double.
//
// Bound by the float64 pipe. RCP: x / scale as Markstein's two steps from the
// correctly rounded reciprocal (q = x * rcp, then q + (x - q * scale) * rcp,
// which is the correctly rounded quotient when rcp is that of a float: its
// significand is never all ones in double, and quotients of floats keep clear
// of double's range). The other form divides: for a scale that is zero,
// infinite or NaN. Every block ends in atomics on the same two words, so a
// thread takes several rows. 640x480 with cold caches: 16.6 us
// with the division and 1020 blocks, 12.3 with this and 600.
template <bool RCP>
__device__ __forceinline__ double over_scale(double x, double scale, double rcp) {
  if (!RCP) return x / scale;
  const double q = x * rcp;
  const double r = __fma_rn(__fma_rn(-q, scale, x), rcp, q);
  return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : r;  // an infinite x: as the division has it
}

template <bool RCP>
__global__ void __launch_bounds__(256) k_rms_remaining(int nx, int ny, const float* __restrict__ p,
                                                       const float* __restrict__ div,
                                                       const uint8_t* __restrict__ code, double scale, double rcp,
                                                       StepAccum* acc) {
  __shared__ double red[32];
  __shared__ unsigned long long redn[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double sq = 0.0;
  unsigned n = 0;
  if (i < nx) {
#pragma unroll 2
    for (int j = blockIdx.y * blockDim.y + threadIdx.y; j < ny; j += gridDim.y * blockDim.y) {
      const long k = i + (long)j * nx;
      const uint8_t c = code[k];
      const float d = div[k], pc = p[k];
      const float xp = (c & LINK_XP) ? p[k + 1] : 0.0f, yp = (c & LINK_YP) ? p[k + nx] : 0.0f;
      const float xm = (c & LINK_XM) ? p[k - 1] : 0.0f, ym = (c & LINK_YM) ? p[k - nx] : 0.0f;
      const float sum = ((xp + yp) + xm) + ym;
      const int cnt = code_count(c);
      const double r = (double)d + over_scale<RCP>((double)(float)cnt * (double)pc - (double)sum, scale, rcp);
      if ((c & 3u) == FLUID && cnt > 0) {
        sq += r * r;
        n += 1;
      }
    }
  }
  const double bs = block_sum(sq, red);
  const unsigned long long bn = block_sum_u64(n, redn);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    atomicAdd(&acc->res_sq, bs);
    atomicAdd(&acc->n_res, bn);
  }
}

// One plain red-black half-sweep (redBlack.wgsl:67-115), for the per-pass
// entry point.
__global__ void k_rb_halfsweep(int nx, int ny, float* __restrict__ p, const float* __restrict__ b,
                               const uint8_t* __restrict__ code, float scale, float omega, int color) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny || ((i + j) & 1) != color) return;
  const long k = i + (long)j * nx;
  const uint8_t c = code[k];
  if ((c & 3u) != FLUID) return;
  const int cnt = code_count(c);
  if (cnt == 0) return;
  float sum = 0.0f;
  if (c & LINK_XP) sum += p[k + 1];
  if (c & LINK_XM) sum += p[k - 1];
  if (c & LINK_YP) sum += p[k + nx];
  if (c & LINK_YM) sum += p[k - nx];
  const float pgs = (sum - scale * b[k]) / (float)cnt;
  p[k] = (1.0f - omega) * p[k] + omega * pgs;
}

// ------------------------------------------------------------- host side

template <int MODE, int NW, int RW>
static void launch_smooth_nw(cudaStream_t s, const SmoothArgs& a, bool early) {
  const int tx = 64 - 2 * a.halo, ty = RW * NW - 2 * a.halo;
  launch_dependent(early, k_smooth<MODE, NW, RW>, dim3((a.nx + tx - 1) / tx, (a.ny + ty - 1) / ty), dim3(32 * NW), s, a);
}

template <int MODE>
static void launch_smooth_mode(cudaStream_t s, const SmoothArgs& a, bool early, int sms) {
  const int t = 64 - 2 * a.halo;
  if ((long)((a.nx + t - 1) / t) * ((a.ny + t - 1) / t) < smooth_small(sms))
    launch_smooth_nw<MODE, 16, 2>(s, a, early);
  else
    launch_smooth_nw<MODE, 8, 8>(s, a, early);
}

static void launch_smooth(cudaStream_t s, SmoothArgs a, int pairs, int mode, bool early, int sms) {
  a.pairs = pairs;
  a.halo = smooth_halo(mode, pairs, a.x_is_zero, a.acc != nullptr);
  if (mode == MODE_PRE)
    launch_smooth_mode<MODE_PRE>(s, a, early, sms);
  else
    launch_smooth_mode<MODE_POST>(s, a, early, sms);
}

static void launch_level_codes(cudaStream_t s, int nx, int ny, const uint8_t* label, uint8_t* code, uint8_t* coarse,
                               const int* only_if) {
  dim3 b(32, 8), g((nx + 31) / 32, (ny + 7) / 8);
  k_build_codes<<<g, b, 0, s>>>(nx, ny, label, code, coarse, only_if);
}

void launch_build_codes(cudaStream_t s, int nx, int ny, const uint8_t* label, uint8_t* code) {
  launch_level_codes(s, nx, ny, label, code, nullptr, nullptr);
}

void launch_rb_halfsweep(cudaStream_t s, int nx, int ny, float* p, const float* b, const uint8_t* code,
                         float scale, float omega, int color) {
  dim3 bl(32, 8), g((nx + 31) / 32, (ny + 7) / 8);
  k_rb_halfsweep<<<g, bl, 0, s>>>(nx, ny, p, b, code, scale, omega, color);
}

// A row of SOR launches: the pairs a launch and the region shape, by the
// estimated time of the row. One region an SM costs its set-up, load and store
// plus its pairs, two an SM the same and nearly twice the pairs (a launch of
// p pairs with obstacles, measured: 16 warps of 2 rows, 128^2, 64 regions of 6
// pairs 3.2 us, 24 of 4 2.7; 192^2 120 of 6 3.3; 384^2 192 of 4 3.5, 288 of 5
// 4.0; 16 of 4, 320x240 140 of 10 6.3; 384^2 144 of 8 5.9; 517x389 130 of 6 5.3;
// 640x480 140 of 4 4.2 (16 of 2: 5.3), 300 of 8 8.6; 800x600 221 of 4 5.6, 300 of
// 6 7.2). So more pairs pay while their regions, which shrink with the halo, fit
// the SMs; with more than two regions an SM it is 8 warps of 8 rows and 4 pairs
// (1024^2 484 regions 8.7; 2048^2 4 pairs 22.3, 5 28.2, 3 17.1).
// A span is what runs between two residual tests, in launches of equal length.
struct RbShape {
  int nw, rw;
  float us;  // a launch
};
static RbShape rb_shape(int nx, int ny, int pairs, int sms) {
  const int tx = 64 - 4 * pairs;
  auto regions = [&](int ty) { return (long)((nx + tx - 1) / tx) * ((ny + ty - 1) / ty); };
  const long four = regions(tx);
  RbShape best{8, 8, 2.736f / sms * four};
  if (four <= 2L * sms) best = {16, 4, four <= sms ? 2.6f + 0.4f * pairs : 2.8f + 0.73f * pairs};
  if (pairs <= 6) {  // a region of 32 rows
    const long two = regions(32 - 4 * pairs);
    const float us = two <= sms ? 1.6f + 0.28f * pairs : 1.7f + 0.48f * pairs;
    if (two <= 2L * sms && us < best.us) best = {16, 2, us};
  }
  return best;
}

int rb_launch_pairs(int nx, int ny, int span, int sms) {
  int best = std::max(1, std::min(span, 4));  // (no sweeps at all: any)
  float time = FLT_MAX;
  for (int p = best; p <= 10 && p <= span; p++) {
    const int launches = (span + p - 1) / p, q = (span + launches - 1) / launches;
    const RbShape sh = rb_shape(nx, ny, q, sms);
    if (sh.rw == 8 && q > 4) continue;
    if (launches * sh.us < time) {
      time = launches * sh.us;
      best = q;
    }
  }
  return best;
}

void launch_rb_sweeps(cudaStream_t s, int nx, int ny, const float* x_in, float* x_out, const float* b,
                      const uint8_t* code, float scale, float omega, int pairs, const float* scale_dev, bool early,
                      int sms) {
  SmoothArgs a{};
  a.scale_dev = scale_dev;
  a.nx = nx;
  a.ny = ny;
  a.xin = x_in;
  a.xout = x_out;
  a.b = b;
  a.code = code;
  a.scale = scale;
  a.omega = omega;
  a.pairs = pairs;
  a.halo = smooth_halo(MODE_PLAIN, pairs, false, false);
  const RbShape sh = rb_shape(nx, ny, pairs, sms);
  if (sh.rw == 2)
    launch_smooth_nw<MODE_PLAIN, 16, 2>(s, a, early);
  else if (sh.rw == 4)
    launch_smooth_nw<MODE_PLAIN, 16, 4>(s, a, early);
  else
    launch_smooth_nw<MODE_PLAIN, 8, 8>(s, a, early);
}

template <bool UPDATE, int RW>
__global__ void __launch_bounds__(32 * DEFECT_WARPS) k_update_resid64(int nx, int ny, double* __restrict__ p64a,
                                                                     double* __restrict__ p64b, SolveCtl* ctl,
                                                                     const float* e,
                                                                     const float* __restrict__ b,
                                                                     const float* __restrict__ b_lo,
                                                                     const uint8_t* __restrict__ code,
                                                                     float* __restrict__ r32, StepAccum* acc, int test,
                                                                     int use_cond, cudaGraphConditionalHandle h) {
  update_resid64_tile<UPDATE, RW>(nx, ny, p64a, p64b, ctl, e, b, b_lo, code, r32, acc, blockIdx.x, blockIdx.y);
  defect_pass_test(acc, ctl, test, use_cond, h);
}

template <bool UPDATE>
__global__ void __launch_bounds__(32 * DEFECT_WARPS) k_update_resid_df(int nx, int ny, float2* __restrict__ p2a,
                                                                      float2* __restrict__ p2b, SolveCtl* ctl,
                                                                      const float* e, const float* __restrict__ b,
                                                                      const float* __restrict__ b_lo,
                                                                      const uint8_t* __restrict__ code,
                                                                      float* __restrict__ r32, StepAccum* acc, int rows,
                                                                      int test, int use_cond,
                                                                      cudaGraphConditionalHandle h) {
  update_resid_df_tile<UPDATE>(nx, ny, p2a, p2b, ctl, e, b, b_lo, code, r32, acc, blockIdx.x, blockIdx.y, rows);
  defect_pass_test(acc, ctl, test, use_cond, h);
}

// The blocks of a pass over nx x ny cells with `rows` rows a warp.
static long defect_blocks(int nx, int ny, bool df, int rows) {
  const int c = defect_cols(df), r = DEFECT_WARPS * rows;
  return (long)((nx + c - 1) / c) * ((ny + r - 1) / r);
}

// Rows a warp. A small grid's pass is the latency of one warp: as few rows as
// there are SMs for; a large one's is throughput: more rows, so that fewer of
// them are formed twice. blocks(rows): the pass's blocks.
// float64 (2, 4 or 8): 256^2 2 rows 7.7 us, 4 rows 7.6, 8 rows 10.0; 512^2
// 14.0 / 12.5 / 12.0; 1024^2 30.2 / 26.2 / 29.4; 2048^2 105 / 89 / 86.
// Double-float (2, 4, 6 or 8): the fewest whose blocks are resident at once (6
// an SM): 256^2 2 rows 6.2 us, 4 rows 7.1, 8 rows 9.3; 724^2 12.6 / 10.6 /
// 11.3; 2048^2 57 / 42 / 36.
// (Each after the POST launch it follows, that launch's time taken off, with
// the cycle test. The form before, 8 rows on every grid: float64 17.9 us at
// 256^2, 94 at 2048^2; double-float 9.2 and 49.)
template <class Blocks>
static int defect_rows(bool df, int sms, Blocks blocks) {
  if (!df) return blocks(2) <= 2L * sms ? 2 : blocks(4) <= 26L * sms ? 4 : 8;
  for (int r = 2; r < 8; r += 2)
    if (blocks(r) <= 6L * sms) return r;
  return 8;
}

void launch_update_resid64(cudaStream_t s, int nx, int ny, double* p64a, double* p64b, SolveCtl* ctl,
                           const float* e, const float* b, const float* b_lo, const uint8_t* code, bool update,
                           float* r32, StepAccum* acc, bool df, int sms, int test, bool use_cond,
                           cudaGraphConditionalHandle h) {
  const int uc = use_cond ? 1 : 0;
  const int rows = defect_rows(df, sms, [&](int r) { return defect_blocks(nx, ny, df, r); });
  const int c = defect_cols(df), r = DEFECT_WARPS * rows;
  const dim3 g((nx + c - 1) / c, (ny + r - 1) / r), t(32 * DEFECT_WARPS);
  // the pass that updates follows the smoother that writes e
  if (df) {
    float2* a = reinterpret_cast<float2*>(p64a);
    float2* bb = reinterpret_cast<float2*>(p64b);
    launch_dependent(update, update ? k_update_resid_df<true> : k_update_resid_df<false>, g, t, s, nx, ny, a, bb, ctl, e,
                     b, b_lo, code, r32, acc, rows, test, uc, h);
    return;
  }
  auto k = update ? (rows == 2 ? k_update_resid64<true, 2> : rows == 4 ? k_update_resid64<true, 4> : k_update_resid64<true, 8>)
                  : (rows == 2 ? k_update_resid64<false, 2> : rows == 4 ? k_update_resid64<false, 4> : k_update_resid64<false, 8>);
  launch_dependent(update, k, g, t, s, nx, ny, p64a, p64b, ctl, e, b, b_lo, code, r32, acc, test, uc, h);
}

void launch_solve_begin(cudaStream_t s, StepAccum* acc, SolveCtl* ctl, bool use_cond, cudaGraphConditionalHandle h) {
  k_solve_begin<<<1, 1, 0, s>>>(acc, ctl, use_cond, h);
}

void launch_solve_check(cudaStream_t s, StepAccum* acc, SolveCtl* ctl, bool use_cond, cudaGraphConditionalHandle h) {
  k_solve_check<<<1, 1, 0, s>>>(acc, ctl, use_cond, h);
}

void launch_zero_if(cudaStream_t s, const SolveCtl* ctl, float* p32, double* p64a, double* p64b, long n) {
  long blocks = std::min((n + 255) / 256, 152L * 4);
  k_zero_if<<<(unsigned)std::max(1L, blocks), 256, 0, s>>>(ctl, p32, p64a, p64b, n);
}

void launch_rms_remaining(cudaStream_t s, int nx, int ny, const float* p, const float* div, const uint8_t* code,
                          float scale, StepAccum* acc) {
  dim3 b(32, 8), g((nx + 31) / 32, (ny + 7) / 8);
  g.y = std::min(g.y, std::max(1u, 608u / g.x));
  const double sd = (double)scale;
  if (std::isfinite(scale) && scale != 0.0f)
    k_rms_remaining<true><<<g, b, 0, s>>>(nx, ny, p, div, code, sd, 1.0 / sd, acc);
  else
    k_rms_remaining<false><<<g, b, 0, s>>>(nx, ny, p, div, code, sd, 0.0, acc);
}

// The side of the frame that holds an nx x ny level of the tail.
static int tail_frame_side(int nx, int ny) {
  int f = 1;
  while (f < nx || f < ny) f *= 2;
  return f;
}

void mg_free(Engine& e) {
  for (auto& L : e.levels) {
    cudaFree(L.x[0]);
    cudaFree(L.x[1]);
    cudaFree(L.b);
    if (&L != &e.levels[0]) cudaFree(L.label);
    cudaFree(L.code);
  }
  cudaFree(e.tail_codes);
  e.tail_codes = nullptr;
  e.levels.clear();
}

void mg_setup(Engine& e) {
  mg_free(e);
  // pressureMultigrid.ts:71-78
  std::vector<std::pair<int, int>> sizes{{e.nx, e.ny}};
  const int coarsest = std::max(1, e.prm.mg_coarsest);
  while (sizes.back().first > coarsest || sizes.back().second > coarsest)
    sizes.push_back({(sizes.back().first + 1) / 2, (sizes.back().second + 1) / 2});
  for (auto& sz : sizes) {
    Level L;
    L.nx = sz.first;
    L.ny = sz.second;
    e.levels.push_back(L);
  }
  for (size_t l = 0; l < e.levels.size(); l++) {
    Level& L = e.levels[l];
    const size_t n = (size_t)L.nx * L.ny;
    cudaMalloc(&L.x[0], n * sizeof(float));
    cudaMalloc(&L.x[1], n * sizeof(float));
    cudaMalloc(&L.b, n * sizeof(float));
    if (l > 0) cudaMalloc(&L.label, n);
    cudaMalloc(&L.code, n);
    cudaMemsetAsync(L.x[0], 0, n * sizeof(float), e.stream);
    cudaMemsetAsync(L.x[1], 0, n * sizeof(float), e.stream);
    cudaMemsetAsync(L.b, 0, n * sizeof(float), e.stream);
  }
  // the tail starts at the first level with both sides <= mg_tail_side (the
  // coarsest level at the latest)
  const int side = e.prm.mg_tail_side > 0 ? e.prm.mg_tail_side : TAIL_SIDE_DEFAULT;
  int lc = (int)e.levels.size() - 1;
  for (int l = 0; l < (int)e.levels.size(); l++)
    if (e.levels[l].nx <= side && e.levels[l].ny <= side) {
      lc = l;
      break;
    }
  e.coarse_level = lc;
  cudaMalloc(&e.tail_codes, TAIL_CODES * sizeof(uint16_t));
  e.codes_valid = false;
}

// Every level's labels and codes on stream s: one launch a level above the
// tail, one for the tail's levels together.
static void enqueue_build_codes(const Engine& e, cudaStream_t s, const int* only_if) {
  const int lc = e.coarse_level, n = (int)e.levels.size();
  for (int l = 0; l < lc; l++) {
    const Level& L = e.levels[l];
    launch_level_codes(s, L.nx, L.ny, L.label, L.code, e.levels[l + 1].label, only_if);
  }
  TailLabels a{};
  a.nx = e.levels[lc].nx;
  a.ny = e.levels[lc].ny;
  a.nlev = n - lc;
  a.frame = tail_frame_side(a.nx, a.ny);
  for (int l = lc; l < n; l++) {
    a.label[l - lc] = e.levels[l].label;
    a.code[l - lc] = e.levels[l].code;
  }
  a.out = e.tail_codes;
  k_tail_labels<<<1, 1024, 0, s>>>(a, only_if);
}

void mg_build_codes(Engine& e) {
  enqueue_build_codes(e, e.stream, nullptr);
  e.codes_valid = true;
}

__global__ void k_clear_flag(int* flag) { *flag = 0; }

// The same rebuild on stream s as kernels that each return at once unless
// *flag is set (the label compare's result), then the flag cleared: a
// plain graph's worth of launches where an IF node would otherwise decide.
void mg_build_codes_if(Engine& e, cudaStream_t s, int* flag) {
  enqueue_build_codes(e, s, flag);
  k_clear_flag<<<1, 1, 0, s>>>(flag);
}

// One V-cycle (pressureMultigrid.ts:253-275) on levels[0].b with the warm
// start in levels[0].x[0]; the result lands back in levels[0].x[0]. When
// `acc` is set, the finest level's residual sum of squares is accumulated
// into it for the tolerance test.
void mg_vcycle(Engine& e, StepAccum* acc) { mg_vcycle_on(e, e.levels[0].b, false, acc); }

// The threads of a frame's warps, at least 64.
static int tail_threads(int frame) { return std::min(1024, std::max(64, frame * frame / 2)); }

// The single-CTA tail's arguments for a V-cycle on b0 (the finest level's
// rhs when the tail starts there), from zero when zero_start, accumulating
// the finest residual into acc when the tail holds the finest level.
static CoarseArgs coarse_args(const Engine& e, const float* b0, bool zero_start, StepAccum* acc) {
  const int lc = e.coarse_level;
  CoarseArgs a{};
  a.nlev = (int)e.levels.size() - lc;
  a.nx = e.levels[lc].nx;
  a.ny = e.levels[lc].ny;
  a.frame = tail_frame_side(a.nx, a.ny);
  a.codes = e.tail_codes;
  a.b_top = lc == 0 ? b0 : e.levels[lc].b;
  a.x_top = e.levels[lc].x[0];
  a.x_is_zero = lc > 0 || zero_start;
  a.pre = e.prm.mg_pre;
  a.post = e.prm.mg_post;
  a.coarse_sweeps = e.prm.mg_coarse_sweeps;
  a.omega = (float)e.prm.mg_omega;
  a.acc = lc == 0 ? acc : nullptr;
  return a;
}

// One V-cycle with level 0's rhs `b0`; with `zero_start` the level-0 unknown
// starts from 0 (the correction equation of the defect-correction loop)
// instead of the warm start in levels[0].x[0].
void mg_vcycle_on(Engine& e, const float* b0, bool zero_start, StepAccum* acc) {
  cudaStream_t s = e.stream;
  const int lc = e.coarse_level;
  const float omega = (float)e.prm.mg_omega;
  auto cells = [&](int l) { return (double)e.levels[l].nx * e.levels[l].ny; };
  for (int l = 0; l < lc; l++) {
    Level& L = e.levels[l];
    Level& C = e.levels[l + 1];
    // x (level 0 only: coarser levels start from zero), b, code, x out, coarse b
    const int tok = prof_begin(e, l == 0 ? FL_PH_MG_PRE_FINE : FL_PH_MG_PRE);
    SmoothArgs a{};
    a.nx = L.nx;
    a.ny = L.ny;
    a.xin = L.x[0];
    a.xout = L.x[1];
    a.b = l == 0 ? b0 : L.b;
    a.code = L.code;
    a.scale = -1.0f;
    a.omega = omega;
    a.bc = C.b;
    a.cnx = C.nx;
    a.cny = C.ny;
    a.x_is_zero = l > 0 || zero_start;
    launch_smooth(s, a, e.prm.mg_pre, MODE_PRE, l > 0, e.sms);
    prof_end(e, tok, (l == 0 ? 13.0 : 9.0) * cells(l) + 4.0 * cells(l + 1), 1);
  }
  {
    const int tok = prof_begin(e, FL_PH_MG_COARSE);
    double bytes = (lc == 0 ? 4.0 : 0.0) * cells(lc) + 8.0 * cells(lc);
    for (int l = lc; l < (int)e.levels.size(); l++) bytes += cells(l);
    const CoarseArgs a = coarse_args(e, b0, zero_start, acc);
    // (lc == 0: the V-cycle's first launch)
    launch_dependent(lc > 0, a.frame == 64 ? k_mg_coarse<64> : k_mg_coarse<32>, dim3(1), dim3(tail_threads(a.frame)), s,
                     a);
    prof_end(e, tok, bytes, 1);
  }
  for (int l = lc - 1; l >= 0; l--) {
    Level& L = e.levels[l];
    Level& C = e.levels[l + 1];
    // x in, b, code, coarse e, x out
    const int tok = prof_begin(e, l == 0 ? FL_PH_MG_POST_FINE : FL_PH_MG_POST);
    SmoothArgs a{};
    a.nx = L.nx;
    a.ny = L.ny;
    a.xin = L.x[1];
    a.xout = L.x[0];
    a.b = l == 0 ? b0 : L.b;
    a.code = L.code;
    a.scale = -1.0f;
    a.omega = omega;
    a.ec = C.x[0];
    a.cnx = C.nx;
    a.cny = C.ny;
    a.acc = l == 0 ? acc : nullptr;
    launch_smooth(s, a, e.prm.mg_post, MODE_POST, true, e.sms);
    prof_end(e, tok, 13.0 * cells(l) + 4.0 * cells(l + 1), 1);
  }
}


// ------------------------------------------------------------ batched solve
//
// The pressure solves of many engines advanced together (fl_batch): each
// V-cycle phase is ONE launch over a list of (scene, level, tile) items
// drawn from every scene of the batch, the scenes' tails aligned (a scene
// with fewer levels above its tail joins the descent later and leaves the
// ascent earlier), and the cycle loop is one device-side WHILE over "some
// scene still iterates". A scene that has converged (its control block's
// `cont` cleared by its own test) leaves its items at once, so every scene
// runs exactly the cycles it would run alone, through the same per-tile code
// (smooth_tile, mg_coarse_body, the defect-pass tiles, solve_begin /
// solve_check): its results are bit-identical to stepping it alone.

struct BatchLevel {
  int nx, ny;
  float* x0;
  float* x1;
  float* b;
  const uint8_t* code;
};

struct BatchScene {
  BatchLevel lv[MAX_LEVELS];
  CoarseArgs tail;
  double* p64a;
  double* p64b;
  float* r32;
  float* b_lo;
  SolveCtl* ctl;
  StepAccum* acc;
  long cells;
  int nlev, lc, mixed;
  float omega;
};

struct BatchItem {
  int scene, level, bx, by;
};

// The plan's device-side lists. Cycle phases ph: PRE at depth d (0..D-1),
// the tail (D), POST at depth d (D+1..2D), the defect pass (2D+1); items of
// scene k in phase ph are items[base[ph][k] .. + count[ph][k]). The begin and
// check kernels compact, per phase, the scenes still iterating: act_scene
// (in the plan's order, largest scenes first), act_pre (exclusive prefix of
// their item counts), act_n and act_total; a phase kernel's blocks walk
// 0 .. act_total by the grid's stride.
struct BatchPlan {
  const BatchScene* sc;
  const BatchItem* items;
  const int* base;
  const int* count;
  int* act_scene;
  int* act_pre;
  int* act_n;
  int* act_total;
  int n, nph;
};

struct BatchSolve {
  int device = 0;
  int n = 0, depth = 0, sms = 0;
  int pre = 0, post = 0;
  bool any_mixed = false;
  int tail_threads = 64;
  BatchScene* scenes = nullptr;  // device, largest scene first
  BatchItem* items = nullptr;    // device
  int* lists = nullptr;          // device: base, count, act_scene, act_pre, act_n, act_total
  BatchPlan plan{};
  std::vector<int> max_items;    // per cycle phase: all scenes' items (the grid's bound)
  int defect_rows[2] = {8, 8};   // the defect pass's rows a warp: float64 scenes, double-float scenes
  std::vector<char> small;       // per cycle phase: its smoother items are the 64 x 32 regions
  std::pair<int, int> init_ph{0, 0}, zero_ph{0, 0};  // prologue defect pass, p = 0 fill: every scene
};

// Before a kernel's dep_wait: the lists are k_batch_check's, of the cycle
// before. A block without items waits all the same (its kernel's end stands for
// the end of all before it).
__device__ __forceinline__ bool batch_item(const BatchPlan& P, int ph, int i, BatchItem& it) {
  if (i >= P.act_total[ph]) {
    dep_wait();
    return false;
  }
  const int* pre = P.act_pre + (long)ph * (P.n + 1);
  int lo = 0, hi = P.act_n[ph] - 1;  // the last active scene whose prefix is <= i
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= i)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int k = P.act_scene[(long)ph * P.n + lo];
  it = P.items[P.base[(long)ph * P.n + k] + (i - pre[lo])];
  return true;
}

// Per phase, the items of the scenes whose control block says they iterate
// (one warp per phase, a warp-wide scan per 32 scenes). Called by a whole
// block after the scenes' tests, behind a barrier.
__device__ void batch_compact(const BatchPlan& P) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int ph = w; ph < P.nph; ph += nw) {
    int run = 0, nact = 0;
    for (int c = 0; c < P.n; c += 32) {
      const int k = c + lane;
      const int cnt = k < P.n && P.sc[k].ctl->cont ? P.count[(long)ph * P.n + k] : 0;
      int x = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      const unsigned on = __ballot_sync(0xffffffffu, cnt > 0);
      if (cnt > 0) {
        const int pos = nact + __popc(on & ((1u << lane) - 1u));
        P.act_scene[(long)ph * P.n + pos] = k;
        P.act_pre[(long)ph * (P.n + 1) + pos] = run + x - cnt;
      }
      run += __shfl_sync(0xffffffffu, x, 31);
      nact += __popc(on);
    }
    if (lane == 0) {
      P.act_total[ph] = run;
      P.act_n[ph] = nact;
      P.act_pre[(long)ph * (P.n + 1) + nact] = run;
    }
  }
}

template <int MODE, int NW, int RW>
__global__ void __launch_bounds__(32 * NW, RW == 8 ? 24 / NW : 32 / NW) k_batch_smooth(BatchPlan plan, int ph, int pairs) {
  __shared__ SmoothShared<NW, RW> sh;
  for (int i = blockIdx.x;; i += gridDim.x) {
    BatchItem it;
    if (!batch_item(plan, ph, i, it)) return;  // the same for the whole block
    const BatchScene& S = plan.sc[it.scene];
    const int l = it.level;
    const BatchLevel& L = S.lv[l];
    const BatchLevel& C = S.lv[l + 1];
    // the arguments mg_vcycle_on gives this level (mixed: a V-cycle on the
    // defect pass's residual from zero; otherwise on b from the warm start)
    SmoothArgs a{};
    a.nx = L.nx;
    a.ny = L.ny;
    a.code = L.code;
    a.scale = -1.0f;
    a.omega = S.omega;
    a.cnx = C.nx;
    a.cny = C.ny;
    a.b = l == 0 && S.mixed ? S.r32 : L.b;
    if (MODE == MODE_PRE) {
      a.xin = L.x0;
      a.xout = L.x1;
      a.bc = C.b;
      a.x_is_zero = l > 0 || S.mixed;
    } else {
      a.xin = L.x1;
      a.xout = L.x0;
      a.ec = C.x0;
      a.acc = l == 0 && !S.mixed ? S.acc : nullptr;
    }
    a.pairs = pairs;
    a.halo = smooth_halo(MODE, pairs, a.x_is_zero, a.acc != nullptr);
    smooth_tile<MODE, NW, RW>(a, it.bx, it.by, sh);
    __syncthreads();  // the next region reuses the shared tiles
  }
}

template <int TOP>
__global__ void __launch_bounds__(TOP == 64 ? 1024 : 512, 1) k_batch_tail(BatchPlan plan, int ph) {
  __shared__ TailShared<TOP> sh;
  for (int i = blockIdx.x;; i += gridDim.x) {
    BatchItem it;
    if (!batch_item(plan, ph, i, it)) return;
    mg_coarse_body<TOP>(plan.sc[it.scene].tail, sh);
    __syncthreads();
  }
}

// RW: the float64 scenes' rows a warp, rows_df: the double-float scenes'.
template <bool UPDATE, int RW>
__device__ __forceinline__ void batch_defect_item(const BatchScene& S, const BatchItem& it, int rows_df) {
  const BatchLevel& L0 = S.lv[0];
  const float* e = UPDATE ? L0.x0 : nullptr;
  if (S.mixed == MIXED_DF)
    update_resid_df_tile<UPDATE>(L0.nx, L0.ny, reinterpret_cast<float2*>(S.p64a), reinterpret_cast<float2*>(S.p64b),
                                 S.ctl, e, L0.b, S.b_lo, L0.code, S.r32, S.acc, it.bx, it.by, rows_df);
  else
    update_resid64_tile<UPDATE, RW>(L0.nx, L0.ny, S.p64a, S.p64b, S.ctl, e, L0.b, S.b_lo, L0.code, S.r32, S.acc, it.bx,
                                it.by);
}

// The defect pass of the iterating scenes with a refined pressure: p += e
// and the new residual.
template <int RW>
__global__ void __launch_bounds__(32 * DEFECT_WARPS) k_batch_defect(BatchPlan plan, int ph, int rows_df) {
  for (int i = blockIdx.x;; i += gridDim.x) {
    BatchItem it;
    if (!batch_item(plan, ph, i, it)) return;
    batch_defect_item<true, RW>(plan.sc[it.scene], it, rows_df);
    __syncthreads();
  }
}

// The initial defect pass of every scene with a refined pressure (before
// the loop), one item per block.
template <int RW>
__global__ void __launch_bounds__(32 * DEFECT_WARPS) k_batch_defect_init(const BatchScene* __restrict__ sc,
                                                                         const BatchItem* __restrict__ items,
                                                                         int rows_df) {
  const BatchItem it = items[blockIdx.x];
  batch_defect_item<false, RW>(sc[it.scene], it, rows_df);
}

// Every scene's begin test, the compacted lists of the first cycle; the
// WHILE node runs while any scene iterates.
__global__ void __launch_bounds__(1024) k_batch_begin(BatchPlan plan, cudaGraphConditionalHandle h) {
  int any = 0;
  for (int k = threadIdx.x; k < plan.n; k += blockDim.x) any |= solve_begin(plan.sc[k].acc, plan.sc[k].ctl);
  any = __syncthreads_or(any);
  batch_compact(plan);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// Every iterating scene's cycle test (the others keep their state), the
// compacted lists of the next cycle.
__global__ void __launch_bounds__(1024) k_batch_check(BatchPlan plan, cudaGraphConditionalHandle h) {
  dep_wait();
  int any = 0;
  for (int k = threadIdx.x; k < plan.n; k += blockDim.x)
    if (plan.sc[k].ctl->cont) any |= solve_check(plan.sc[k].acc, plan.sc[k].ctl);
  any = __syncthreads_or(any);
  batch_compact(plan);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// k_zero_if per scene: item (scene, -, block, blocks of the scene).
__global__ void __launch_bounds__(256) k_batch_zero(const BatchScene* __restrict__ sc,
                                                    const BatchItem* __restrict__ items) {
  const BatchItem it = items[blockIdx.x];
  const BatchScene& S = sc[it.scene];
  if (!S.ctl->zero_p) return;
  float* p32 = S.mixed ? nullptr : S.lv[0].x0;
  double* p64 = S.mixed ? (S.ctl->par ? S.p64b : S.p64a) : nullptr;
  for (long k = it.bx * 256L + threadIdx.x; k < S.cells; k += (long)it.by * 256) {
    if (p32) p32[k] = 0.0f;
    if (p64) p64[k] = 0.0;
  }
}

BatchSolve* batch_solve_create(const std::vector<Engine*>& es_in, std::string& why) {
  if (es_in.empty()) {
    why = "no scenes";
    return nullptr;
  }
  const fl_params& p0 = es_in[0]->prm;
  for (const Engine* e : es_in) {
    if (e->prm.solver != FL_SOLVER_MG) why = "a scene solves with red-black SOR";
    else if (e->prm.mg_pre != p0.mg_pre || e->prm.mg_post != p0.mg_post)
      why = "the scenes' V-cycle shapes differ";
    else if (e->prm.mg_pre < 0 || e->prm.mg_pre > 4 || e->prm.mg_post < 0 || e->prm.mg_post > 4)
      why = "sweep pairs beyond 4";
    else if ((int)e->levels.size() > MAX_LEVELS || e->levels.empty())
      why = "too many levels";
    if (!why.empty()) return nullptr;
  }
  // the plan's scenes, largest first (blocks walk the items in this order)
  std::vector<const Engine*> es(es_in.begin(), es_in.end());
  std::stable_sort(es.begin(), es.end(), [](const Engine* x, const Engine* y) { return x->cells() > y->cells(); });
  BatchSolve* b = new BatchSolve();
  b->device = es[0]->device;
  b->n = (int)es.size();
  b->pre = p0.mg_pre;
  b->post = p0.mg_post;
  cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device);
  if (b->sms < 1) b->sms = 1;
  std::vector<BatchScene> hs(es.size());
  for (size_t k = 0; k < es.size(); k++) {
    const Engine& e = *es[k];
    BatchScene& S = hs[k];
    std::memset(&S, 0, sizeof S);
    S.nlev = (int)e.levels.size();
    S.lc = e.coarse_level;
    S.mixed = e.prm.mixed;
    S.omega = (float)e.prm.mg_omega;
    S.cells = e.cells();
    for (int l = 0; l < S.nlev; l++) {
      const Level& L = e.levels[l];
      S.lv[l] = BatchLevel{L.nx, L.ny, L.x[0], L.x[1], L.b, L.code};
    }
    const bool mixed = e.prm.mixed != 0;
    S.tail = coarse_args(e, mixed ? e.r32 : e.levels[0].b, mixed, mixed ? nullptr : e.acc);
    S.p64a = e.p64[0];
    S.p64b = e.p64[1];
    S.r32 = e.r32;
    S.b_lo = e.b_lo;
    S.ctl = e.ctl;
    S.acc = e.acc;
    b->any_mixed = b->any_mixed || mixed;
    b->tail_threads = std::max(b->tail_threads, tail_threads(S.tail.frame));
    b->depth = std::max(b->depth, S.lc);
  }
  const int n = b->n, depth = b->depth, nph = 2 * depth + 2;
  std::vector<BatchItem> items;
  std::vector<int> base((size_t)nph * n, 0), count((size_t)nph * n, 0);
  b->max_items.assign(nph, 0);
  // scene k's items of phase ph, appended
  auto add = [&](int ph, int k, auto&& emit) {
    base[(size_t)ph * n + k] = (int)items.size();
    emit();
    count[(size_t)ph * n + k] = (int)items.size() - base[(size_t)ph * n + k];
    b->max_items[ph] += count[(size_t)ph * n + k];
  };
  // the level scene k smooths in phase ph (-1: none) and its region's halo;
  // PRE: level lc_k - depth + d at phase d (the tails aligned); POST: level
  // lc_k - 1 - d at phase depth + 1 + d
  auto smooth_level = [&](int ph, int k, int* halo) {
    const bool pre = ph < depth;
    const int l = pre ? hs[k].lc - depth + ph : hs[k].lc - 1 - (ph - depth - 1);
    *halo = pre ? smooth_halo(MODE_PRE, b->pre, l > 0 || hs[k].mixed, false)
                : smooth_halo(MODE_POST, b->post, false, l == 0 && !hs[k].mixed);
    return l;
  };
  auto regions = [&](int k, int l, int halo, int rows, int* gx, int* gy) {
    const int tx = 64 - 2 * halo, ty = rows - 2 * halo;
    *gx = (hs[k].lv[l].nx + tx - 1) / tx;
    *gy = (hs[k].lv[l].ny + ty - 1) / ty;
  };
  // a phase's regions as launch_smooth chooses them, for all its scenes together
  b->small.assign(nph, 0);
  for (int ph = 0; ph < 2 * depth + 1; ph++) {
    if (ph == depth) continue;
    long total = 0;
    for (int k = 0; k < n; k++) {
      int halo, gx, gy;
      const int l = smooth_level(ph, k, &halo);
      if (l < 0) continue;
      regions(k, l, halo, 64, &gx, &gy);
      total += (long)gx * gy;
    }
    b->small[ph] = total < smooth_small(b->sms);
  }
  auto smooth_items = [&](int ph, int k) {
    int halo, gx, gy;
    const int l = smooth_level(ph, k, &halo);
    if (l < 0) return;
    regions(k, l, halo, b->small[ph] ? 32 : 64, &gx, &gy);
    for (int by = 0; by < gy; by++)
      for (int bx = 0; bx < gx; bx++) items.push_back(BatchItem{k, l, bx, by});
  };
  // the defect pass's rows a warp, for all scenes of a kind together
  auto defect_total = [&](bool df, int rows) {
    long total = 0;
    for (const BatchScene& S : hs)
      if (S.mixed != 0 && (S.mixed == MIXED_DF) == df) total += defect_blocks(S.lv[0].nx, S.lv[0].ny, df, rows);
    return total;
  };
  for (int df = 0; df < 2; df++)
    b->defect_rows[df] = defect_rows(df, b->sms, [&](int r) { return defect_total(df, r); });
  auto defect_items = [&](int k) {
    const BatchLevel& L = hs[k].lv[0];
    const bool df = hs[k].mixed == MIXED_DF;
    const int cols = defect_cols(df), rows = DEFECT_WARPS * b->defect_rows[df];
    for (int by = 0; by < (L.ny + rows - 1) / rows; by++)
      for (int bx = 0; bx < (L.nx + cols - 1) / cols; bx++) items.push_back(BatchItem{k, 0, bx, by});
  };
  for (int k = 0; k < n; k++) {
    for (int ph = 0; ph < depth; ph++) add(ph, k, [&] { smooth_items(ph, k); });
    add(depth, k, [&] { items.push_back(BatchItem{k, hs[k].lc, 0, 0}); });
    for (int ph = depth + 1; ph < 2 * depth + 1; ph++) add(ph, k, [&] { smooth_items(ph, k); });
    if (hs[k].mixed) add(2 * depth + 1, k, [&] { defect_items(k); });
  }
  b->init_ph.first = (int)items.size();
  for (int k = 0; k < n; k++)
    if (hs[k].mixed) defect_items(k);
  b->init_ph.second = (int)items.size() - b->init_ph.first;
  b->zero_ph.first = (int)items.size();
  for (int k = 0; k < n; k++) {
    const int blocks = (int)std::min<long>(64, std::max<long>(1, (hs[k].cells + 255) / 256));
    for (int q = 0; q < blocks; q++) items.push_back(BatchItem{k, 0, q, blocks});
  }
  b->zero_ph.second = (int)items.size() - b->zero_ph.first;
  // lists: base, count [nph*n]; act_scene [nph*n]; act_pre [nph*(n+1)]; act_n, act_total [nph]
  const size_t nl = 3 * (size_t)nph * n + (size_t)nph * (n + 1) + 2 * (size_t)nph;
  cudaError_t err = cudaMalloc(&b->scenes, hs.size() * sizeof(BatchScene));
  if (err == cudaSuccess) err = cudaMalloc(&b->items, items.size() * sizeof(BatchItem));
  if (err == cudaSuccess) err = cudaMalloc(&b->lists, nl * sizeof(int));
  if (err == cudaSuccess) err = cudaMemset(b->lists, 0, nl * sizeof(int));
  if (err == cudaSuccess)
    err = cudaMemcpy(b->scenes, hs.data(), hs.size() * sizeof(BatchScene), cudaMemcpyHostToDevice);
  if (err == cudaSuccess)
    err = cudaMemcpy(b->items, items.data(), items.size() * sizeof(BatchItem), cudaMemcpyHostToDevice);
  if (err == cudaSuccess)
    err = cudaMemcpy(b->lists, base.data(), base.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (err == cudaSuccess)
    err = cudaMemcpy(b->lists + base.size(), count.data(), count.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (err != cudaSuccess) {
    why = cudaGetErrorString(err);
    batch_solve_destroy(b);
    return nullptr;
  }
  BatchPlan& P = b->plan;
  P.sc = b->scenes;
  P.items = b->items;
  P.base = b->lists;
  P.count = b->lists + (size_t)nph * n;
  P.act_scene = b->lists + 2 * (size_t)nph * n;
  P.act_pre = b->lists + 3 * (size_t)nph * n;
  P.act_n = P.act_pre + (size_t)nph * (n + 1);
  P.act_total = P.act_n + nph;
  P.n = n;
  P.nph = nph;
  return b;
}

void batch_solve_destroy(BatchSolve* b) {
  if (!b) return;
  cudaFree(b->scenes);
  cudaFree(b->items);
  cudaFree(b->lists);
  delete b;
}

// A cycle phase: a grid of at most `per_sm` blocks per SM (bounded by the
// phase's items over all scenes) walking the iterating scenes' items.
static unsigned phase_grid(const BatchSolve& b, int ph, int per_sm) {
  return (unsigned)std::max(1, std::min(b.max_items[ph], b.sms * per_sm));
}

template <int MODE>
static void launch_batch_smooth(cudaStream_t s, const BatchSolve& b, int pairs, int ph, bool& early) {
  if (b.max_items[ph] == 0) return;
  if (b.small[ph])
    launch_dependent(early, k_batch_smooth<MODE, 16, 2>, phase_grid(b, ph, 2), 512, s, b.plan, ph, pairs);
  else
    launch_dependent(early, k_batch_smooth<MODE, 8, 8>, phase_grid(b, ph, 3), 256, s, b.plan, ph, pairs);
  early = true;
}

// The whole batched solve, enqueued on `s` while it is being captured: the
// initial defect pass and begin test, a WHILE node whose body (captured from
// `body`) is one V-cycle of every iterating scene plus the defect pass and
// the cycle tests, then the p = 0 fill of scenes whose rhs vanished.
cudaError_t batch_solve_enqueue(const BatchSolve& b, cudaStream_t s, cudaStream_t body) {
  const int rows = b.defect_rows[0];
  if (b.init_ph.second > 0)
    (rows == 2 ? k_batch_defect_init<2> : rows == 4 ? k_batch_defect_init<4> : k_batch_defect_init<8>)<<<
        b.init_ph.second, 32 * DEFECT_WARPS, 0, s>>>(b.scenes, b.items + b.init_ph.first, b.defect_rows[1]);
  cudaStreamCaptureStatus cst;
  cudaGraph_t cap = nullptr;
  cudaError_t err = cudaStreamGetCaptureInfo(s, &cst, nullptr, &cap, nullptr, nullptr, nullptr);
  cudaGraphConditionalHandle h = 0;
  if (err == cudaSuccess) err = cudaGraphConditionalHandleCreate(&h, cap, 0, cudaGraphCondAssignDefault);
  if (err != cudaSuccess) return err;
  k_batch_begin<<<1, 1024, 0, s>>>(b.plan, h);
  const cudaGraphNode_t* deps = nullptr;
  size_t ndeps = 0;
  err = cudaStreamGetCaptureInfo(s, &cst, nullptr, &cap, &deps, nullptr, &ndeps);
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node = nullptr;
  if (err == cudaSuccess) err = cudaGraphAddNode(&node, cap, deps, nullptr, ndeps, &cp);
  if (err == cudaSuccess) err = cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies);
  if (err == cudaSuccess)
    err = cudaStreamBeginCaptureToGraph(body, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal);
  if (err != cudaSuccess) return err;
  // each but the body's first may start while the one before it drains
  // (launch_dependent): 12 uneven scenes up to 512^2, three steps 8.1 -> 7.5 ms
  const int D = b.depth;
  bool early = false;
  for (int d = 0; d < D; d++) launch_batch_smooth<MODE_PRE>(body, b, b.pre, d, early);
  launch_dependent(early, b.tail_threads > 512 ? k_batch_tail<64> : k_batch_tail<32>, phase_grid(b, D, 1), b.tail_threads,
                   body, b.plan, D);
  early = true;
  for (int d = 0; d < D; d++) launch_batch_smooth<MODE_POST>(body, b, b.post, D + 1 + d, early);
  if (b.max_items[2 * D + 1] > 0)
    launch_dependent(early, rows == 2 ? k_batch_defect<2> : rows == 4 ? k_batch_defect<4> : k_batch_defect<8>,
                     phase_grid(b, 2 * D + 1, 8), 32 * DEFECT_WARPS, body, b.plan, 2 * D + 1, b.defect_rows[1]);
  launch_dependent(early, k_batch_check, 1, 1024, body, b.plan, h);
  cudaGraph_t done = nullptr;
  err = cudaStreamEndCapture(body, &done);
  if (err != cudaSuccess) return err;
  k_batch_zero<<<b.zero_ph.second, 256, 0, s>>>(b.scenes, b.items + b.zero_ph.first);
  return cudaGetLastError();
}

}  // namespace fl
