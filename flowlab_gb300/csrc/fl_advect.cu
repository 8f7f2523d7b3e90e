// Semi-Lagrangian / MacCormack advection of the MAC velocity and the dye
// (src/core/advect.ts:41-312; the reference's WGSL twin is
// src/gpu/advect.wgsl:225-356).
//
// Velocity: one launch over (nx+1) x (ny+1) threads covers both face grids —
// thread (i,j) owns u-face (i,j) where it exists and v-face (i,j) where it
// exists. MacCormack is two launches: the forward pass writes uHat, the
// correction fuses the reverse pass (read only at its own face) with the
// clamp, as the reverse pass's value is needed nowhere else.
//
// Dye: one backtrace per dye cell serves all three channels. The correction
// launch (or the forward launch for semi-Lagrangian) also applies the step's
// per-channel decay and the dye inlet patch, in that order (simulation.ts:
// 569-581), so the dye is touched once per step after advection.
//
// All reads of the carrier and source fields are gathers through the
// read-only cache; at the 1024^2 working set they are served from L2.
#include "fl_internal.h"

namespace fl {

// advect.ts:41-55 (FRESH: sample's)
template <bool FRESH = false, class S>
__device__ __forceinline__ void backtrace(const float* uc, const float* vc, int nx, int ny, const S& h, float x,
                                          float y, float u0, float v0, float dt, float& bx, float& by) {
  float midX = x - 0.5f * dt * u0;
  float midY = y - 0.5f * dt * v0;
  bx = x - dt * sample_u<FRESH>(uc, nx, ny, h, midX, midY);
  by = y - dt * sample_v<FRESH>(vc, nx, ny, h, midX, midY);
}

// The carrier at a face's own position, where the face holds only one of its
// components: with h a power of two (x / h exact) an interior face's four
// neighbours of the other kind with weights 1/2, otherwise the general sample.
__device__ __forceinline__ float v_at_u_face(const float* __restrict__ v, int nx, int ny, const SpacingPow2&, int i,
                                             int j, float, float) {
  return sample(v, Stencil{i - 1 + j * nx, 0.5f, 0.5f}, nx);
}
__device__ __forceinline__ float v_at_u_face(const float* __restrict__ v, int nx, int ny, const SpacingAny& h, int,
                                             int, float x, float y) {
  return sample_v(v, nx, ny, h, x, y);
}
__device__ __forceinline__ float u_at_v_face(const float* __restrict__ u, int nx, int ny, const SpacingPow2&, int i,
                                             int j, float, float) {
  return sample(u, Stencil{i + (j - 1) * (nx + 1), 0.5f, 0.5f}, nx + 1);
}
__device__ __forceinline__ float u_at_v_face(const float* __restrict__ u, int nx, int ny, const SpacingAny& h, int,
                                             int, float x, float y) {
  return sample_u(u, nx, ny, h, x, y);
}

// MODE 0: forward pass (advectFaces with src = carrier), writes `out`; with
//         `at` (MacCormack) also the offset of the backtraced point's stencil,
//         as an integer in the correction's output.
// MODE 1: MacCormack correction: `hat` is the forward result, `out` holds the
//         stencil offsets and receives clamp(hat + 0.5*(in - reverse(hat)))
//         (advect.ts:177-210).
// Bound by instruction issue (67% active) and the chains of gathers. Both
// launches of a MacCormack step in a graph: 1024^2 32.2 us (47.1 with the
// samplers' floor, index and division as conversion and division instructions
// and the two faces one after the other), 256^2 6.2 (9.6).
template <int MODE, class S>
__device__ __forceinline__ void advect_faces(int nx, int ny, const S& h, const float* __restrict__ u_in,
                                             const float* __restrict__ v_in, const float* u_hat, const float* v_hat,
                                             float* u_out, float* v_out, const uint8_t* __restrict__ label,
                                             const StepScalars* __restrict__ sc, float* u_at, float* v_at) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const float dt = MODE == 0 ? sc->dt : -sc->dt;
  // Both faces go through the arithmetic together, without branches, so that
  // their chains of gathers overlap; a face that is not advected (beside a
  // solid cell, or outside the grid) stands in for one that is in range.
  const bool u_in_grid = i <= nx && j < ny, v_in_grid = i < nx && j <= ny;
  const bool u_fixed = solid_or_outside(label, nx, ny, i - 1, j) || solid_or_outside(label, nx, ny, i, j);
  const bool v_fixed = solid_or_outside(label, nx, ny, i, j - 1) || solid_or_outside(label, nx, ny, i, j);
  const int iu = u_fixed ? 1 : i, ju = u_fixed ? 0 : j, iv = v_fixed ? 0 : i, jv = v_fixed ? 1 : j;
  const int ku = iu + ju * (nx + 1), kv = iv + jv * nx;
  const float xu = (float)iu * h.h, yu = ((float)ju + 0.5f) * h.h;
  const float xv = ((float)iv + 0.5f) * h.h, yv = (float)jv * h.h;
  const float uu = u_in[ku], vv = v_in[kv];
  const float vu = v_at_u_face(v_in, nx, ny, h, iu, ju, xu, yu);
  const float uv = u_at_v_face(u_in, nx, ny, h, iv, jv, xv, yv);
  float bxu, byu, bxv, byv;
  backtrace(u_in, v_in, nx, ny, h, xu, yu, uu, vu, dt, bxu, byu);
  backtrace(u_in, v_in, nx, ny, h, xv, yv, uv, vv, dt, bxv, byv);
  const Stencil pu = stencil_u(nx, ny, h, bxu, byu), pv = stencil_v(nx, ny, h, bxv, byv);
  // the correction's launch starts while the forward pass drains: only what
  // that wrote (hat, the offsets in out) is read after the wait
  if (MODE == 1) {
    dep_wait();
    dep_trigger();
  }
  float ru, rv;
  if (MODE == 0) {
    ru = sample(u_in, pu, nx + 1);
    rv = sample(v_in, pv, nx);
  } else {
    const int au = u_fixed ? 0 : __float_as_int(u_out[ku]), av = v_fixed ? 0 : __float_as_int(v_out[kv]);
    ru = clamp_at(u_in, au, nx + 1, u_hat[ku] + 0.5f * (uu - sample<true>(u_hat, pu, nx + 1)));
    rv = clamp_at(v_in, av, nx, v_hat[kv] + 0.5f * (vv - sample<true>(v_hat, pv, nx)));
  }
  if (u_in_grid) {
    const int k = i + j * (nx + 1);
    if (MODE == 0 && u_at != nullptr) u_at[k] = __int_as_float(pu.k);
    u_out[k] = u_fixed ? u_in[k] : ru;
  }
  if (v_in_grid) {
    const int k = i + j * nx;
    if (MODE == 0 && v_at != nullptr) v_at[k] = __int_as_float(pv.k);
    v_out[k] = v_fixed ? v_in[k] : rv;
  }
}

template <int MODE>
__global__ void __launch_bounds__(256) k_advect_velocity(int nx, int ny, Spacing h, const float* __restrict__ u_in,
                                                         const float* __restrict__ v_in, const float* u_hat,
                                                         const float* v_hat, float* u_out, float* v_out,
                                                         const uint8_t* __restrict__ label,
                                                         const StepScalars* __restrict__ sc, float* u_at,
                                                         float* v_at) {
  if (MODE == 0) dep_trigger();
  if (h.pow2)
    advect_faces<MODE>(nx, ny, SpacingPow2(h), u_in, v_in, u_hat, v_hat, u_out, v_out, label, sc, u_at, v_at);
  else
    advect_faces<MODE>(nx, ny, SpacingAny(h), u_in, v_in, u_hat, v_hat, u_out, v_out, label, sc, u_at, v_at);
}

// Dye. MODE 0 forward (advect.ts:241-270), MODE 1 correction (advect.ts:
// 294-311); the backtraced point's stencil offset passes from one to the other
// in `at`, the first plane of the correction's output. TAIL applies decay then
// the inlet patch (simulation.ts:569-581, dye.ts:158-175) to the value this
// thread writes.
template <int MODE, bool TAIL, class S>
__device__ __forceinline__ void advect_cells(int nx, int ny, const S& h, int dnx, int dny, const S& dh,
                                             const float* u, const float* v, const float* __restrict__ q_in,
                                             const float* q_hat, float* q_out,
                                             const uint8_t* __restrict__ label, const StepScalars* __restrict__ sc,
                                             const float* __restrict__ patch, int pi0, int pj0, int pnx, int pny,
                                             float* at) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= dnx || j >= dny) return;
  // 64-bit: the three planes together may hold more than 2^31 values
  const long cells = (long)dnx * dny;
  const int k = i + j * dnx;
  const float dt = sc->dt;
  const float ratio = dh.h / h.h;
  const int lj = (int)floorf(((float)j + 0.5f) * ratio);
  const int li = (int)floorf(((float)i + 0.5f) * ratio);
  float q[DYE_CHANNELS];
  if (solid_or_outside(label, nx, ny, li, lj)) {
#pragma unroll
    for (int c = 0; c < DYE_CHANNELS; c++) q[c] = q_in[k + c * cells];
    if (MODE == 1) {
      dep_wait();
      dep_trigger();
    }
  } else {
    const float x = ((float)i + 0.5f) * dh.h;
    const float y = ((float)j + 0.5f) * dh.h;
    // u and v are the projection's, which the forward pass starts behind; the
    // correction starts once every block of that pass has seen its end
    constexpr bool FRESH = MODE == 0;
    const float u0 = sample_u<FRESH>(u, nx, ny, h, x, y);
    const float v0 = sample_v<FRESH>(v, nx, ny, h, x, y);
    float bx, by;
    backtrace<FRESH>(u, v, nx, ny, h, x, y, u0, v0, MODE == 0 ? dt : -dt, bx, by);
    const Stencil p = stencil_p(dnx, dny, dh, bx, by);
    if (MODE == 0) {
      if (at != nullptr) at[k] = __int_as_float(p.k);
#pragma unroll
      for (int c = 0; c < DYE_CHANNELS; c++) q[c] = sample(q_in + c * cells, p, dnx);
    } else {
      dep_wait();  // hat and the offset in q_out are the forward pass's, whose end this launch need not await
      dep_trigger();
      const int ck = __float_as_int(q_out[k]);
#pragma unroll
      for (int c = 0; c < DYE_CHANNELS; c++) {
        const float corrected =
            q_hat[k + c * cells] + 0.5f * (q_in[k + c * cells] - sample<true>(q_hat + c * cells, p, dnx));
        q[c] = clamp_at(q_in + c * cells, ck, dnx, corrected);
      }
    }
  }
  if (TAIL) {
#pragma unroll
    for (int c = 0; c < DYE_CHANNELS; c++) {
      const float keep = sc->keep[c];
      if (keep != 1.0f) q[c] *= keep;
    }
    if (patch != nullptr) {
      const int pi = i - pi0, pj = j - pj0;
      if (pi >= 0 && pj >= 0 && pi < pnx && pj < pny) {
        const long pc = (long)pnx * pny;  // 64-bit: five planes
        const int s = pi + pj * pnx;
        const float cov = patch[DYE_CHANNELS * pc + s];
        if (cov != 0.0f) {
#pragma unroll
          for (int c = 0; c < DYE_CHANNELS; c++) q[c] += cov * (patch[c * pc + s] - q[c]);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < DYE_CHANNELS; c++) q_out[k + c * cells] = q[c];
}

template <int MODE, bool TAIL>
__global__ void __launch_bounds__(256) k_advect_dye(int nx, int ny, Spacing h, int dnx, int dny, Spacing dh,
                                                    const float* u, const float* v, const float* __restrict__ q_in,
                                                    const float* q_hat, float* q_out,
                                                    const uint8_t* __restrict__ label,
                                                    const StepScalars* __restrict__ sc,
                                                    const float* __restrict__ patch, int pi0, int pj0, int pnx,
                                                    int pny, float* at) {
  if (MODE == 0) {
    dep_wait();  // u and v are the launch before's
    dep_trigger();
  }
  if (h.pow2 && dh.pow2)
    advect_cells<MODE, TAIL>(nx, ny, SpacingPow2(h), dnx, dny, SpacingPow2(dh), u, v, q_in, q_hat, q_out, label, sc,
                             patch, pi0, pj0, pnx, pny, at);
  else
    advect_cells<MODE, TAIL>(nx, ny, SpacingAny(h), dnx, dny, SpacingAny(dh), u, v, q_in, q_hat, q_out, label, sc,
                             patch, pi0, pj0, pnx, pny, at);
}

void launch_advect_velocity(cudaStream_t s, int nx, int ny, float h, int mac, const float* u_in, const float* v_in,
                            float* u_hat, float* v_hat, float* u_out, float* v_out, const uint8_t* label,
                            const StepScalars* sc) {
  const Spacing hs = make_spacing(h);
  dim3 blk(32, 8);
  dim3 grd((nx + 1 + blk.x - 1) / blk.x, (ny + 1 + blk.y - 1) / blk.y);
  if (mac) {
    // the forward pass leaves its stencils' offsets in the correction's output
    k_advect_velocity<0><<<grd, blk, 0, s>>>(nx, ny, hs, u_in, v_in, nullptr, nullptr, u_hat, v_hat, label, sc, u_out,
                                             v_out);
    launch_dependent(true, k_advect_velocity<1>, grd, blk, s, nx, ny, hs, u_in, v_in, u_hat, v_hat, u_out, v_out, label,
                     sc, nullptr, nullptr);
  } else {
    k_advect_velocity<0><<<grd, blk, 0, s>>>(nx, ny, hs, u_in, v_in, nullptr, nullptr, u_out, v_out, label, sc,
                                             nullptr, nullptr);
  }
}

cudaError_t preload_advect_kernels() {
  cudaFuncAttributes a;
  cudaError_t err = cudaFuncGetAttributes(&a, k_advect_velocity<0>);
  if (err == cudaSuccess) err = cudaFuncGetAttributes(&a, k_advect_velocity<1>);
  return err;
}

void launch_advect_dye(cudaStream_t s, int nx, int ny, float h, int dnx, int dny, float dh, int mac, const float* u,
                       const float* v, const float* q_in, float* q_hat, float* q_out, const uint8_t* label,
                       const StepScalars* sc, bool tail, const float* patch, int pi0, int pj0, int pnx, int pny,
                       bool early) {
  const Spacing hs = make_spacing(h), ds = make_spacing(dh);
  dim3 blk(32, 8);
  dim3 grd((dnx + blk.x - 1) / blk.x, (dny + blk.y - 1) / blk.y);
  if (mac) {
    launch_dependent(early, k_advect_dye<0, false>, grd, blk, s, nx, ny, hs, dnx, dny, ds, u, v, q_in, nullptr, q_hat,
                     label, sc, nullptr, 0, 0, 0, 0, q_out);
    launch_dependent(true, tail ? k_advect_dye<1, true> : k_advect_dye<1, false>, grd, blk, s, nx, ny, hs, dnx, dny, ds,
                     u, v, q_in, q_hat, q_out, label, sc, tail ? patch : nullptr, pi0, pj0, pnx, pny, nullptr);
  } else {
    launch_dependent(early, tail ? k_advect_dye<0, true> : k_advect_dye<0, false>, grd, blk, s, nx, ny, hs, dnx, dny, ds,
                     u, v, q_in, nullptr, q_out, label, sc, tail ? patch : nullptr, pi0, pj0, pnx, pny, nullptr);
  }
}

}  // namespace fl
