// gs_raster.cu -- the tiled rasteriser: forward composite, loss + stats and
// the back-to-front backward of the reference's render pass
// (shaders.js:544-700), over a shared (view, tile) work queue.
//
// k_raster_warp runs every pass but the stored-state one: one warp per 8x8
// block of a tile (TILE = 8, 16 or 32), two pixels per lane.  It is described
// at the kernel.
//
// k_raster_stored (forward + loss + backward that reads the transmittance the
// forward saved, instead of recovering it from the final one): one CTA per
// tile, one thread per pixel, each warp covering an 8x4 block.  Splat records
// of the tile's sorted entries are staged in shared memory BATCH at a time;
// the block leaves the tile's forward when __syncthreads_count (a block-wide
// ballot) finds every pixel saturated.  Each warp records, per entry, whether
// any of its pixels composited it (a ballot bit in shared memory), and the
// backward walks the marked entries back to front (entries past the bit
// capacity are all visited).
//
// The ten gradient contributions of each pixel are truncated to i32 fixed
// point (the reference's i32(clamp(v*16384, +-1e9))) and summed exactly, with
// a warp REDUX per slot and integer atomics.  Integer sums commute, so results
// are bit-identical in any order -- the deterministic mode is the only mode.
//
// Control flow is warp-uniform (votes); per-lane work runs predicated, so
// no divergent branch needs a reconvergence scaffold in the hot loops.
// The per-pair arithmetic is the canonical FP32 sequence the CPU
// restatement performs.  The 2^14 fixed-point scale is folded into upstream
// factors (gC, hence galpha, which is accumulated from the scaled gC):
// scaling by a power of two is exact, so every truncated integer equals the
// one the unfolded sequence produces.  The
// +-1e9 clamp is skipped when the scaled galpha is below 1e7: the conic
// normaliser bounds every slot by 80 |galpha * 2^14| (slots 7-9 by
// |gC * 2^14|), so the clamp cannot change a value then.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gs_common.cuh"
#include "gs_kernels.h"

namespace gs {

constexpr int MASKW = 128;        // ballot-bit words per warp: entries 0..4095 of a tile
constexpr uint32_t FULL = 0xFFFFFFFFu;

// e = max(fma(fma(cA/2, dx, cB*dy), dx, ((cC/2)*dy)*dy), 0); r0 = (mx, my, cA/2, cB)
__device__ __forceinline__ float pairExponent(const float4& r0, float hC, float dx, float dy) {
  const float u = __fmaf_rn(r0.z, dx, r0.w * dy);
  return fmaxf(__fmaf_rn(u, dx, (hC * dy) * dy), 0.0f);
}

// trunc(clamp(x, -1e9, 1e9)) for an already scaled value
__device__ __forceinline__ int32_t fix_scaled(float x) { return __float2int_rz(fminf(fmaxf(x, -1.0e9f), 1.0e9f)); }


// Which of the tile's 8x4 warp blocks (k_raster_stored) can the splat reach?  Bit w = warp w
// (block row w / (TILE/8), column w % (TILE/8)).  For each 4-row band, the
// splat's pixels lie within |dx - kA dy| <= sqrt(p - q dmin^2) (cull
// parameters (p, q, kA) from the projection; dmin = the band's smallest |dy|),
// an x interval checked against each block of the band.  Slack covers this
// FP32 evaluation, so a cleared bit means no pixel of the block can pass the
// rasteriser's cutoffs: skipping the entry there changes nothing.
template <int TILE>
__device__ __forceinline__ uint32_t warp_block_mask(const float4 cq, float mx, float my, int tx, int ty) {
  constexpr int NB = TILE / 4, WPR = TILE / 8;
  constexpr uint32_t ALL = NB * WPR >= 32 ? 0xFFFFFFFFu : (1u << (NB * WPR)) - 1u;
  if (!(cq.x < 3.0e38f)) return ALL;
  uint32_t m = 0;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const float Y0 = ((float)(ty * TILE + 4 * b) + 0.5f) - my;
    float xl, xr;
    if (!bandInterval(cq, Y0, Y0 + 3.0f, xl, xr)) continue;
#pragma unroll
    for (int wb = 0; wb < WPR; ++wb) {
      const float bx0 = ((float)(tx * TILE + 8 * wb) + 0.5f) - mx;
      if (bx0 + 7.0f >= xl && bx0 <= xr) m |= 1u << (b * WPR + wb);
    }
  }
  return m;
}

#ifndef GS_RASTER16_MIN_BLOCKS
#define GS_RASTER16_MIN_BLOCKS 5  // resident 16x16-tile blocks per SM the register allocation must allow
#endif
// TILE x TILE pixels per CTA, one per thread; warps cover 8x4 blocks.
template <int TILE, int BATCH>
__global__ void __launch_bounds__(TILE * TILE, TILE == 16 ? GS_RASTER16_MIN_BLOCKS : TILE == 8 ? 16 : 1)
    k_raster_stored(RasterArgs a) {
  constexpr int RT = TILE;
  constexpr int RTHREADS = TILE * TILE;
  constexpr int NW = RTHREADS / 32;  // warps
  constexpr int WPR = TILE / 8;      // 8-wide warp blocks per tile row
  static_assert(BATCH % 32 == 0, "batches hold whole ballot words");
  __shared__ RenderRec s_rec[BATCH];
  __shared__ uint32_t s_id[BATCH];
  __shared__ int32_t s_acc[BATCH * 10];
  __shared__ uint32_t s_mask[NW * MASKW];
  __shared__ uint32_t s_live[NW][BATCH / 32];  // per warp: staged entries its block can reach
  __shared__ uint32_t s_item;
  __shared__ uint32_t s_redu[NW][5];
  __shared__ uint32_t s_endmax[NW];
  __shared__ __align__(16) int32_t s_stage[NW][12];  // per warp: the 10 sums of one entry

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int lx = (wid % WPR) * 8 + (lane & 7);
  const int ly = (wid / WPR) * 4 + (lane >> 3);
  const float E_CUT = a.eCut, A_MIN = a.aMin;
  uint32_t* wmask = s_mask + wid * MASKW;

  for (int k = tid; k < BATCH * 10; k += RTHREADS) s_acc[k] = 0;

  for (uint32_t iter = 0;; ++iter) {
    // ---- next work item (a global tile of the batch) ----
    if (tid == 0) s_item = a.workCounter ? atomicAdd(a.workCounter, 1u) : (iter == 0 ? blockIdx.x : 0xFFFFFFFFu);
    __syncthreads();
    const uint32_t item = s_item;
    __syncthreads();
    if (item >= a.totalTiles) break;
    const uint32_t gt = a.workOrder ? a.workOrder[item] : item;
    int v = 0;
    while (v + 1 < a.V && a.cams[v + 1].tileBase <= gt) ++v;
    const DevCam& c = a.cams[v];
    const uint32_t t = gt - c.tileBase;
    const int tx = (int)(t % (uint32_t)c.tilesX), ty = (int)(t / (uint32_t)c.tilesX);
    const int x = tx * RT + lx, y = ty * RT + ly;
    const bool inside = x < c.W && y < c.H;
    const float px = (float)x + 0.5f, py = (float)y + 0.5f;
    const uint2 rg = a.ranges[gt];
    const uint32_t s = rg.x, e = rg.y;
    const size_t pix = (size_t)c.pixBase + (size_t)y * c.W + x;
    const RenderRec* recs = a.recs + (size_t)v * a.n;
    const float4* cullRecs = a.cullRecs + (size_t)v * a.n;

    float T = 1.0f;
    float C0 = 0.0f, C1 = 0.0f, C2 = 0.0f;
    uint32_t cnt = e - s;  // one past the last processed entry (relative)
    {
      bool done = !inside;
      for (int k = lane; k < MASKW; k += 32) wmask[k] = 0u;
      __syncwarp();
      for (uint32_t base = s; base < e; base += BATCH) {
        if (__syncthreads_count(!done) == 0) break;
        const uint32_t nb = min((uint32_t)BATCH, e - base);
        // stage the batch; each staging thread also finds which warp blocks
        // its entry can reach, and a ballot per warp block transposes that
        // into one word per 32 entries
        for (uint32_t kb = 0; kb < (uint32_t)BATCH; kb += RTHREADS) {
          const uint32_t k = kb + tid;
          uint32_t m = 0;
          if (k < nb) {
            const uint32_t id = a.ids[base + k] & a.idMask;
            s_id[k] = id;
            const RenderRec rec = recs[id];
            s_rec[k] = rec;
            m = warp_block_mask<TILE>(cullRecs[id], rec.r0.x, rec.r0.y, tx, ty);
          }
          const uint32_t word = (kb >> 5) + (uint32_t)wid;
#pragma unroll
          for (int w = 0; w < NW; ++w) {
            const uint32_t bw = __ballot_sync(FULL, (m >> w) & 1u);
            if (lane == 0 && word < (uint32_t)(BATCH / 32)) s_live[w][word] = bw;
          }
        }
        __syncthreads();
        if (!__all_sync(FULL, done)) {
          const uint32_t rbase = base - s;
          for (uint32_t jw = 0; jw < nb; jw += 32) {  // one ballot word per 32 entries
            uint32_t live = s_live[wid][jw >> 5];  // entries this warp's block can reach
            uint32_t bits = 0;
            while (live) {
              const uint32_t jj = (uint32_t)__ffs(live) - 1u;
              live &= live - 1u;
              const RenderRec& rr = s_rec[jw + jj];
              const float4 r0 = rr.r0;
              const float4 r1 = rr.r1;
              const float dx = px - r0.x, dy = py - r0.y;
              const float ee = pairExponent(r0, r1.x, dx, dy);
              const bool c1 = !done && ee <= E_CUT;
              // warp-uniform branch; the body runs predicated per lane (lanes
              // outside the cutoff see a clamped exponent and are masked off)
              if (__any_sync(FULL, c1)) {
                const float araw = r1.y * gexp(-fminf(ee, 80.0f));
                const float alpha = fminf(0.99f, araw);
                const bool c2 = c1 && alpha >= A_MIN;
                if (c2) a.tStore[(size_t)(base + jw + jj) * RTHREADS + tid] = T;
                const float ta = T * alpha;
                const float cb = rr.r2.x;
                if (c2) {
                  C0 = __fmaf_rn(ta, r1.z, C0);
                  C1 = __fmaf_rn(ta, r1.w, C1);
                  C2 = __fmaf_rn(ta, cb, C2);
                  T = T * (1.0f - alpha);
                  if (T < 1e-4f) { done = true; cnt = rbase + jw + jj + 1; }
                }
                bits |= (__ballot_sync(FULL, c2) != 0u ? 1u : 0u) << jj;
              }
            }
            const uint32_t w = (rbase + jw) >> 5;
            if (lane == 0 && w < MASKW) wmask[w] = bits;
            if (__all_sync(FULL, done)) break;
          }
        }
        __syncthreads();
      }
      C0 = C0 + T * c.bg[0];
      C1 = C1 + T * c.bg[1];
      C2 = C2 + T * c.bg[2];
      if (inside) {
        a.outImg[pix] = make_float4(C0, C1, C2, 1.0f - T);
        a.finalT[pix] = T;
        a.endIdx[pix] = cnt;
      }
    }

    {
      // ---- loss (shaders.js:589-618) ----
      bool lossOk = false;
      float g16_0 = 0.0f, g16_1 = 0.0f, g16_2 = 0.0f;  // gC * 2^14
      uint32_t st0 = 0, st1 = 0, st2 = 0;
      int32_t cg6 = 0, cg7 = 0;
      if (inside) {
        const uint32_t pi = (uint32_t)(y * c.W + x);
        const uint32_t packed = a.targets[(size_t)c.offset + pi];
        if ((packed >> 24) != 0u) {
          lossOk = true;
          const float t0 = (float)(packed & 0xFFu) / 255.0f;
          const float t1 = (float)((packed >> 8) & 0xFFu) / 255.0f;
          const float t2 = (float)((packed >> 16) & 0xFFu) / 255.0f;
          st2 = 1u;
          const float gain = c.gain;
          const float er0 = (gain * C0 + c.bias) - t0;
          const float er1 = (gain * C1 + c.bias) - t1;
          const float er2 = (gain * C2 + c.bias) - t2;
          st0 = u32sat((er0 * er0 + er1 * er1 + er2 * er2) * 16.0f + dither(pi));
          const float D2 = 9.0000000000000003e-04f;  // f32(0.03 * 0.03), a WGSL const-expression
          const float rt0 = sqrtf(er0 * er0 + D2), rt1 = sqrtf(er1 * er1 + D2), rt2 = sqrtf(er2 * er2 + D2);
          const float eg0 = er0 / rt0, eg1 = er1 / rt1, eg2 = er2 / rt2;
          g16_0 = (gain * eg0) * FIXED; g16_1 = (gain * eg1) * FIXED; g16_2 = (gain * eg2) * FIXED;
          const float lossv = (rt0 + rt1 + rt2) - 8.9999999999999997e-02f;  // f32(3 * 0.03)
          st1 = u32sat(lossv * 32768.0f);
          cg6 = fixq((eg0 * C0 + eg1 * C1 + eg2 * C2) * gain, FIXCAM);
          cg7 = fixq(eg0 + eg1 + eg2, FIXCAM);
        }
      }
      // slots 7-9 stay within +-1e9 without clamping when |gC * 2^14| < 9e8
      const bool pixFast = fabsf(g16_0) < 9.0e8f && fabsf(g16_1) < 9.0e8f && fabsf(g16_2) < 9.0e8f;
      // block sums of the per-pixel stats (wrapping u32 / i32, as the
      // reference's atomics) and the largest end index of the tile
      const uint32_t myEnd = lossOk ? cnt : 0u;
      {
        const uint32_t r0 = __reduce_add_sync(FULL, st0);
        const uint32_t r1 = __reduce_add_sync(FULL, st1);
        const uint32_t r2 = __reduce_add_sync(FULL, st2);
        const uint32_t r3 = __reduce_add_sync(FULL, (uint32_t)cg6);
        const uint32_t r4 = __reduce_add_sync(FULL, (uint32_t)cg7);
        const uint32_t mx = __reduce_max_sync(FULL, myEnd);
        if (lane == 0) {
          s_redu[wid][0] = r0; s_redu[wid][1] = r1; s_redu[wid][2] = r2;
          s_redu[wid][3] = r3; s_redu[wid][4] = r4;
          s_endmax[wid] = mx;
        }
      }
      __syncthreads();
      if (tid < 5) {
        uint32_t sum = 0;
        for (int w = 0; w < NW; ++w) sum += s_redu[w][tid];
        if (sum) {
          if (tid < 3) atomicAdd(&a.stats[tid], sum);
          else atomicAdd(&a.gradCam[c.camIdx * 8u + 3u + (uint32_t)tid], (int32_t)sum);
        }
      }
      uint32_t endMax = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) endMax = max(endMax, s_endmax[w]);
      // ---- backward (shaders.js:632-700) ----
      float S0 = c.bg[0] * T, S1 = c.bg[1] * T, S2 = c.bg[2] * T;
      float Ta = T;
      int32_t* gradP = a.gradP + (size_t)v * a.n * GP_STRIDE;
      for (uint32_t hi = endMax; hi > 0;) {
        const uint32_t lo = hi > (uint32_t)BATCH ? hi - BATCH : 0u;
        const uint32_t nb = hi - lo;
        __syncthreads();
        for (uint32_t k = tid; k < nb; k += RTHREADS) {
          const uint32_t id = a.ids[s + lo + k] & a.idMask;
          s_id[k] = id;
          s_rec[k] = recs[id];
        }
        __syncthreads();
        // this warp's entries in [lo, hi), back to front, one ballot word at a time
        for (int32_t w = (int32_t)((hi - 1) >> 5); w >= (int32_t)(lo >> 5); --w) {
          const uint32_t wb = (uint32_t)w << 5;
          uint32_t word = (uint32_t)w < (uint32_t)MASKW ? wmask[w] : FULL;
          if (wb + 32u > hi) word &= FULL >> (wb + 32u - hi);
          if (wb < lo) word &= FULL << (lo - wb);
          while (word) {
            const uint32_t bit = 31u - (uint32_t)__clz(word);
            word &= ~(1u << bit);
            const uint32_t j = wb + bit;
            const RenderRec& rr = s_rec[j - lo];
            const float4 r0 = rr.r0;
            const float4 r1 = rr.r1;
            const float4 r2 = rr.r2;
            // Straight-line body, predicated per lane: lanes that do not
            // composite this entry (past their end, outside a cutoff) compute
            // on a clamped exponent and have their contribution zeroed
            // through galpha and aT, and keep S and Ta.  Compositing lanes
            // perform exactly the canonical sequence.
            const float dx = px - r0.x, dy = py - r0.y;
            const float ee = pairExponent(r0, r1.x, dx, dy);
            const float G = gexp(-fminf(ee, 80.0f));
            const float araw = r1.y * G;
            const float alpha = fminf(0.99f, araw);
            const bool c2 = j < myEnd && ee <= E_CUT && alpha >= A_MIN;
            if (!__any_sync(FULL, c2)) continue;
            const float inv = rcp_unit(1.0f - alpha);  // 1 - alpha in [0.01, 1]: IEEE 1/x exactly
            const float Tb = c2 ? a.tStore[(size_t)(s + j) * RTHREADS + tid] : 0.0f;
            const float aT = c2 ? alpha * Tb : 0.0f;
            const float g0 = __fmaf_rn(r1.z, Tb, -(S0 * inv));
            const float g1 = __fmaf_rn(r1.w, Tb, -(S1 * inv));
            const float g2 = __fmaf_rn(r2.x, Tb, -(S2 * inv));
            // galpha * 2^14, accumulated from gC * 2^14
            const float gal16 = c2 && !(araw > 0.99f) ? __fmaf_rn(g16_2, g2, __fmaf_rn(g16_1, g1, g16_0 * g0)) : 0.0f;
            const float ga16 = gal16 * araw;
            const float cA = r0.z + r0.z, cC = r1.x + r1.x;  // exact doubling of the stored halves
            const float gq16 = ga16 * r2.z;  // r2.z = -cnorm / 2
            const float gqx16 = gq16 * dx;
            float xs[10];
            xs[0] = ga16 * __fmaf_rn(cA, dx, r0.w * dy);
            xs[1] = ga16 * __fmaf_rn(r0.w, dx, cC * dy);
            xs[2] = gqx16 * dx;
            xs[3] = (gqx16 * dy) * 2.0f;
            xs[4] = (gq16 * dy) * dy;
            xs[5] = (gal16 * r2.y) * G;
            xs[6] = ga16 * r2.w;  // r2.w = 1 - opacity
            xs[7] = g16_0 * aT;
            xs[8] = g16_1 * aT;
            xs[9] = g16_2 * aT;
            uint32_t rsum[10];
            if (__all_sync(FULL, fabsf(gal16) < 1.0e7f && pixFast)) {
#pragma unroll
              for (int k = 0; k < 10; ++k) rsum[k] = __reduce_add_sync(FULL, (uint32_t)__float2int_rz(xs[k]));
            } else {
#pragma unroll
              for (int k = 0; k < 10; ++k) rsum[k] = __reduce_add_sync(FULL, c2 ? (uint32_t)fix_scaled(xs[k]) : 0u);
            }
            if (c2) {
              S0 = __fmaf_rn(r1.z, aT, S0);
              S1 = __fmaf_rn(r1.w, aT, S1);
              S2 = __fmaf_rn(r2.x, aT, S2);
              Ta = Tb;
            }
            // lane 0 stages the 10 warp sums; lanes 0-9 add one each
            if (lane == 0) {
              int4* st = reinterpret_cast<int4*>(s_stage[wid]);
              st[0] = make_int4((int)rsum[0], (int)rsum[1], (int)rsum[2], (int)rsum[3]);
              st[1] = make_int4((int)rsum[4], (int)rsum[5], (int)rsum[6], (int)rsum[7]);
              reinterpret_cast<int2*>(s_stage[wid])[4] = make_int2((int)rsum[8], (int)rsum[9]);
            }
            __syncwarp();
            if (lane < 10) atomicAdd(&s_acc[(j - lo) * 10 + (uint32_t)lane], s_stage[wid][lane]);
            __syncwarp();
          }
        }
        __syncthreads();
        for (uint32_t k = tid; k < nb * 10; k += RTHREADS) {
          const int32_t val = s_acc[k];
          if (val) {
            const uint32_t jl = k / 10, slot = k - jl * 10;
            atomicAdd(&gradP[(size_t)s_id[jl] * GP_STRIDE + slot], val);
            s_acc[k] = 0;
          }
        }
        hi = lo;
      }
    }
    __syncthreads();
  }
}

// Can the splat (cull parameters cq, mean (mx, my)) reach the 8x8 pixel block
// whose first pixel is (x0, y0)?  The same band test as warp_block_mask on an
// 8-row band.
__device__ __forceinline__ bool block_reach(const float4 cq, float mx, float my, int x0, int y0) {
  if (!(cq.x < 3.0e38f)) return true;
  const float Y0 = ((float)y0 + 0.5f) - my, X0 = ((float)x0 + 0.5f) - mx;
  float xl, xr;
  if (!bandIntervalMask(cq, Y0, Y0 + 7.0f, xl, xr)) return false;
  return X0 + 7.0f >= xl && X0 <= xr;
}

// e = max(fma(fma(cA/2, dx, cB*dy), dx, ((cC/2)*dy)*dy), 0) for two pixels
// that share dx; Bdy returns cB*dy.
__device__ __forceinline__ float2 pairExponent2(const float4& r0, float hC, float dx, float2 dy, float2& Bdy) {
  Bdy = __fmul2_rn(bc2(r0.w), dy);
  const float2 u = __ffma2_rn(bc2(r0.z), bc2(dx), Bdy);
  const float2 e = __ffma2_rn(u, bc2(dx), __fmul2_rn(__fmul2_rn(bc2(hC), dy), dy));
  return make_float2(fmaxf(e.x, 0.0f), fmaxf(e.y, 0.0f));
}

__device__ __forceinline__ void cp_async_rec(RenderRec* dst, const RenderRec* src) {
  cp_async16(&dst->r0, &src->r0);
  cp_async16(&dst->r1, &src->r1);
  cp_async16(&dst->r2, &src->r2);
}

// Shared memory by 32-bit address: the hot loops step such an address in one
// register.  (Indexing the arrays instead had the compiler form the address
// anew for every entry.)
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  uint32_t r;  // opaque, so that it stays in a register
  asm volatile("mov.u32 %0, %1;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)));
  return r;
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds1(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts4(uint32_t a, int x, int y, int z, int w) {
  asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts2(uint32_t a, int x, int y) {
  asm volatile("st.shared.v2.s32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
// *p += v unless v is 0, without a branch
__device__ __forceinline__ void red_nz(int32_t* p, int32_t v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %1, 0;\n @q red.global.add.s32 [%0], %1;\n}" ::"l"(p), "r"(v)
               : "memory");
}

constexpr uint32_t REDO = 8;  // entries past the cache whose exponentials are computed together

struct StagedRec {
  RenderRec rec;
  uint32_t id;   // splat
  uint32_t raw;  // place in its chunk of list entries
  uint32_t pad[2];
};
// The rasteriser: one warp per 8x8 pixel block of a tile, with no barrier
// between warps.  Lane l holds pixels (l % 8, l / 8) and (l % 8, l / 8 + 4),
// which share dx; every per-pixel operation runs on the pair as one packed
// instruction (or twice, for comparisons, selects and conversions).
//
// Forward: the tile's list is read 32 entries at a time.  An entry whose
// block bit is clear cannot reach the block (k_expand computed the bits; with
// MASKED off the warp tests the cull parameters itself); the records of the
// others are copied to shared memory with cp.async, compacted, one chunk
// ahead of the one being composited.
// Backward (BWD): walks the composited entries back to front.  The forward
// left their ids and, per pixel, the exponential G (0 where the pixel did not
// composite the entry) in the warp's slice of a cache in global memory, so the
// backward neither evaluates the exponential again nor tests the cutoffs.
// Entries past the slice (cacheCap of them fit) are recomputed from the list:
// the records staged a chunk ahead, the exponentials of eight entries computed
// together into shared memory, then taken in pairs like cached ones.  (One
// entry at a time, with its record, its exponential and the clamped sums in one
// chain, blocks with hundreds of entries past the slice took up to 29% longer
// than the kernel before this one: a step of 200k splats at 128x128, tile 8,
// 1155 us then, 1490 us, now 1378 us; at tile 16 2223, 1657, 1530 us.)
// The ten integer sums of an entry go from the warp straight to gradP.
//
// The backward takes two entries at a time and the forward is unrolled by
// two, so that one entry's chain of dependent instructions runs under the
// other's; that needs 96 registers, so 5 blocks (20 warps) per SM.  One entry at
// a time with 72 registers and 7 blocks is 1.2% slower on full grids and 5-9%
// slower where a few long blocks decide the time (an evaluation pass, one
// 1080p view: 6830 -> 6506 us; 555x419, 180k splats: 7009 -> 6376 us).
//
// What bounds it: instruction issue (69% active), with the conversions to
// integers (F2I: 8 cycles a warp) at 56% of their pipe and FMA at 60%.  Measured
// on 1M splats, two 1080p views: 2.01 ms, 1.57 G warp instructions; the block
// per tile of four warps it replaced, which met at a barrier every batch and
// recomputed G: 2.49 ms, 2.08 G.  The cache's traffic goes through DRAM (3.0 GB
// in that pass, 1.5 TB/s), loaded two entries ahead; without the cache a train
// step is 7% slower.
template <int TILE, bool MASKED, bool BWD>
__global__ void __launch_bounds__(RW_WARPS * 32, BWD ? 5 : 6) k_raster_warp(RasterArgs a) {
  constexpr int SUB = (TILE / 8) * (TILE / 8);  // 8x8 blocks per tile
  constexpr int SPR = TILE / 8;                 // of them in one row
  static_assert(!MASKED || TILE <= 16, "entry values carry at most four block bits");
  __shared__ StagedRec s_rec[RW_WARPS][2][32];
  __shared__ __align__(256) int32_t s_stage[BWD ? RW_WARPS : 1][4][16];
  __shared__ float2 s_redo[BWD ? RW_WARPS : 1][BWD ? REDO : 1][32];
  __shared__ uint32_t s_stat[3];
  __shared__ int32_t s_cam[MAX_VIEWS][2];

  const int wid = threadIdx.x >> 5;
  int lane;  // opaque, so that it stays in a register instead of being read again per entry
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  // alpha = min(0.99, w G) is tested as w G, which is the same for cutoffs up
  // to 0.99 (a larger one accepts nothing)
  const float E_CUT = a.eCut, A_MIN = a.aMin <= 0.99f ? a.aMin : __int_as_float(0x7F800000);
  const uint32_t ltm = (1u << lane) - 1u;
  if (BWD) {
    if (threadIdx.x < 3) s_stat[threadIdx.x] = 0u;
    if (threadIdx.x < 2 * MAX_VIEWS) (&s_cam[0][0])[threadIdx.x] = 0;
    if (threadIdx.x < RW_WARPS * 4) s_stage[threadIdx.x >> 2][threadIdx.x & 3][10] = 0;  // word 10 of each row
    __syncthreads();
  }
  const uint32_t warp = blockIdx.x * RW_WARPS + (uint32_t)wid;
  const uint32_t items = a.totalTiles * (uint32_t)SUB;
  // this warp's slice of the exponential cache: slots 2 to cacheCap + 1 keep
  // entries.  The slot after the last kept one takes the stores of entries
  // that are not kept, which for a full slice is slot 0 of the next one;
  // slots 0 and 1 are only ever loaded ahead of use, and never used.
  const uint32_t slice = BWD ? (warp % a.cacheWarps) * (a.cacheCap + 2u) : 0u;
  float2* const gFirst = BWD ? a.cacheG + ((size_t)(slice + 2u) * 32 + lane) : nullptr;
  uint32_t* const cacheId = BWD ? a.cacheId + slice : nullptr;

  for (uint32_t iter = 0;; ++iter) {
    uint32_t item = iter == 0 ? warp : 0xFFFFFFFFu;
    if (a.workCounter) {
      if (lane == 0) item = atomicAdd(a.workCounter, 1u);
      item = __shfl_sync(FULL, item, 0);
    }
    if (item >= items) break;
    const uint32_t ti = item / SUB, sub = item % SUB;
    const uint32_t gt = a.workOrder ? a.workOrder[ti] : ti;
    int v = 0;
    while (v + 1 < a.V && a.cams[v + 1].tileBase <= gt) ++v;
    const DevCam& c = a.cams[v];
    const uint32_t t = gt - c.tileBase;
    const int x = (int)(t % (uint32_t)c.tilesX) * TILE + (int)(sub % SPR) * 8 + (lane & 7);
    const int ya = (int)(t / (uint32_t)c.tilesX) * TILE + (int)(sub / SPR) * 8 + (lane >> 3), yb = ya + 4;
    const bool inA = x < c.W && ya < c.H, inB = x < c.W && yb < c.H;
    if (!__any_sync(FULL, inA)) continue;  // the block lies outside the image
    const float px = (float)x + 0.5f;
    const float2 py = make_float2((float)ya + 0.5f, (float)yb + 0.5f);
    const uint2 rg = a.ranges[gt];
    const uint32_t s = rg.x, e = rg.y;
    const RenderRec* recs = a.recs + (size_t)v * a.n;

    // Stage the chunk of entry values `val` (lane l: list entry base + l) into
    // buffer b: the live entries' records, compacted.  Returns their bits.
    auto stage = [&](uint32_t val, bool have, int b) {
      bool live = have;
      uint32_t id = val;
      if (MASKED) {
        id = val & ID_MASK;
        live = have && ((val >> (ID_BITS + sub)) & 1u);
      } else if (TILE > 8) {
        if (have) {
          const float4 cq = a.cullRecs[(size_t)v * a.n + id];
          const float2 m = *reinterpret_cast<const float2*>(&recs[id].r0);
          live = block_reach(cq, m.x, m.y, x - (lane & 7), ya - (lane >> 3));
        }
      }
      const uint32_t bits = __ballot_sync(FULL, live);
      if (live) {
        const uint32_t pos = (uint32_t)__popc(bits & ltm);
        StagedRec* d = &s_rec[wid][b][pos];
        cp_async_rec(&d->rec, recs + id);
        d->id = id;
        d->raw = (uint32_t)lane;
      }
      cp_async_commit();
      return bits;
    };

    // ---- forward ----
    // A pixel is done once its transmittance is below 1e-4; pixels outside the
    // image start at 0, so they never composite.
    float2 T = make_float2(inA ? 1.0f : 0.0f, inB ? 1.0f : 0.0f);
    float2 C0 = bc2(0.0f), C1 = bc2(0.0f), C2 = bc2(0.0f);
    uint32_t cntA = 0u, cntB = 0u;  // end index of a pixel that is done, 0 before
    float2* gp = gFirst;            // next cache slot
    uint32_t uncached = e;          // first list entry (at a chunk start) past the cache
    uint32_t seenEnd = s;           // one past the last chunk processed
    {
      auto load = [&](uint32_t base) { return base + lane < e ? a.ids[base + lane] : 0u; };
      int b = 0;
      uint32_t bits = stage(load(s), s + lane < e, 0);
      uint32_t nextVal = s + 32 < e ? load(s + 32) : 0u;
      for (uint32_t base = s; base < e; base += 32) {
        uint32_t nextBits = 0;
        if (base + 32 < e) {
          nextBits = stage(nextVal, base + 32 + lane < e, b ^ 1);
          nextVal = base + 64 < e ? load(base + 64) : 0u;
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncwarp();
        const uint32_t n = (uint32_t)__popc(bits);
        if (BWD && uncached == e && (uint32_t)((gp - gFirst) >> 5) + n > a.cacheCap) uncached = base;
        const uint32_t step = BWD && uncached == e ? 32u : 0u;
        uint32_t hit = 0;
        uint32_t kA = 0, kB = 0;  // last entry of the chunk that each pixel composited
        const StagedRec* sr = s_rec[wid][b];
#pragma unroll 2
        for (uint32_t k = 0; k < n; ++k, ++sr) {
          const float4 r0 = sr->rec.r0;
          const float4 r1 = sr->rec.r1;
          const float dx = px - r0.x;
          const float2 dy = __fadd2_rn(py, bc2(-r0.y));
          float2 Bdy;
          const float2 ee = pairExponent2(r0, r1.x, dx, dy, Bdy);
          // beyond the cutoff (at most 80) G may be anything: it is masked below
          const float2 G = gexp2(make_float2(-ee.x, -ee.y));
          const float2 araw = __fmul2_rn(bc2(r1.y), G);
          const bool c2a = T.x >= 1e-4f && ee.x <= E_CUT && araw.x >= A_MIN;
          const bool c2b = T.y >= 1e-4f && ee.y <= E_CUT && araw.y >= A_MIN;
          // a pixel that does not composite sees alpha 0: T stays exactly as it is, and C does while the colour is finite
          const float2 Gm = make_float2(c2a ? G.x : 0.0f, c2b ? G.y : 0.0f);
          const float2 aw = __fmul2_rn(bc2(r1.y), Gm);
          const float2 am = make_float2(fminf(0.99f, aw.x), fminf(0.99f, aw.y));
          const float2 ta = __fmul2_rn(T, am);
          C0 = __ffma2_rn(ta, bc2(r1.z), C0);
          C1 = __ffma2_rn(ta, bc2(r1.w), C1);
          C2 = __ffma2_rn(ta, bc2(sr->rec.r2.x), C2);
          T = __fmul2_rn(T, __fadd2_rn(bc2(1.0f), make_float2(-am.x, -am.y)));
          kA = c2a ? k : kA;
          kB = c2b ? k : kB;
          if (BWD) {
            __stcg(gp, Gm);
            hit >>= 1;
            if (__any_sync(FULL, c2a || c2b)) {
              hit |= 0x80000000u;
              gp += step;
            }
          }
        }
        hit = n ? hit >> (32u - n) : 0u;  // bit k: entry k
        if (step && ((hit >> lane) & 1u))
          __stcg(cacheId + ((uint32_t)((gp - gFirst) >> 5) - (uint32_t)__popc(hit & ~ltm)), s_rec[wid][b][lane].id);
        if (T.x < 1e-4f && cntA == 0u) cntA = base - s + s_rec[wid][b][kA].raw + 1u;
        if (T.y < 1e-4f && cntB == 0u) cntB = base - s + s_rec[wid][b][kB].raw + 1u;
        seenEnd = base + 32;
        if (__all_sync(FULL, T.x < 1e-4f && T.y < 1e-4f)) break;
        __syncwarp();  // every lane is done with buffer b: the next chunk but one may overwrite it
        bits = nextBits;
        b ^= 1;
      }
      cp_async_wait<0>();
      __syncwarp();
      if (cntA == 0u) cntA = e - s;
      if (cntB == 0u) cntB = e - s;
    }
    // An infinite colour (a model's SH coefficients may hold one) made the sums
    // of the pixels that do not composite its splat 0 * infinity, a NaN.  Colours
    // are never negative or NaN, so nothing else makes one: then the block's
    // colours are summed again, each pixel only over what it composites.
    const float2 cs = __fadd2_rn(__fadd2_rn(C0, C1), C2);
    if (__any_sync(FULL, isnan(cs.x + cs.y))) {
      C0 = C1 = C2 = bc2(0.0f);
      float2 U = make_float2(inA ? 1.0f : 0.0f, inB ? 1.0f : 0.0f);
      for (uint32_t base = s; base < min(seenEnd, e); base += 32) {
        const uint32_t n = (uint32_t)__popc(stage(base + lane < e ? a.ids[base + lane] : 0u, base + lane < e, 0));
        cp_async_wait<0>();
        __syncwarp();
#pragma unroll 1
        for (uint32_t k = 0; k < n; ++k) {
          const RenderRec& r = s_rec[wid][0][k].rec;
          float2 Bdy;
          const float2 ee = pairExponent2(r.r0, r.r1.x, px - r.r0.x, __fadd2_rn(py, bc2(-r.r0.y)), Bdy);
          const float2 G = gexp2(make_float2(-ee.x, -ee.y));
          const float2 araw = __fmul2_rn(bc2(r.r1.y), G);
          if (U.x >= 1e-4f && ee.x <= E_CUT && araw.x >= A_MIN) {
            const float alpha = fminf(0.99f, araw.x), ta = U.x * alpha;
            C0.x = __fmaf_rn(ta, r.r1.z, C0.x);
            C1.x = __fmaf_rn(ta, r.r1.w, C1.x);
            C2.x = __fmaf_rn(ta, r.r2.x, C2.x);
            U.x = U.x * (1.0f - alpha);
          }
          if (U.y >= 1e-4f && ee.y <= E_CUT && araw.y >= A_MIN) {
            const float alpha = fminf(0.99f, araw.y), ta = U.y * alpha;
            C0.y = __fmaf_rn(ta, r.r1.z, C0.y);
            C1.y = __fmaf_rn(ta, r.r1.w, C1.y);
            C2.y = __fmaf_rn(ta, r.r2.x, C2.y);
            U.y = U.y * (1.0f - alpha);
          }
        }
        __syncwarp();
      }
    }
    C0 = __fadd2_rn(C0, __fmul2_rn(T, bc2(c.bg[0])));
    C1 = __fadd2_rn(C1, __fmul2_rn(T, bc2(c.bg[1])));
    C2 = __fadd2_rn(C2, __fmul2_rn(T, bc2(c.bg[2])));
    {
      const size_t pixA = (size_t)c.pixBase + (size_t)ya * c.W + x;
      const size_t pixB = pixA + (size_t)4 * c.W;
      if (inA) {
        a.outImg[pixA] = make_float4(C0.x, C1.x, C2.x, 1.0f - T.x);
        a.finalT[pixA] = T.x;
        a.endIdx[pixA] = cntA;
      }
      if (inB) {
        a.outImg[pixB] = make_float4(C0.y, C1.y, C2.y, 1.0f - T.y);
        a.finalT[pixB] = T.y;
        a.endIdx[pixB] = cntB;
      }
    }
    if (!BWD) continue;

    // ---- loss (shaders.js:589-618), per pixel ----
    float2 g16_0 = bc2(0.0f), g16_1 = bc2(0.0f), g16_2 = bc2(0.0f);
    bool okA = false, okB = false;  // pixels with a valid target
    {
      uint32_t st0 = 0, st1 = 0, st2 = 0, cg6 = 0, cg7 = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool in = h ? inB : inA;
        if (!in) continue;
        const int yy = h ? yb : ya;
        const uint32_t pi = (uint32_t)(yy * c.W + x);
        const uint32_t packed = a.targets[(size_t)c.offset + pi];
        if ((packed >> 24) == 0u) continue;
        const float Cx = h ? C0.y : C0.x, Cy = h ? C1.y : C1.x, Cz = h ? C2.y : C2.x;
        const float t0 = (float)(packed & 0xFFu) / 255.0f;
        const float t1 = (float)((packed >> 8) & 0xFFu) / 255.0f;
        const float t2 = (float)((packed >> 16) & 0xFFu) / 255.0f;
        st2 += 1u;
        const float gain = c.gain;
        const float er0 = (gain * Cx + c.bias) - t0;
        const float er1 = (gain * Cy + c.bias) - t1;
        const float er2 = (gain * Cz + c.bias) - t2;
        st0 += u32sat((er0 * er0 + er1 * er1 + er2 * er2) * 16.0f + dither(pi));
        const float D2 = 9.0000000000000003e-04f;  // f32(0.03 * 0.03), a WGSL const-expression
        const float rt0 = sqrtf(er0 * er0 + D2), rt1 = sqrtf(er1 * er1 + D2), rt2 = sqrtf(er2 * er2 + D2);
        const float eg0 = er0 / rt0, eg1 = er1 / rt1, eg2 = er2 / rt2;
        const float q0 = gain * eg0, q1 = gain * eg1, q2 = gain * eg2;
        const float lossv = (rt0 + rt1 + rt2) - 8.9999999999999997e-02f;  // f32(3 * 0.03)
        st1 += u32sat(lossv * 32768.0f);
        cg6 += (uint32_t)fixq((eg0 * Cx + eg1 * Cy + eg2 * Cz) * gain, FIXCAM);
        cg7 += (uint32_t)fixq(eg0 + eg1 + eg2, FIXCAM);
        if (h) {
          g16_0.y = q0 * FIXED; g16_1.y = q1 * FIXED; g16_2.y = q2 * FIXED;
          okB = true;
        } else {
          g16_0.x = q0 * FIXED; g16_1.x = q1 * FIXED; g16_2.x = q2 * FIXED;
          okA = true;
        }
      }
      // wrapping sums of the per-pixel stats, kept per block until the kernel's end
      const uint32_t r0 = __reduce_add_sync(FULL, st0);
      const uint32_t r1 = __reduce_add_sync(FULL, st1);
      const uint32_t r2 = __reduce_add_sync(FULL, st2);
      const uint32_t r3 = __reduce_add_sync(FULL, cg6);
      const uint32_t r4 = __reduce_add_sync(FULL, cg7);
      if (lane == 0) {
        atomicAdd(&s_stat[0], r0);
        atomicAdd(&s_stat[1], r1);
        atomicAdd(&s_stat[2], r2);
        atomicAdd(&s_cam[v][0], (int32_t)r3);
        atomicAdd(&s_cam[v][1], (int32_t)r4);
      }
    }
    if (!__any_sync(FULL, okA || okB)) continue;
    // Clamping (see fix_scaled) changes nothing while every value stays within
    // +-1e9: slots 0-6 within 80 |galpha * 2^14|, slots 7-9 within |gC * 2^14|.
    // galpha is at most the pixel's sum of |gC| times the largest colour of
    // the splats from the back to here (a blend of them in front of or behind
    // the splat, times a transmittance of at most 1); 2.5 leaves room for the
    // rounding.  Both maxima are taken on the float's bits, so infinities and
    // NaN count as larger than every number.
    const float gMax = __uint_as_float(__reduce_max_sync(
        FULL, max(__float_as_uint(fabsf(g16_0.x) + fabsf(g16_1.x) + fabsf(g16_2.x)),
                  __float_as_uint(fabsf(g16_0.y) + fabsf(g16_1.y) + fabsf(g16_2.y)))));
    uint32_t cMax = __float_as_uint(fmaxf(fabsf(c.bg[0]), fmaxf(fabsf(c.bg[1]), fabsf(c.bg[2]))));
    bool fast = false;
    auto widen = [&](const StagedRec* sr, uint32_t n) {  // the chunk's colours join cMax
      uint32_t m = 0;
      if ((uint32_t)lane < n)
        m = max(__float_as_uint(fabsf(sr[lane].rec.r1.z)),
                max(__float_as_uint(fabsf(sr[lane].rec.r1.w)), __float_as_uint(fabsf(sr[lane].rec.r2.x))));
      cMax = max(cMax, __reduce_max_sync(FULL, m));
      fast = gMax < 9.0e8f && gMax * 2.5f * __uint_as_float(cMax) < 1.0e7f;
    };

    // ---- backward (shaders.js:632-700) ----
    float2 S0 = __fmul2_rn(bc2(c.bg[0]), T), S1 = __fmul2_rn(bc2(c.bg[1]), T), S2 = __fmul2_rn(bc2(c.bg[2]), T);
    float2 Ta = T;
    int32_t* gradP = a.gradP + (size_t)v * a.n * GP_STRIDE + lane;
    asm volatile("mov.u64 %0, %1;" : "=l"(gradP) : "l"(gradP));  // opaque: not formed anew per entry
    uint32_t row = smem_addr(s_stage[wid][0]);  // the staging rows in use: this one and the one 64 bytes on
    uint32_t slotOff;                            // this lane's word of a row
    asm volatile("mov.u32 %0, %1;" : "=r"(slotOff) : "r"((lane < 10 ? lane : 10) * 4));
    // One composited entry at shared address sr, G the pixels' exponentials (0
    // where a pixel does not composite it).  FAST: every product is finite and
    // within +-1e9, so a pixel with G = 0 or without a target (gC = 0)
    // contributes zeros, and keeps S, without being masked.  Advances Ta and S and returns
    // the lane's ten integer values.
    auto backward = [&](uint32_t sr, float2 G, auto FAST, int32_t q[10]) {
      const float4 r0 = lds4(sr);
      const float4 r1 = lds4(sr + 16);
      const float4 r2 = lds4(sr + 32);
      const float dx = px - r0.x, dx2 = dx + dx;
      const float2 dy = __fadd2_rn(py, bc2(-r0.y)), dy2 = __fadd2_rn(dy, dy);
      const float2 Bdy = __fmul2_rn(bc2(r0.w), dy);
      const float2 araw = __fmul2_rn(bc2(r1.y), G);
      const float2 alpha = make_float2(fminf(0.99f, araw.x), fminf(0.99f, araw.y));
      const float2 inv = rcp_unit2(__fadd2_rn(bc2(1.0f), make_float2(-alpha.x, -alpha.y)));
      // a pixel that does not composite has alpha 0: inv is 1, and Ta and S stay exactly as they are
      const float2 Tb = __fmul2_rn(Ta, inv);
      const float2 aT = __fmul2_rn(alpha, Tb);
      const float2 g0 = __ffma2_rn(bc2(r1.z), Tb, __fmul2_rn(make_float2(-S0.x, -S0.y), inv));
      const float2 g1 = __ffma2_rn(bc2(r1.w), Tb, __fmul2_rn(make_float2(-S1.x, -S1.y), inv));
      const float2 g2 = __ffma2_rn(bc2(r2.x), Tb, __fmul2_rn(make_float2(-S2.x, -S2.y), inv));
      // galpha * 2^14, accumulated from gC * 2^14
      const float2 gal16r = __ffma2_rn(g16_2, g2, __ffma2_rn(g16_1, g1, __fmul2_rn(g16_0, g0)));
      const bool useA = decltype(FAST)::value || (okA && G.x > 0.0f), useB = decltype(FAST)::value || (okB && G.y > 0.0f);
      const float2 gal16 = make_float2(useA && !(araw.x > 0.99f) ? gal16r.x : 0.0f,
                                       useB && !(araw.y > 0.99f) ? gal16r.y : 0.0f);
      const float2 ga16 = __fmul2_rn(gal16, araw);
      const float2 gq16 = __fmul2_rn(ga16, bc2(r2.z));
      const float2 gqx16 = __fmul2_rn(gq16, bc2(dx));
      // the conic's halves times doubled offsets: doubling commutes with rounding
      float2 xs[10];
      xs[0] = __fmul2_rn(ga16, __ffma2_rn(bc2(r0.z), bc2(dx2), Bdy));
      xs[1] = __fmul2_rn(ga16, __ffma2_rn(bc2(r0.w), bc2(dx), __fmul2_rn(bc2(r1.x), dy2)));
      xs[2] = __fmul2_rn(gqx16, bc2(dx));
      xs[3] = __fmul2_rn(gqx16, dy2);
      xs[4] = __fmul2_rn(__fmul2_rn(gq16, dy), dy);
      xs[5] = __fmul2_rn(__fmul2_rn(gal16, bc2(r2.y)), G);
      xs[6] = __fmul2_rn(ga16, bc2(r2.w));
      xs[7] = __fmul2_rn(g16_0, aT);
      xs[8] = __fmul2_rn(g16_1, aT);
      xs[9] = __fmul2_rn(g16_2, aT);
      if (!decltype(FAST)::value &&
          !__all_sync(FULL, fabsf(gal16.x) < 1.0e7f && fabsf(gal16.y) < 1.0e7f && gMax < 9.0e8f)) {
#pragma unroll
        for (int k = 0; k < 10; ++k)
          xs[k] = make_float2(useA ? fminf(fmaxf(xs[k].x, -1.0e9f), 1.0e9f) : 0.0f,
                              useB ? fminf(fmaxf(xs[k].y, -1.0e9f), 1.0e9f) : 0.0f);
      }
      const bool setA = decltype(FAST)::value || G.x > 0.0f, setB = decltype(FAST)::value || G.y > 0.0f;
      const float2 n0 = __ffma2_rn(bc2(r1.z), aT, S0);
      const float2 n1 = __ffma2_rn(bc2(r1.w), aT, S1);
      const float2 n2 = __ffma2_rn(bc2(r2.x), aT, S2);
      S0 = make_float2(setA ? n0.x : S0.x, setB ? n0.y : S0.y);
      S1 = make_float2(setA ? n1.x : S1.x, setB ? n1.y : S1.y);
      S2 = make_float2(setA ? n2.x : S2.x, setB ? n2.y : S2.y);
      Ta = Tb;
#pragma unroll
      for (int k = 0; k < 10; ++k) q[k] = __float2int_rz(xs[k].x) + __float2int_rz(xs[k].y);
    };
    // The ten sums over the warp (every lane has them) go through shared memory,
    // and lanes 0-9 add one each to the splat's slots.
    auto put = [&](uint32_t at, const int32_t q[10]) {
      sts4(at, __reduce_add_sync(FULL, q[0]), __reduce_add_sync(FULL, q[1]), __reduce_add_sync(FULL, q[2]),
           __reduce_add_sync(FULL, q[3]));
      sts4(at + 16, __reduce_add_sync(FULL, q[4]), __reduce_add_sync(FULL, q[5]), __reduce_add_sync(FULL, q[6]),
           __reduce_add_sync(FULL, q[7]));
      sts2(at + 32, __reduce_add_sync(FULL, q[8]), __reduce_add_sync(FULL, q[9]));
    };
    auto add = [&](uint32_t at, uint32_t sr) {  // lanes from 10 on read word 10, which stays 0
      red_nz(gradP + (size_t)lds1(sr + 48) * GP_STRIDE, (int32_t)lds1(at + slotOff));
    };
    // one barrier per entry (or pair): the rows alternate with those 128 bytes away
    auto one = [&](uint32_t sr, float2 G, auto FAST) {
      int32_t q[10];
      backward(sr, G, FAST, q);
      put(row, q);
      __syncwarp();
      add(row, sr);
      row ^= 128u;
    };
    auto two = [&](uint32_t sr0, float2 A, uint32_t sr1, float2 B, auto FAST) {
      int32_t q0[10], q1[10];
      backward(sr0, A, FAST, q0);
      backward(sr1, B, FAST, q1);
      put(row, q0);
      put(row + 64u, q1);
      __syncwarp();
      add(row, sr0);
      add(row + 64u, sr1);
      row ^= 128u;
    };
    // List entries past the cache, chunk by chunk from the back, the records one
    // chunk ahead.  The exponentials of up to REDO entries are computed again --
    // independent of one another, so two at a time -- and left in shared memory;
    // then the entries that a pixel composites are taken as the cached ones are.
    if (uncached < e) {
      const uint32_t endA = inA ? cntA : 0u, endB = inB ? cntB : 0u;
      auto load = [&](uint32_t base) { return base + lane < e ? a.ids[base + lane] : 0u; };
      float2* const redo = s_redo[wid][0] + lane;
      int b = 0;
      uint32_t base = seenEnd - 32;  // both a whole number of chunks after s
      uint32_t bits = stage(load(base), base + lane < e, 0);
      uint32_t nextVal = base > uncached ? load(base - 32) : 0u;
      for (;;) {
        uint32_t nextBits = 0;
        if (base > uncached) {
          nextBits = stage(nextVal, true, b ^ 1);
          nextVal = base - 32 > uncached ? load(base - 64) : 0u;
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncwarp();
        const StagedRec* sr = s_rec[wid][b];
        const uint32_t n = (uint32_t)__popc(bits);
        widen(sr, n);
        for (uint32_t hi = n; hi > 0;) {
          const uint32_t lo = hi > REDO ? hi - REDO : 0u;
          uint32_t hit = 0;
#pragma unroll 2
          for (uint32_t k = lo; k < hi; ++k) {
            const float4 r0 = sr[k].rec.r0;
            const float2 wc = *reinterpret_cast<const float2*>(&sr[k].rec.r1);
            const uint32_t j = base - s + sr[k].raw;
            float2 Bdy;
            const float2 ee = pairExponent2(r0, wc.x, px - r0.x, __fadd2_rn(py, bc2(-r0.y)), Bdy);
            const float2 G = gexp2(make_float2(-ee.x, -ee.y));
            const float2 araw = __fmul2_rn(bc2(wc.y), G);
            const bool c2a = j < endA && ee.x <= E_CUT && araw.x >= A_MIN;
            const bool c2b = j < endB && ee.y <= E_CUT && araw.y >= A_MIN;
            redo[(k - lo) * 32] = make_float2(c2a ? G.x : 0.0f, c2b ? G.y : 0.0f);
            hit |= (__any_sync(FULL, c2a || c2b) ? 1u : 0u) << (k - lo);
          }
          constexpr uint32_t STEP = (uint32_t)sizeof(StagedRec);
          const uint32_t at = smem_addr(sr + lo);
          while (hit) {  // the last entry first
            const uint32_t i0 = 31u - (uint32_t)__clz((int)hit);
            hit ^= 1u << i0;
            if (fast && hit) {
              const uint32_t i1 = 31u - (uint32_t)__clz((int)hit);
              hit ^= 1u << i1;
              two(at + i0 * STEP, redo[i0 * 32], at + i1 * STEP, redo[i1 * 32], std::true_type{});
            } else {
              one(at + i0 * STEP, redo[i0 * 32], std::false_type{});
            }
          }
          hi = lo;
        }
        __syncwarp();  // every lane is done with buffer b
        if (base == uncached) break;
        base -= 32;
        bits = nextBits;
        b ^= 1;
      }
    }
    // cached entries, back to front, 32 records at a time; the exponentials
    // load two entries ahead (they mostly come from DRAM)
    const uint32_t vis = (uint32_t)((gp - gFirst) >> 5);
    if (vis) {
      const float2* gl = gp - 32;
      float2 G0 = __ldcg(gl), G1 = __ldcg(gl - 32);  // this entry's exponentials and the next one's
      auto stage_cached = [&](uint32_t hi, int b) {  // entries [max(hi - 32, 0), hi): lane l holds entry hi - 1 - l
        if ((uint32_t)lane < hi) {
          const uint32_t id = __ldcg(cacheId + (hi - 1 - lane));
          s_rec[wid][b][lane].id = id;
          cp_async_rec(&s_rec[wid][b][lane].rec, recs + id);
        }
        cp_async_commit();
      };
      int b = 0;
      __syncwarp();
      stage_cached(vis, 0);
      for (uint32_t hi = vis; hi > 0;) {
        const uint32_t n = hi < 32u ? hi : 32u;
        if (hi > 32u) {
          stage_cached(hi - 32u, b ^ 1);
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncwarp();
        const StagedRec* sr = s_rec[wid][b];
        widen(sr, n);
        auto chunk = [&](auto FAST) {
          constexpr uint32_t STEP = (uint32_t)sizeof(StagedRec);
          uint32_t at = smem_addr(sr);
          const uint32_t end = at + n * STEP;
          for (; end - at >= 2u * STEP; at += 2u * STEP) {
            const float2 A = G0, B = G1;
            G0 = __ldcg(gl - 64);
            G1 = __ldcg(gl - 96);
            gl -= 64;
            two(at, A, at + STEP, B, FAST);
          }
          for (; at != end; at += STEP) {
            const float2 G = G0;
            G0 = G1;
            G1 = __ldcg(gl - 64);
            gl -= 32;
            one(at, G, FAST);
          }
        };
        if (fast) chunk(std::true_type{});
        else chunk(std::false_type{});
        __syncwarp();
        hi -= n;
        b ^= 1;
      }
    }
  }
  if (BWD) {
    __syncthreads();
    if (threadIdx.x < 3 && s_stat[threadIdx.x]) atomicAdd(&a.stats[threadIdx.x], s_stat[threadIdx.x]);
    if (threadIdx.x < 2 * a.V) {
      const int v = threadIdx.x >> 1, k = threadIdx.x & 1;
      if (s_cam[v][k]) atomicAdd(&a.gradCam[a.cams[v].camIdx * 8u + 6u + (uint32_t)k], s_cam[v][k]);
    }
  }
}

template <int TILE, bool MASKED>
static const void* warp_kernel(bool train) {
  return train ? (const void*)k_raster_warp<TILE, MASKED, true> : (const void*)k_raster_warp<TILE, MASKED, false>;
}
static const void* warp_kernel(int tile, bool masked, bool train) {
  if (tile == 8) return warp_kernel<8, false>(train);
  if (tile == 32) return warp_kernel<32, false>(train);
  return masked ? warp_kernel<16, true>(train) : warp_kernel<16, false>(train);
}

template <int TILE>
static void launch_stored(const RasterArgs& a, int batchDepth, unsigned grid, cudaStream_t s) {
  switch (batchDepth) {
    case 64: k_raster_stored<TILE, 64><<<grid, TILE * TILE, 0, s>>>(a); break;
    case 128: k_raster_stored<TILE, 128><<<grid, TILE * TILE, 0, s>>>(a); break;
    default: k_raster_stored<TILE, 256><<<grid, TILE * TILE, 0, s>>>(a); break;
  }
}

void launch_raster_stored(const RasterArgs& a, int tile, int batchDepth, unsigned grid, cudaStream_t s) {
  if (grid == 0) return;
  if (tile == 8) launch_stored<8>(a, batchDepth, grid, s);
  else if (tile == 32) launch_stored<32>(a, batchDepth, grid, s);
  else launch_stored<16>(a, batchDepth, grid, s);
}

void launch_raster(const RasterArgs& a, bool train, int tile, unsigned grid, cudaStream_t s) {
  if (grid == 0) return;
  RasterArgs copy = a;
  void* args[] = {&copy};
  cudaLaunchKernel(warp_kernel(tile, a.idMask != 0xFFFFFFFFu, train), dim3(grid), dim3(RW_WARPS * 32), args, 0, s);
}

int raster_blocks_per_sm(int tile, bool train) {
  int a = 0, b = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, warp_kernel(tile, false, train), RW_WARPS * 32, 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, warp_kernel(tile, true, train), RW_WARPS * 32, 0);
  const int perSm = std::min(a, b);
  return perSm < 1 ? 1 : perSm;
}

// Blocks of the persistent raster over `items` 8x8 blocks.  The longest tiles
// are taken first, and with every warp slot filled they share an SM with 19
// others and finish last, so when there are only a few items per slot fewer
// blocks are launched: about 5.3 items a warp, at least 2 blocks per SM.
// Train passes at 5 / 4 / 3 / 2 blocks per SM, us a pass of the same steps:
// 3780 items 6987 / 6679 / 6322 / 5970; 10032 items 11862 / 11635 / 11796 /
// 12813; 15504 items 7239 / 7332 / 8071 / 9583; 32640 items 45740 / 48037 /
// 52569 / 63085.
unsigned raster_grid(uint32_t items, int sms, int perSm) {
  const unsigned all = (items + RW_WARPS - 1) / RW_WARPS;
  const double k = std::ceil((double)items / (5.3 * RW_WARPS * sms));
  const unsigned blocks = (unsigned)(std::min((double)perSm, std::max(2.0, k)) * sms);
  return all < blocks ? all : blocks;
}

// Work order for the persistent queue: global tiles by descending entry
// count (bucketed by log2), so the heaviest tiles start first.  The kernels
// that write the ranges count the buckets; here every tile is placed at its
// bucket's start (the exclusive scan of the 33 sizes, done by each warp) plus
// its bucket's cursor.  The order inside a bucket follows the cursor atomics;
// no result depends on it (tiles write disjoint pixels and integer gradient
// sums), only the schedule does.  One launch of about 2 us; counting, scanning
// (on one thread) and placing in three launches took 15 us whatever the size.
__global__ void __launch_bounds__(256) k_work_place(const uint2* ranges, uint32_t totalTiles, const uint32_t* counts,
                                                    uint32_t* cursors, uint32_t* order) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = t < totalTiles;
  const uint32_t c = counts[lane];
  uint32_t start = c;  // inclusive, then exclusive, scan of buckets 0..31; bucket 32 starts after them
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, start, o);
    if ((int)lane >= o) start += y;
  }
  const uint32_t all = __shfl_sync(0xFFFFFFFFu, start, 31);
  start -= c;
  const uint32_t b = valid ? tile_bucket(ranges[t]) : 64u;
  const uint32_t at = __shfl_sync(0xFFFFFFFFu, start, b & 31u);
  const uint32_t peers = __match_any_sync(0xFFFFFFFFu, b);
  const uint32_t lead = (uint32_t)(__ffs(peers) - 1);
  uint32_t base = 0;
  if (valid && lane == lead) base = (b < 32u ? at : all) + atomicAdd(&cursors[b], (uint32_t)__popc(peers));
  base = __shfl_sync(0xFFFFFFFFu, base, lead);
  if (valid) order[base + (uint32_t)__popc(peers & ((1u << lane) - 1u))] = t;
}

// counts: 33 bucket sizes (tile_bucket) of the ranges; cursors: 33 words, zero
void launch_work_place(const uint2* ranges, uint32_t totalTiles, const uint32_t* counts, uint32_t* cursors,
                       uint32_t* order, cudaStream_t s) {
  if (totalTiles) k_work_place<<<(totalTiles + 255) / 256, 256, 0, s>>>(ranges, totalTiles, counts, cursors, order);
}

}  // namespace gs
