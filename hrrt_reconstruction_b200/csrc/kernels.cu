// kernels.cu -- sm_100a kernels of the hrrt_osem3d OSEM hot path.
//
// Compiled with -fmad=false: the reference (x86-64 SSE2 build) never fuses a
// multiply with an add, and every expression below keeps the reference's
// association, so the forward projector, the rotate-back and the update are
// bit-identical to the reference on the same inputs.
#include "kernels.cuh"

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <type_traits>

namespace hrrt {

namespace {

__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float4 operator+(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ float4 operator*(float4 a, float s) {
  return make_float4(a.x * s, a.y * s, a.z * s, a.w * s);
}

// ---- storage-type helpers for the sinogram inputs ----
struct P4 { float v[4]; };
__device__ __forceinline__ P4 load_p4(const __half *p, size_t i) {
  const uint2 u = reinterpret_cast<const uint2 *>(p)[i];
  const __half2 a = *reinterpret_cast<const __half2 *>(&u.x);
  const __half2 b = *reinterpret_cast<const __half2 *>(&u.y);
  return P4{{__low2float(a), __high2float(a), __low2float(b), __high2float(b)}};
}
__device__ __forceinline__ P4 load_p4(const float *p, size_t i) {
  const float4 f = reinterpret_cast<const float4 *>(p)[i];
  return P4{{f.x, f.y, f.z, f.w}};
}
__device__ __forceinline__ P4 load_p4(const __nv_bfloat16 *p, size_t i) {
  const uint2 u = reinterpret_cast<const uint2 *>(p)[i];
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(&u.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(&u.y);
  return P4{{__low2float(a), __high2float(a), __low2float(b), __high2float(b)}};
}
// lanes 0,1 or 2,3 of a quad: pair i of the array
__device__ __forceinline__ float2 load_p2(const int16_t *p, size_t i) {
  const short2 s = reinterpret_cast<const short2 *>(p)[i];
  return make_float2((float)s.x, (float)s.y);
}
__device__ __forceinline__ float2 load_p2(const float *p, size_t i) { return reinterpret_cast<const float2 *>(p)[i]; }
__device__ __forceinline__ float2 load_p2(const __half *p, size_t i) {
  return __half22float2(reinterpret_cast<const __half2 *>(p)[i]);
}
__device__ __forceinline__ float2 load_p2(const __nv_bfloat16 *p, size_t i) {
  return __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 *>(p)[i]);
}
__device__ __forceinline__ void store_p4(int16_t *p, size_t i, const float *v) {
  reinterpret_cast<short4 *>(p)[i] = make_short4((short)v[0], (short)v[1], (short)v[2], (short)v[3]);
}
__device__ __forceinline__ void store_p4(__half *p, size_t i, const float *v) {
  __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t *>(&a);
  u.y = *reinterpret_cast<uint32_t *>(&b);
  reinterpret_cast<uint2 *>(p)[i] = u;
}
__device__ __forceinline__ void store_p4(float *p, size_t i, const float *v) {
  reinterpret_cast<float4 *>(p)[i] = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store_p4(__nv_bfloat16 *p, size_t i, const float *v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t *>(&a);
  u.y = *reinterpret_cast<uint32_t *>(&b);
  reinterpret_cast<uint2 *>(p)[i] = u;
}



// ---- packed pairs of IEEE single-precision values (sm_100 f32x2) ----
// Each op is element-wise round-to-nearest, exactly the scalar add/sub/mul of
// the reference, two values per instruction.  A quad value (4 lanes) is two
// pairs: lanes (0,1) and (2,3).
struct Q2 {
  uint64_t lo, hi;
};
__device__ __forceinline__ uint64_t pk(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 upk(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0,%1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a + p where p is a packed product.  The code generator contracts a packed
// multiply that feeds a packed add into a fused multiply-add (which rounds once
// instead of twice), even with -fmad=false and explicit .rn, and folds a
// multiply by a literal 1 away; a packed fused multiply-add of p by a run-time
// (1, 1) and a cannot absorb p's multiply and rounds p + a once, as the
// reference's add does (measured bit-identical on B200; two scalar adds, the
// alternative, cost one more instruction per pair).
__device__ __forceinline__ uint64_t addp(uint64_t a, uint64_t p, uint64_t one) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(p), "l"(one), "l"(a));
  return r;
}
__device__ __forceinline__ Q2 ldq(const float4 *p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
  return Q2{v.x, v.y};
}
__device__ __forceinline__ Q2 qadd(Q2 a, Q2 b) { return Q2{add2(a.lo, b.lo), add2(a.hi, b.hi)}; }
// packed a * b + c (one rounding), where no reference rounding order is to
// be kept: the back projector (held to the reference within 2e-6, its sums
// being incremental there and direct here) and the exact adjoint (held to
// the FP64 oracle)
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ Q2 qfma(Q2 a, uint64_t b, Q2 c) { return Q2{fma2(a.lo, b, c.lo), fma2(a.hi, b, c.hi)}; }

// ---- bulk copies + mbarriers (sm_90+ async proxy) ----
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// whole 16-byte words of [p, p + bytes) brought into L2
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
  const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
  const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + bytes) & ~(uintptr_t)15;
  if (e > a)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(e - a)) : "memory");
}
// bounded wait on an mbarrier phase; on timeout records the error and returns false
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err) {
  const uint32_t a = smem_u32(bar);
  for (int i = 0; i < (1 << 22); i++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  if (err) atomicExch(err, 1);
  return false;
}

// Rotated-grid sample point (sbrt:1866-1871): position of rotated-frame voxel
// (a,b) in the image, as flat column index of its (ix,iy) corner and the four
// bilinear weights.  base < 0: outside (the reference zeroes that sample).
struct SamplePt {
  int base;
  float c0, c1, c2, c3;
};
__device__ __forceinline__ SamplePt sample_point(int a, int b, int c, int N, int zp, float cosv, float sinv) {
  SamplePt s;
  const float fa = (float)(a - c), fb = (float)(b - c), fc = (float)c;
  const float xx0 = fa * cosv - fb * sinv + fc;
  const float yy0 = fa * sinv + fb * cosv + fc;
  const float lim = (float)(N - 2);
  // the reference tests xx0 against the upper limit twice and never yy0
  if (xx0 < 0 || xx0 > lim || yy0 < 0 || xx0 > lim) {
    s.base = -1;
    s.c0 = s.c1 = s.c2 = s.c3 = 0.f;
    return s;
  }
  const int ix = (int)xx0, iy = (int)yy0;
  const float x1 = xx0 - ix, y1 = yy0 - iy;
  s.c0 = (1 - x1) * (1 - y1);
  s.c1 = x1 * (1 - y1);
  s.c2 = y1 * (1 - x1);
  s.c3 = y1 * x1;
  // contiguous [x][y][zp] addressing, as the reference's matrix3dm128 image
  if ((ix + 1) * N + iy + 1 >= N * N) {
    s.base = -1;
    return s;
  }
  s.base = (ix * N + iy) * zp;
  return s;
}
// ============================================================================
// Forward projection (+ fused OP ratio), restating forward_proj3d_view1_thread
// (sbrt:1728-1978) for one (view pair, quad x) in two kernels:
//   fp_sample_kernel : the eight symmetric rotated-grid columns at every row y
//                      (pam: lanes (x,y),(N-x,y),(N-y,x),(N-y,N-x); pam2:
//                      (x,N-y),(N-x,N-y),(y,x),(y,N-x)), the quad's lanes
//                      interleaved; and the centre column (pam of y = c);
//   fp_kernel        : every thread accumulates its own (segment, plane-run)
//                      outputs, row by row in the reference's order.
// Samples of a quad, entries of 4 lanes: [zp] centre column, then per row
// y = cyl0[x] .. c-1 [2 halves][zp], at g.samp_off[x] of its pair slot.
// fp_kernel is bound by shared memory (L1 92 % busy at span 3: 2 x 8 bytes for
// 6 packed operations), fp_sample_kernel by L1 (76 % busy) and the latency of
// its L2 reads.
// Measured on B200, us a subset: span 3 1892 -> 1037 + 241, span 9 860 -> 475
// + 241, a 24-ring scanner 53 -> 26 + 6; before, one kernel sampled with four
// warps (bulk tensor copies of the corner columns) beside 28 warps of 9-plane
// 4-lane tasks, whose accumulators and end-plane entries spilled.
// Measured at span 3 and not used: sampling warps in fp_kernel with plain
// loads (2151: too few in flight), all warps sampling 8 rows at a time (2497:
// spills), runs of 17 planes without the order of build_fp_tasks (bank
// conflicts 53 M -> 36 M, 1092 -> 1053).
// ============================================================================
// A warp takes one quad and half and `steps` rows, every other one; a CTA's
// four warps are 2 quads x 2 rows at a time, whose points lie close together
// in each of the four image regions they map to and share corner columns in
// L1.  16 loads of 16 bytes in flight per lane (112 registers) and 16 rows a
// warp measured 241 us for 9 span-3 pairs; 8-byte loads with twice the warps
// 266, 4-byte loads 306, 4 x 4 tiles 270.
constexpr int kSampleTile = 2;
__global__ void __launch_bounds__(kSampleTile * kSampleTile * 32, 4)
    fp_sample_kernel(DevGeom g, const float *__restrict__ image, const int *__restrict__ pair_views, int view0,
                     int npairs, float4 *__restrict__ samples, FrameStrides fr, int steps) {
  const int h = blockIdx.z & 1, frame = (blockIdx.z >> 1) / npairs, slot = (blockIdx.z >> 1) - frame * npairs;
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31, N = g.nx, c = g.c, zp = g.zp;
  const int x = blockIdx.x * kSampleTile + 1 + wid % kSampleTile;
  if (x > c) return;
  const int ystart = g.cyl0[x];
  if (ystart == g.cyl1[x]) return;
  const int view = pair_views ? __ldg(pair_views + slot) : view0 + slot;
  const float cosv = g.cos_psi[view], sinv = g.sin_psi[view];
  const uint64_t one = g.unit2;
  image += (size_t)(fr.map ? __ldg(fr.map + frame) : frame) * fr.image;
  float4 *quad = samples + (size_t)frame * (fr.samples / 4) + (size_t)slot * g.samp_pair + g.samp_off[x];
  const char *k1 = reinterpret_cast<const char *>(image), *k2 = k1 + (size_t)N * zp * 4;
  const char *k3 = k1 + (size_t)zp * 4, *k4 = k2 + (size_t)zp * 4;
  auto ld = [](const char *k, uint32_t o) { return __ldg(reinterpret_cast<const ulonglong2 *>(k + o)); };
  const int y1 = blockIdx.y * kSampleTile * steps + wid / kSampleTile;
  for (int y = y1; y < y1 + kSampleTile * steps; y += kSampleTile) {
    // row y = c is the centre column: pam only
    if (y < ystart || y > c || (y == c && h)) continue;
    float4 *dst = quad + (y == c ? 0 : (size_t)(2 * (y - ystart) + 1 + h) * zp);
    SamplePt pt;
    {
      const int l = ln & 3, yy = h ? N - y : y;
      const int a = l == 0 ? x : l == 1 ? N - x : N - yy, b = l < 2 ? yy : l == 2 ? x : N - x;
      pt = sample_point(a, b, c, N, zp, cosv, sinv);
    }
    // Four planes a lane: the corner columns (ix,iy), (ix+1,iy), (ix,iy+1),
    // (ix+1,iy+1) of the four points in 16-byte loads, all in flight together,
    // and the quad's 4 x 4 values in two 32-byte stores.
    uint32_t o[4];
    uint64_t wt[4][4];
    bool in[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const int b = __shfl_sync(0xffffffffu, pt.base, l);
      in[l] = b >= 0;
      o[l] = 4u * (uint32_t)max(b, 0);
      auto dup = [&](float w) {
        const float u = __shfl_sync(0xffffffffu, w, l);
        return pk(u, u);
      };
      wt[l][0] = dup(pt.c0);
      wt[l][1] = dup(pt.c1);
      wt[l][2] = dup(pt.c2);
      wt[l][3] = dup(pt.c3);
    }
    for (int z = 4 * ln; z < zp; z += 128) {
      ulonglong2 c[4][4];
#pragma unroll
      for (int l = 0; l < 4; l++) {
        c[l][0] = ld(k1, o[l] + 4u * z);
        c[l][1] = ld(k2, o[l] + 4u * z);
        c[l][2] = ld(k3, o[l] + 4u * z);
        c[l][3] = ld(k4, o[l] + 4u * z);
      }
      float2 v[4][2];
#pragma unroll
      for (int l = 0; l < 4; l++) {
        // sums in the reference's corner order; outside points sample as zero
        const uint64_t a = add2(addp(mul2(c[l][0].x, wt[l][0]), mul2(c[l][1].x, wt[l][1]), one),
                                addp(mul2(c[l][2].x, wt[l][2]), mul2(c[l][3].x, wt[l][3]), one));
        const uint64_t b = add2(addp(mul2(c[l][0].y, wt[l][0]), mul2(c[l][1].y, wt[l][1]), one),
                                addp(mul2(c[l][2].y, wt[l][2]), mul2(c[l][3].y, wt[l][3]), one));
        v[l][0] = upk(in[l] ? a : 0ull);
        v[l][1] = upk(in[l] ? b : 0ull);
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
        asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + z + 2 * i), "f"(v[0][i].x),
                     "f"(v[1][i].x), "f"(v[2][i].x), "f"(v[3][i].x), "f"(v[0][i].y), "f"(v[1][i].y), "f"(v[2][i].y),
                     "f"(v[3][i].y)
                     : "memory");
    }
  }
}

// a pair of lanes at a byte offset of the dynamic shared memory
__device__ __forceinline__ uint64_t lds2(const float4 *P, int at) {
  return *reinterpret_cast<const uint64_t *>(reinterpret_cast<const char *>(P) + at);
}

// One CTA per (view pair, quad x): one warp brings the rows in by bulk copies,
// a ring of kFpSlots ahead; the others pass through them each at its own pace.
template <int MODE, int PL, typename PT, typename AT>
__global__ void __launch_bounds__(kFpMaxWarps * 32, 1) fp_kernel(DevGeom g, const float4 *__restrict__ samples,
                                                     const QuadWork *__restrict__ work,
                                                     const PT *__restrict__ prompts, const AT *__restrict__ add,
                                                     float4 *__restrict__ out, long long out_pair_stride,
                                                     FrameStrides fr) {
  // shared memory: [kFpSlots][2 halves][ZS] sampled rows, [ZS] centre column,
  // [kFpSlots][groupmax] the rows' middle-plane sampling entries
  extern __shared__ __align__(128) float4 smem[];
  const int ZS = g.zp + kFpZPad, zp = g.zp, G = g.groupmax;
  const int row_bytes = 2 * ZS * 16;
  float4 *cen = smem + 2 * kFpSlots * ZS;
  FpMid *s_mid = reinterpret_cast<FpMid *>(cen + ZS);
  __shared__ __align__(8) uint64_t s_full[kFpSlots], s_empty[kFpSlots], s_cen;

  const int nwork = gridDim.x / fr.n, frame = blockIdx.x / nwork, item = blockIdx.x - frame * nwork;
  const QuadWork w = work[item];
  const int x = w.x, N = g.nx, ystart = g.cyl0[x], nrows = g.c - ystart;
  const int tid = threadIdx.x, ln = tid & 31, ncons = (blockDim.x >> 5) - 1;

  if (tid < kFpSlots) {
    mbar_init(&s_full[tid], 1);
    mbar_init(&s_empty[tid], ncons);
    if (tid == 0) mbar_init(&s_cen, 1);
    fence_mbar_init();
  }
  // zeroes past the end of every sampled row and of the centre column
  for (int i = tid; i < (2 * kFpSlots + 1) * kFpZPad; i += blockDim.x)
    smem[(i / kFpZPad) * ZS + zp + i % kFpZPad] = f4(0.f);
  __syncthreads();

  if (tid >= 32 * ncons) {
    if (ln != 0) return;
    const float4 *src = samples + (size_t)frame * (fr.samples / 4) + (size_t)w.slot * g.samp_pair + g.samp_off[x];
    const uint32_t half = (uint32_t)zp * 16u, mids = (uint32_t)G * 16u;
    mbar_arrive_tx(&s_cen, half);
    bulk_g2s(cen, src, half, &s_cen);
    src += zp;
    if (MODE == 1) {
      // the quad's prompts and additive terms, for the ratio at the end, into L2
      const int fs = fr.map ? __ldg(fr.map + frame) : frame;
      const size_t i0 = (size_t)fs * fr.input + 4 * ((size_t)w.view * g.nquads + x) * g.pplanes;
      prefetch_l2(prompts + i0, 4 * (size_t)g.pplanes * sizeof(PT));
      prefetch_l2(add + i0, 4 * (size_t)g.pplanes * sizeof(AT));
    }
    for (int r = 0; r < nrows; r++, src += 2 * zp) {
      const int sl = r & (kFpSlots - 1);
      if (r >= kFpSlots && !mbar_wait(&s_empty[sl], (uint32_t)((r / kFpSlots - 1) & 1), g.err)) break;
      fence_proxy_async();
      mbar_arrive_tx(&s_full[sl], 2u * half + mids);
      float4 *row = smem + (size_t)sl * 2 * ZS;
      bulk_g2s(row, src, half, &s_full[sl]);
      bulk_g2s(row + ZS, src + zp, half, &s_full[sl]);
      bulk_g2s(s_mid + sl * G, g.fpmid + (size_t)(ystart + r) * G, mids, &s_full[sl]);
    }
    // stay until the last copies have landed, whatever the consumers did
    mbar_wait(&s_cen, 0, nullptr);
    for (int r = max(0, nrows - kFpSlots); r < nrows; r++)
      mbar_wait(&s_full[r & (kFpSlots - 1)], (uint32_t)((r / kFpSlots) & 1), nullptr);
    return;
  }

  // Two threads a task, for lanes 2q and 2q + 1 of the quad; accumulators
  // start at the centre sample of their plane (the reference assigns the
  // centre column before accumulating rows y < c).
  const uint64_t one = g.unit2;
  const FpTask tk = g.fptasks[tid >> 1];
  const int q8 = 8 * (tid & 1);
  const int sg = tk.seg, gg = (sg + 1) / 2 - 1;
  // a warp's tasks are of one kind but for empty ones at its end
  const int kind = __shfl_sync(0xffffffffu, (int)tk.type, 0);
  const int ybot = tk.type > 0 ? g.ybot[sg] : 0, ns = tk.type > 0 ? g.ytop[sg] - ybot + 1 : g.nz;
  // segment 2k takes pam at z and pam2 at z2, segment 2k-1 the converse
  const int oA = q8 + ((sg & 1) ? 16 * ZS : 0), oB = q8 + ((sg & 1) ? 0 : 16 * ZS);
  const FpMid *mid = s_mid + (gg < 0 ? 0 : gg);
  auto centre = [&](int p) { return lds2(cen, 16 * min(ybot + p, ZS - 1) + q8); };
  auto next_row = [&](int r) { return mbar_wait(&s_full[r & (kFpSlots - 1)], (uint32_t)((r / kFpSlots) & 1), g.err); };
  auto row_done = [&](int r) {
    __syncwarp();
    if (ln == 0) mbar_arrive(&s_empty[r & (kFpSlots - 1)]);
  };
  // n planes (plane_of(j), values val(j)) of the task's segment: scale
  // (sbrt:1953-1975), then either store the estimate or the OP ratio
  // (pt_update_est_w3, drv:2474-2520) pre-multiplied by the back projector's
  // segment weight (sbrt:1637-1649); kBatch planes' loads go out together
  auto finish = [&](auto count, int n, auto plane_of, auto val) {
    constexpr int kCount = decltype(count)::value, kBatch = 6;
    const size_t q0 = 2 * ((size_t)x * g.pplanes + g.poff[sg]) + (tid & 1);  // lane pairs
    const int fs = fr.map ? __ldg(fr.map + frame) : frame;
    const size_t i0 = (size_t)fs * (fr.input / 2) + 2 * (size_t)w.view * g.nquads * g.pplanes + q0;
    float2 *o2 = reinterpret_cast<float2 *>(out + (size_t)frame * (fr.ratio / 4) + (size_t)w.slot * out_pair_stride) + q0;
    const float bs = MODE == 1 ? g.bp_scale[sg] : 0.f;
    const float *rescale = g.rescale + (gg < 0 ? 0 : gg * g.nz + ybot);
#pragma unroll
    for (int j0 = 0; j0 < kCount; j0 += kBatch) {
      float sc[kBatch];
      float2 num[kBatch], ad[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        if (j0 + k >= kCount) continue;
        const int p = plane_of(j0 + k < n ? j0 + k : 0);
        sc[k] = (sg == 0) ? g.y_size : rescale[p];
        if (MODE == 1) {
          num[k] = load_p2(prompts, i0 + 2 * p);
          ad[k] = load_p2(add, i0 + 2 * p);
        }
      }
#pragma unroll
      for (int k = 0; k < kBatch; k++) {
        if (j0 + k >= kCount) continue;
        float2 est = upk(mul2(val(j0 + k), pk(sc[k], sc[k])));
        if (MODE == 1) {
          const float d0 = est.x + ad[k].x, d1 = est.y + ad[k].y;
          const float r0 = num[k].x == 0.f ? 0.f : d0 > g.eps3 ? num[k].x / d0 : 1.0f;
          const float r1 = num[k].y == 0.f ? 0.f : d1 > g.eps3 ? num[k].y / d1 : 1.0f;
          est = make_float2(r0 * bs, r1 * bs);
        }
        if (j0 + k < n) o2[2 * plane_of(j0 + k)] = est;
      }
    }
  };
  if (!mbar_wait(&s_cen, 0, g.err)) return;
  if (kind == 2) {
    // end planes: per-plane flookup entries (sbrt:1925-1931, :1948-1952), the
    // next row's in flight under this one's; entry i is plane i (bottom) or
    // ns - 2*zshift + i (top)
    auto plane = [&](int i) { return i >= g.zshift ? ns - 2 * g.zshift + i : i; };
    const int n = tk.type == 2 ? tk.n : 0, FS = G * 2 * g.zshift;
    const int2 *fl = g.fl_zf + (n ? gg * 2 * g.zshift + tk.p0 : 0);
    uint64_t acc[kFpEndPlanes];
    int2 n1[kFpEndPlanes], n2[kFpEndPlanes];
#pragma unroll
    for (int j = 0; j < kFpEndPlanes; j++) {
      acc[j] = centre(plane(tk.p0 + j));
      n1[j] = n2[j] = make_int2(0, 0);
    }
    auto entries = [&](int y) {
#pragma unroll
      for (int j = 0; j < kFpEndPlanes; j++)
        if (j < n) {
          n1[j] = __ldg(fl + y * FS + j);
          n2[j] = __ldg(fl + (N - y) * FS + j);
        }
    };
    if (nrows > 0) entries(ystart);
    for (int r = 0; r < nrows; r++) {
      int2 e1[kFpEndPlanes], e2[kFpEndPlanes];
#pragma unroll
      for (int j = 0; j < kFpEndPlanes; j++) {
        e1[j] = n1[j];
        e2[j] = n2[j];
      }
      if (r + 1 < nrows) entries(ystart + r + 1);
      if (!next_row(r)) return;
      const int sl = r & (kFpSlots - 1), at = sl * row_bytes;
      if (mid[sl * G].z >= 0) {
#pragma unroll
        for (int j = 0; j < kFpEndPlanes; j++) {
          if (j < n) {
            const int pa = at + oA + 16 * e1[j].x, pb = at + oB + 16 * e2[j].x;
            const float f = __int_as_float(e1[j].y), f2 = __int_as_float(e2[j].y);
            const uint64_t ff = pk(f, f), ff2 = pk(f2, f2);
            acc[j] = add2(acc[j], addp(mul2(add2(lds2(smem, pb + 16), lds2(smem, pa)), ff2),
                                       mul2(add2(lds2(smem, pa + 16), lds2(smem, pb)), ff), one));
          }
        }
      }
      row_done(r);
    }
    if (n) finish(std::integral_constant<int, kFpEndPlanes>{}, n, [&](int j) { return plane(tk.p0 + j); },
                  [&](int j) { return acc[j]; });
    return;
  }
  uint64_t acc[PL];
#pragma unroll
  for (int j = 0; j < PL; j++) acc[j] = centre(tk.p0 + j);
  if (kind == 1) {
    // middle planes: z, z2 advance with the plane (sbrt:1933-1947)
    const int o = 16 * (tk.p0 - g.zshift);
    for (int r = 0; r < nrows; r++) {
      if (!next_row(r)) return;
      const int sl = r & (kFpSlots - 1);
      const FpMid m = mid[sl * G];
      if (tk.type == 1 && m.z >= 0) {  // else the group is skipped for this row (sbrt:1923-1924)
        const int at = sl * row_bytes + o, pa = at + oA + 16 * m.z, pb = at + oB + 16 * m.z2;
        const uint64_t f = pk(m.f, m.f), f2 = pk(m.f2, m.f2);
        uint64_t a0 = lds2(smem, pa), b0 = lds2(smem, pb);
#pragma unroll
        for (int j = 0; j < PL; j++) {
          const uint64_t a1 = lds2(smem, pa + 16 * (j + 1)), b1 = lds2(smem, pb + 16 * (j + 1));
          acc[j] = add2(acc[j], addp(mul2(add2(b1, a0), f2), mul2(add2(a1, b0), f), one));
          a0 = a1;
          b0 = b1;
        }
      }
      row_done(r);
    }
  } else {
    // theta = 0 (sbrt:1907-1910)
    for (int r = 0; r < nrows; r++) {
      if (!next_row(r)) return;
      const int at = (r & (kFpSlots - 1)) * row_bytes + 16 * tk.p0 + q8;
#pragma unroll
      for (int j = 0; j < PL; j++)
        acc[j] = add2(acc[j], add2(lds2(smem, at + 16 * j), lds2(smem, at + 16 * ZS + 16 * j)));
      row_done(r);
    }
  }
  if (tk.type < 0) return;
  finish(std::integral_constant<int, PL>{}, tk.n, [&](int j) { return tk.p0 + j; }, [&](int j) { return acc[j]; });
}

// ============================================================================
// Back projection, one CTA (or `split` CTAs) per (view pair, quad x).
// Voxel-driven restatement of back_proj3d_view_n1thread (sbrt:4162-4668): the
// quad's four sinogram lanes sit in shared memory; each thread evaluates, for
// kBpRows rotated-grid rows y and a run of kBpZ planes, the two 4-lane sums the
// reference builds incrementally (sumt1 for voxels (x,y),(N-x,y),(N-y,x),
// (N-y,N-x); sumt2 for (x,N-y),(N-x,N-y),(y,x),(y,N-x)) as direct linear
// interpolations of the zero-padded sinogram at yr = z + d.  Each voxel
// receives two partial sums, one from the ray of view p (its column quad) and
// one from the ray of view p+nviews/2 (its row quad); they go to Bc and Br and
// are added in the rotate-back, which is the reference's assign-then-
// accumulate order.
// What bounds it is instruction issue and the latency that 16 warps an SM leave
// uncovered (issue 55 %, FMA pipe 48 %, L1 45 % busy at span 3): per (row
// group, side of a group) a thread reads 6 shared planes for 16 outputs --
// adjacent rows read the segment less than a plane apart, so four rows share a
// window -- and issues 64 packed FMAs and about as many other instructions.
// One row and 8 planes a thread (9 shared planes for 8 outputs, an address
// each) took 1.384 ms a span-3 subset and 0.509 ms a span-9 one; this 0.990
// and 0.375, to the same bits (one pair with ACC: 385 us and 154).  Measured
// and not used: one plane for all rows and differences (bp_rows: 0.892 and
// 0.343 ms; loses sparse data's accuracy), and in that form the row pattern as
// arithmetic instead of a branch (1.021 ms), lane pairs split over two threads
// for twice the warps (0.941 ms), no prefetch of the next entry (0.977 ms).
// ============================================================================
// The shared planes are stored by phase, plane i at slot bp_slot(i): eight
// lanes of a warp take consecutive 4-plane runs of one row group, so that
// their loads of the same window offset are of one phase and contiguous.  The
// segments sit at offsets that keep a plane's phase (context creation), so
// the slots of a window's first four planes come from the row group's table
// entry, and the next two are one slot after the first two.
__device__ __forceinline__ int bp_slot(int i, int s4) { return (i & 3) * s4 + (i >> 2); }
// the shared plane at a byte address
__device__ __forceinline__ Q2 ldb(const float4 *P, int at) {
  return ldq(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(P) + at));
}

// one row of a wide entry on its own (steep segments of short scanners)
template <int KB>
__device__ __forceinline__ void bp_lerp(Q2 (&s)[KB], const float4 *__restrict__ P, int s4, int pbase, const BpLut &bl,
                                        int z0) {
  // windows wholly outside [zs, ze] contribute nothing; a window that
  // straddles an end reads the segment's zero planes for its outside planes
  if (z0 + KB - 1 < bl.zs || z0 > bl.ze) return;
  const int i0 = pbase + z0 + bl.d;
  const uint64_t f = pk(bl.f, bl.f), g = pk(1.0f - bl.f, 1.0f - bl.f);
  Q2 a = ldq(P + bp_slot(i0, s4));
#pragma unroll
  for (int j = 0; j < KB; j++) {
    const Q2 b = ldq(P + bp_slot(i0 + j + 1, s4));
    s[j] = qfma(b, f, qfma(a, g, s[j]));
    a = b;
  }
}

// one side of a segment group for a row group and a run of planes (BpRows):
// the first (SIDE 0) or last (SIDE 1) K rows are one plane further on; A[k]
// is where plane k of the window lies, A[0] + 16 and A[1] + 16 the next two.
// Each output adds its lower, then its upper plane by their own weights, as
// bp_lerp does.  Adding one plane to all rows and the planes' differences to
// each takes fewer operations (50 packed ones for 64), but cancels where a row
// gives a large plane next to no weight.
template <int SIDE, int K>
__device__ __forceinline__ void bp_rows(Q2 (&s)[kBpRows][kBpZ], const float4 *__restrict__ P, const int (&A)[4],
                                        const float4 &v) {
  const uint64_t f[kBpRows] = {pk(v.x, v.x), pk(v.y, v.y), pk(v.z, v.z), pk(v.w, v.w)};
  const uint64_t g[kBpRows] = {pk(1.0f - v.x, 1.0f - v.x), pk(1.0f - v.y, 1.0f - v.y), pk(1.0f - v.z, 1.0f - v.z),
                               pk(1.0f - v.w, 1.0f - v.w)};
#pragma unroll
  for (int k = 0; k < kBpZ + (K > 0 ? 2 : 1); k++) {
    const Q2 w = ldb(P, k < 4 ? A[k] : A[k - 4] + 16);
#pragma unroll
    for (int r = 0; r < kBpRows; r++) {
      const int on = (SIDE ? r >= kBpRows - K : r < K) ? 1 : 0;
      const int jl = k - on, ju = jl - 1;
      if (ju >= 0 && ju < kBpZ) s[r][ju] = qfma(w, f[r], s[r][ju]);
      if (jl >= 0 && jl < kBpZ) s[r][jl] = qfma(w, g[r], s[r][jl]);
    }
  }
}

template <int KB>
__device__ __forceinline__ void store_lane(float *__restrict__ dst, const Q2 (&s)[KB], int l) {
  float v[KB];
#pragma unroll
  for (int j = 0; j < KB; j++) {
    const float2 t = upk(l < 2 ? s[j].lo : s[j].hi);
    v[j] = (l & 1) ? t.y : t.x;
  }
  if constexpr (KB == 8) {
    // one 32-byte store (sm_100): a whole sector per lane, one line touched
    // per row of the warp's task tile instead of two stores to each
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < KB; j += 4)
      *reinterpret_cast<float4 *>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  }
}
// one lane of a run: stored, or (ACC) added to what is there by one 16-byte
// reduction (sm_90+) where the caller's buffer is aligned for it
template <bool ACC>
__device__ __forceinline__ void put(float *__restrict__ dst, const Q2 (&s)[kBpZ], int l, bool vec) {
  if constexpr (!ACC) {
    store_lane<kBpZ>(dst, s, l);
  } else {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 t = upk(l < 2 ? s[j].lo : s[j].hi);
      v[j] = (l & 1) ? t.y : t.x;
    }
    if (vec) {
      asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                   : "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) atomicAdd(dst + j, v[j]);
    }
  }
}

// Two CTAs per SM (their shared planes fill it at span 3) of 128 registers a
// thread.  Measured on B200 (span 3 / span 9 subset): 192 threads 1146 / 438
// us, 224 threads 1005 / 382 us, 256 threads 996 / 381 us.
constexpr int kBpThreads = 256;

template <bool ACC, bool MULTI>
__global__ void __launch_bounds__(kBpThreads, 2) bp_kernel(DevGeom g, const float4 *__restrict__ in,
                                                           long long in_pair_stride, const QuadWork *__restrict__ work,
                                                           float *__restrict__ bc, float *__restrict__ br,
                                                           long long vol, FrameStrides fr, int view0, int x0,
                                                           int split) {
  constexpr int KB = kBpZ, KR = kBpRows, NT = kBpThreads;
  extern __shared__ float4 P[];  // [bp_splanes]: segments with kBpPad zero planes each side
  __shared__ int2 s_base[kFpMaxGroups];  // per group: byte offset of yr 0 of its even / odd segment (of its slot)
  // ACC: one view pair, quads x0.., both partial sums added into bc (each
  // voxel receives exactly two terms, so the atomic adds onto a zeroed buffer
  // give a + b whatever their order)
  // MULTI: several frames per launch
  int item = blockIdx.x / split;
  const int part = blockIdx.x - item * split;
  if (MULTI) {
    const int nwork = gridDim.x / split / fr.n, frame = item / nwork;
    item -= frame * nwork;
    in += (size_t)frame * fr.ratio / 4;
    bc += (size_t)frame * fr.bc;
    br += (size_t)frame * fr.bc;
  }
  const QuadWork w = ACC ? QuadWork{0, (int16_t)(x0 + item), (int16_t)view0, 0} : work[item];
  const int x = w.x, N = g.nx, c = g.c, zp = g.zp, G = g.groupmax, s4 = g.bp_s4;
  const bool masked = g.nzmask[w.view * g.nquads + x] == 0;
  const float4 *src = in + (size_t)w.slot * in_pair_stride + (size_t)x * g.pplanes;
  if (!masked) {
#pragma unroll 8
    for (int i = threadIdx.x; i < g.bp_splanes; i += NT) {
      const int q = __ldg(g.bp_src + i);
      P[bp_slot(i, s4)] = (q >= 0) ? __ldg(src + q) : f4(0.f);
    }
    if (threadIdx.x < G)
      s_base[threadIdx.x] = make_int2(4 * (g.bp_soff[2 * threadIdx.x + 2] - g.ybot[2 * threadIdx.x + 2]),
                                      4 * (g.bp_soff[2 * threadIdx.x + 1] - g.ybot[2 * threadIdx.x + 2]));
  }
  __syncthreads();

  // ACC: both partial sums go through bc (br is unused and may be null), so
  // the two destinations derive from one restrict pointer
  float *bcp = bc + (size_t)w.slot * vol;
  float *brp = (ACC ? bc : br) + (size_t)w.slot * vol;
  const bool vec = ACC && (reinterpret_cast<uintptr_t>(bc) & 15) == 0;
  const int ystart = g.cyl0[x], o0 = g.bp_soff[0];
  const int m0 = ystart / KR, nm = max(0, (c - 1) / KR + 1 - m0), nzc = zp / KB;
  // A warp takes 16 consecutive plane runs of one row group in both halves:
  // half 0 builds sumt1, half 1 sumt2.  The halves read the two segments of a
  // group at the same position, so a warp's lanes take the same path through
  // bp_rows.  The last tiles are 32 plane runs of the centre row, y = c.
  const int lane = threadIdx.x & 31, half = lane >> 4;
  const int CT = (nzc + 15) / 16, tiles = nm * CT;
  const int step = split * (NT / 32);
  // column voxels (x, yc), (N-x, yc); row voxels (yr, x), (yr, N-x)
  auto put4 = [&](const Q2 (&v)[KB], int yc, int yr, int z0) {
    put<ACC>(bcp + ((size_t)x * N + yc) * zp + z0, v, 0, vec);
    put<ACC>(brp + ((size_t)yr * N + x) * zp + z0, v, 2, vec);
    if (x != c) {
      put<ACC>(bcp + ((size_t)(N - x) * N + yc) * zp + z0, v, 1, vec);
      put<ACC>(brp + ((size_t)yr * N + N - x) * zp + z0, v, 3, vec);
    }
  };
  for (int tile = part * (NT / 32) + (threadIdx.x >> 5); tile < tiles + (nzc + 31) / 32; tile += step) {
    if (tile >= tiles) {
      // centre row (sbrt:4260-4284): a single voxel set, rays pass plane
      // yr = z exactly
      const int zc = (tile - tiles) * 32 + lane, z0 = zc * KB;
      if (zc >= nzc) continue;
      Q2 t[KB];
#pragma unroll
      for (int j = 0; j < KB; j++) t[j] = masked ? Q2{0ull, 0ull} : ldq(P + o0 / 4 + zc + j * s4);
      for (int gg = 0; gg < (masked ? 0 : G); gg++) {
        const int2 base = s_base[gg];
        const int yb = g.ybot[2 * gg + 2], yt = g.ytop[2 * gg + 2];
#pragma unroll
        for (int j = 0; j < KB; j++) {
          const int at = 16 * (zc + j * s4);
          if (z0 + j >= yb && z0 + j <= yt) t[j] = qadd(t[j], qadd(ldb(P, base.x + at), ldb(P, base.y + at)));
        }
      }
#pragma unroll
      for (int j = 0; j < KB; j++)
        if (z0 + j >= g.nz) t[j] = Q2{0ull, 0ull};
      put4(t, c, c, z0);
      continue;
    }
    const int ty = tile / CT, tc = tile - ty * CT;
    const int m = m0 + ty, zc = tc * 16 + (lane & 15), z0 = zc * KB;
    if (zc >= nzc) continue;
    Q2 s[KR][KB];
    // masked quads contribute zero (sbrt:4223-4258, :4595-4640)
#pragma unroll
    for (int j = 0; j < KB; j++) {
      s[0][j] = masked ? Q2{0ull, 0ull} : ldq(P + o0 / 4 + zc + j * s4);
#pragma unroll
      for (int r = 1; r < KR; r++) s[r][j] = s[0][j];
    }
    if (!masked) {
      const int4 *e = reinterpret_cast<const int4 *>(g.bprows + (size_t)m * G * 2);
      int4 hn = __ldg(e);
      float4 fn = __ldg(reinterpret_cast<const float4 *>(e + 1));
      // one side of group gg; sumt1: segment 2k at +u (side 0, rows y) and
      // 2k-1 at -u (side 1, rows N-y); sumt2: the converse
      auto side_of = [&](auto side_c, int gg, int seg, bool last) {
        constexpr int SIDE = decltype(side_c)::value;
        const int4 h = hn;
        const float4 v = fn;
        if (!last) {  // the next entry, in flight under this one's planes
          e += 2;
          hn = __ldg(e);
          fn = __ldg(reinterpret_cast<const float4 *>(e + 1));
        }
        if (z0 + KB - 1 < (int)(int16_t)(h.z & 0xffff) || z0 > (h.z >> 16)) return;
        const int B = seg + 16 * zc;
        const int A[4] = {B + 16 * (int)(int16_t)(h.x & 0xffff), B + 16 * (h.x >> 16),
                          B + 16 * (int)(int16_t)(h.y & 0xffff), B + 16 * (h.y >> 16)};
        switch (h.w) {
          case 0: bp_rows<SIDE, 0>(s, P, A, v); break;
          case 1: bp_rows<SIDE, 1>(s, P, A, v); break;
          case 2: bp_rows<SIDE, 2>(s, P, A, v); break;
          case 3: bp_rows<SIDE, 3>(s, P, A, v); break;
          default:
#pragma unroll
            for (int r = 0; r < KR; r++) {
              const int y = min(max(KR * m + r, 1), c - 1);
              bp_lerp<KB>(s[r], P, s4, seg / 4, g.bplut[(size_t)gg * N + (SIDE ? N - y : y)], z0);
            }
        }
      };
      for (int gg = 0; gg < G; gg++) {
        const int2 base = s_base[gg];
        side_of(std::integral_constant<int, 0>{}, gg, half ? base.y : base.x, false);
        side_of(std::integral_constant<int, 1>{}, gg, half ? base.x : base.y, gg + 1 == G);
      }
    }
#pragma unroll
    for (int r = 0; r < KR; r++) {
      const int y = KR * m + r;
      if (y < ystart || y >= c) continue;
      // the reference writes planes z < nz only
#pragma unroll
      for (int j = 0; j < KB; j++)
        if (z0 + j >= g.nz) s[r][j] = Q2{0ull, 0ull};
      put4(s[r], half ? N - y : y, half ? y : N - y, z0);
    }
  }
}

// ============================================================================
// Exact adjoint of the forward projector (no counterpart in the reference,
// whose back projector is not the transpose of its forward projector).
//
// adj_kernel: per (pair, quad x) the forward projector's z interpolation
// transposed -- every rotated-frame sample of the forward projection receives
// the rows it fed, weighted as it was weighted (sbrt:1914-1951 read backwards:
// the middle planes are two windows of the segment, the end planes one
// position each), with the rows first scaled as the forward projector scales
// them (sbrt:1953-1976).  The samples are the back projector's voxel roles, so
// the lanes go to the same column / row partials.  An output plane gathers
// its end planes by table (at most four consecutive ones); where it takes
// more, or an end has few planes, the task walks the entries in order (GATHER
// false).  Bound by
// the shared reads and the chain of table -> end plane -> FMA: four planes'
// entries in flight at three CTAs an SM measured 1057 us a span-9 subset of
// the HRRT (1329 entry by entry; one plane at a time 1322, eight planes at
// two CTAs 1315, two at four 1621); without any end planes 560.
// adj_rotate_kernel: the bilinear sampling transposed as a gather: an image
// voxel collects from the <= 16 rotated-frame points around its inverse
// rotation whose sample footprint (recomputed with the forward projector's own
// float expressions) holds it, with that footprint's weight.
// ============================================================================


// One side of a segment group's middle planes transposed: for the task's
// planes z0 + j, s[j] += w0 * P[a0 + j - d0] + w1 * P[a0 + j - d1] over the
// window entries inside [lo, hi] (d0, d1 in {0, 1}).  Windows wholly inside
// the middle planes slide without checks; windows that straddle an end check
// each entry.
template <int KB>
__device__ __forceinline__ void adj_side(Q2 (&s)[KB], const float4 *__restrict__ P, int a0, int lo, int hi,
                                         uint64_t w_at, uint64_t w_below) {
  // w_at multiplies P[a0 + j], w_below multiplies P[a0 + j - 1]
  if (a0 - 1 >= lo && a0 + KB - 1 <= hi) {
    Q2 prev = ldq(P + a0 - 1);
#pragma unroll
    for (int j = 0; j < KB; j++) {
      const Q2 cur = ldq(P + a0 + j);
      s[j] = qfma(prev, w_below, qfma(cur, w_at, s[j]));
      prev = cur;
    }
  } else if (a0 + KB - 1 >= lo && a0 - 1 <= hi) {
#pragma unroll
    for (int j = 0; j < KB; j++) {
      const int ya = a0 + j;
      if (ya >= lo && ya <= hi) s[j] = qfma(ldq(P + ya), w_at, s[j]);
      if (ya - 1 >= lo && ya - 1 <= hi) s[j] = qfma(ldq(P + ya - 1), w_below, s[j]);
    }
  }
}

constexpr int kAdjBatch = 4;
template <int KB, bool GATHER>
__global__ void __launch_bounds__(256, 3) adj_kernel(DevGeom g, const float4 *__restrict__ in, long long in_pair_stride,
                                                  const QuadWork *__restrict__ work, float *__restrict__ bc,
                                                  float *__restrict__ br, long long vol, FrameStrides fr) {
  extern __shared__ float4 P[];
  const int nwork = gridDim.x / fr.n, frame = blockIdx.x / nwork, item = blockIdx.x - frame * nwork;
  const QuadWork w = work[item];
  in += (size_t)frame * fr.ratio / 4;
  bc += (size_t)frame * fr.bc;
  br += (size_t)frame * fr.bc;
  const int x = w.x, N = g.nx, c = g.c, zp = g.zp, G = g.groupmax, ZS = g.zshift, nz = g.nz;
  const bool masked = g.nzmask[w.view * g.nquads + x] == 0 || g.cyl0[x] == g.cyl1[x];
  const float4 *src = in + (size_t)w.slot * in_pair_stride + (size_t)x * g.pplanes;
  if (!masked)
    for (int i = threadIdx.x; i < g.bp_splanes; i += blockDim.x) {
      const int q = __ldg(g.bp_src + i);
      float4 v = f4(0.f);
      if (q >= 0) {
        const int sg = g.pplane_seg[q];
        const int yb = g.ybot[sg], yr = yb + (q - g.poff[sg]);
        float sc = g.y_size;
        if (sg > 0) {
          int zs = yr - yb;
          if (zs >= ZS) zs = g.ytop[sg] - yr;
          sc = g.rescale[((sg - 1) >> 1) * nz + (zs < ZS ? yr : yb + ZS)];
        }
        v = src[q] * sc;
      }
      P[i] = v;
    }
  __syncthreads();
  float *bcp = bc + (size_t)w.slot * vol;
  float *brp = br + (size_t)w.slot * vol;
  const int ystart = g.cyl0[x];
  const int nyq = c - ystart + 1, nzc = zp / KB;
  const float4 *P0 = P + g.bp_soff[0];
  // a warp's 32 tasks are 32 consecutive rows at one plane run: the rows'
  // table entries ([group][row]) are contiguous, the stores whole sectors
  const int per_half = nyq * nzc;
  for (int task = threadIdx.x; task < 2 * per_half; task += blockDim.x) {
    const int half = task >= per_half;
    const int t2 = task - half * per_half;
    const int zc = t2 / nyq, yi = t2 - zc * nyq, z0 = zc * KB;
    const int y = ystart + yi;
    if (half && y == c) continue;
    Q2 s[KB];
#pragma unroll
    for (int j = 0; j < KB; j++) s[j] = Q2{0ull, 0ull};
    if (!masked) {
#pragma unroll
      for (int j = 0; j < KB; j++) s[j] = ldq(P0 + z0 + j);
      if (y == c) {
        // centre row: every plane of every segment took the centre samples
        for (int gg = 0; gg < G; gg++) {
          const int se = 2 * gg + 2, so = 2 * gg + 1;
          const int yb = g.ybot[se], yt = g.ytop[se];
          const float4 *pe = P + g.bp_soff[se] - yb, *po = P + g.bp_soff[so] - yb;
#pragma unroll
          for (int j = 0; j < KB; j++) {
            const int z = z0 + j;
            if (z >= yb && z <= yt) s[j] = qadd(s[j], qadd(ldq(pe + z), ldq(po + z)));
          }
        }
      } else {
        const FpMid *mrow = g.fpmid_t + y;
        const int2 *e1 = g.fl_t + y, *e2 = g.fl_t + (N - y);
        for (int gg = 0; gg < G; gg++) {
          const FpMid m = mrow[(size_t)gg * c];
          if (m.z < 0) continue;  // the forward projector skipped this group for this row
          const int se = 2 * gg + 2, so = 2 * gg + 1;
          const int yb = g.ybot[se], yt = g.ytop[se], ym = yb + ZS, ye = yt - ZS;
          // A: the rows that read this sample at (z, z+1) with (f2, f); B:
          // the rows that read it at (z2+1, z2) with (f2, f)
          const float4 *A = P + g.bp_soff[half ? so : se] - yb, *B = P + g.bp_soff[half ? se : so] - yb;
          const uint64_t f = pk(m.f, m.f), f2 = pk(m.f2, m.f2);
          adj_side<KB>(s, A, z0 - m.z + ym, ym, ye, f2, f);
          adj_side<KB>(s, B, z0 - m.z2 + ym, ym, ye, f, f2);
          if (GATHER) {
            // end planes: what each output plane takes from them, by table
#pragma unroll 1
            for (int k = 0; k < 4; k++) {  // side k / 2, end k & 1
              const size_t zb = ((size_t)gg * 4 + k) * c + y;
              const short2 zr = __ldg(g.adj_endz + zb);
              if (z0 > zr.y || z0 + KB - 1 < zr.x) continue;
              const float4 *E = (k < 2 ? A : B) + ((k & 1) ? yt - ZS + 1 : yb);
              const size_t tb = ((size_t)gg * 4 + k) * kAdjEndOut * c + y;
#pragma unroll
              for (int j0 = 0; j0 < KB; j0 += kAdjBatch) {
                // kAdjBatch planes' entries in flight together
                int en[kAdjBatch];
                float4 wt[kAdjBatch];
#pragma unroll
                for (int i = 0; i < kAdjBatch; i++) {
                  const int z = z0 + j0 + i;
                  const bool in = z >= zr.x && z <= zr.y;
                  const size_t at = tb + (size_t)(in ? z - zr.x : 0) * c;
                  en[i] = __ldg(reinterpret_cast<const int *>(g.adj_ends) + at);
                  wt[i] = __ldg(g.adj_endw + at);
                  if (!in) en[i] = 0;
                }
#pragma unroll
                for (int i = 0; i < kAdjBatch; i++) {
                  const float4 *e0 = E + (int)(int16_t)(en[i] & 0xffff);
                  const int n = en[i] >> 16;
                  Q2 &t = s[j0 + i];
                  if (n > 0) t = qfma(ldq(e0), pk(wt[i].x, wt[i].x), t);
                  if (n > 1) t = qfma(ldq(e0 + 1), pk(wt[i].y, wt[i].y), t);
                  if (n > 2) t = qfma(ldq(e0 + 2), pk(wt[i].z, wt[i].z), t);
                  if (n > 3) t = qfma(ldq(e0 + 3), pk(wt[i].w, wt[i].w), t);
                }
              }
            }
            continue;
          }
          // end planes: one position per plane; an end whose entries touch
          // no plane of this task's run is skipped whole
          const size_t eb = (size_t)gg * 2 * ZS * N;
          const int4 er = __ldg(g.adj_endr + (size_t)gg * c + y);
          const bool bot = er.x < z0 + KB && er.y >= z0, top = er.z < z0 + KB && er.w >= z0;
          for (int i = bot ? 0 : ZS; i < (top ? 2 * ZS : ZS); i++) {
            const int2 u = __ldg(e1 + eb + (size_t)i * N), v = __ldg(e2 + eb + (size_t)i * N);
            const int za = u.x, zb = v.x;
            if ((za + 1 < z0 || za >= z0 + KB) && (zb + 1 < z0 || zb >= z0 + KB)) continue;
            const int yr = (i < ZS) ? yb + i : yt - 2 * ZS + 1 + i;
            const float fa = __int_as_float(u.y), fb = __int_as_float(v.y);
            const uint64_t pfa = pk(fa, fa), pfb = pk(fb, fb);
            const Q2 a = ldq(A + yr), b = ldq(B + yr);
#pragma unroll
            for (int j = 0; j < KB; j++) {
              const int z = z0 + j;
              if (z == za) s[j] = qfma(a, pfb, s[j]);
              if (z == za + 1) s[j] = qfma(a, pfa, s[j]);
              if (z == zb + 1) s[j] = qfma(b, pfb, s[j]);
              if (z == zb) s[j] = qfma(b, pfa, s[j]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KB; j++)
      if (z0 + j >= nz) s[j] = Q2{0ull, 0ull};
    const size_t cz = (size_t)z0;
    if (!half) {
      store_lane<KB>(bcp + ((size_t)x * N + y) * zp + cz, s, 0);
      store_lane<KB>(brp + ((size_t)(N - y) * N + x) * zp + cz, s, 2);
      if (x != c) {
        store_lane<KB>(bcp + ((size_t)(N - x) * N + y) * zp + cz, s, 1);
        store_lane<KB>(brp + ((size_t)(N - y) * N + N - x) * zp + cz, s, 3);
      }
    } else {
      store_lane<KB>(bcp + ((size_t)x * N + N - y) * zp + cz, s, 0);
      store_lane<KB>(brp + ((size_t)y * N + x) * zp + cz, s, 2);
      if (x != c) {
        store_lane<KB>(bcp + ((size_t)(N - x) * N + N - y) * zp + cz, s, 1);
        store_lane<KB>(brp + ((size_t)y * N + N - x) * zp + cz, s, 3);
      }
    }
  }
}

// For each pair slot and voxel column (every column for MODE 2, the FOV
// columns otherwise): the rotated-frame points (a, b) around the column's
// inverse rotation whose forward-projection sample footprint -- recomputed
// with the forward projector's own float expressions -- covers the column,
// with that footprint's weight, in scan order.  One thread per (pair, column);
// the rotate then reads these instead of every thread of a column repeating
// the 16 candidate footprints.
template <int MODE>
__global__ void __launch_bounds__(256) adj_cover_kernel(DevGeom g, const int *__restrict__ pair_views, int npairs) {
  const int N = g.nx, c = g.c;
  const long long ncols = (MODE == 2) ? (long long)N * N : g.fov_columns;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncols * npairs) return;
  const int p = (int)(t / ncols);
  const int col = (int)(t - (long long)p * ncols);
  int i, j;
  if (MODE == 2) {
    i = col / N;
    j = col - i * N;
  } else {
    const short2 xy = g.fov_xy[col];
    i = xy.x;
    j = xy.y;
  }
  const int view = pair_views[p];
  const float cosv = g.cos_psi[view], sinv = g.sin_psi[view];
  const float di = (float)(i - c), dj = (float)(j - c);
  const int qx0 = (int)floorf(di * cosv + dj * sinv + (float)c) - 1;
  const int qy0 = (int)floorf(-di * sinv + dj * cosv + (float)c) - 1;
  int2 *ent = g.adj_ent + t * kAdjCover;
  int n = 0;
  for (int a = qx0; a < qx0 + 4; a++) {
    if (a < 0 || a >= N) continue;
    for (int b = qy0; b < qy0 + 4; b++) {
      if (b < 0 || b >= N) continue;
      const SamplePt pt = sample_point(a, b, c, N, g.zp, cosv, sinv);
      if (pt.base < 0) continue;
      const int ix = pt.base / (N * g.zp), iy = (pt.base / g.zp) - ix * N;
      const int dx = i - ix, dy = j - iy;
      if (dx < 0 || dx > 1 || dy < 0 || dy > 1) continue;
      const float wgt = dx ? (dy ? pt.c3 : pt.c1) : (dy ? pt.c2 : pt.c0);
      if (n < kAdjCover) ent[n] = make_int2(a * N + b, __float_as_int(wgt));
      n++;
    }
  }
  if (n > kAdjCover) atomicExch(g.err, 2);  // more covering points than the table holds: results void
  g.adj_cnt[t] = min(n, kAdjCover);
}

// MODE 0: OSEM update, 1: inverse sensitivity (both over the FOV columns, as
// the rotate-back), 2: out += adjoint over every image column.
template <int MODE>
__global__ void __launch_bounds__(256) adj_rotate_kernel(DevGeom g, const int *__restrict__ pair_views, int npairs,
                                                         const float *__restrict__ bc, const float *__restrict__ br,
                                                         long long vol, float *__restrict__ image,
                                                         float *__restrict__ nf_inv, float *__restrict__ out,
                                                         FrameStrides fr) {
  const int nq = g.zp / 4, N = g.nx;
  if (MODE == 0) {
    image += (size_t)(fr.map ? __ldg(fr.map + blockIdx.y) : (int)blockIdx.y) * fr.image;
    bc += (size_t)blockIdx.y * fr.bc;
    br += (size_t)blockIdx.y * fr.bc;
  }
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int col = (int)(t / nq), q = (int)(t - (long long)col * nq);
  int i, j;
  if (MODE == 2) {
    if (col >= N * N) return;
    i = col / N;
    j = col - i * N;
  } else {
    if (col >= g.fov_columns) return;
    const short2 xy = g.fov_xy[col];
    i = xy.x;
    j = xy.y;
  }
  // the covering points of this column, found once per pair by
  // adj_cover_kernel in this scan order
  const long long ncols = (MODE == 2) ? (long long)N * N : g.fov_columns;
  float4 acc = f4(0.f);
  for (int p = 0; p < npairs; p++) {
    const float4 *Bc = reinterpret_cast<const float4 *>(bc + (size_t)p * vol);
    const float4 *Br = reinterpret_cast<const float4 *>(br + (size_t)p * vol);
    const long long e0 = (long long)p * ncols + col;
    const int n = __ldg(g.adj_cnt + e0);
    const int2 *ent = g.adj_ent + e0 * kAdjCover;
    for (int k = 0; k < n; k++) {
      const int2 u = __ldg(ent + k);
      const size_t o = (size_t)u.x * nq + q;
      acc = acc + (__ldg(Bc + o) + __ldg(Br + o)) * __int_as_float(u.y);
    }
  }
  const size_t o = ((size_t)i * N + j) * nq + q;
  if (MODE == 0) {
    float4 *im = reinterpret_cast<float4 *>(image);
    const float4 nf = reinterpret_cast<const float4 *>(nf_inv)[o];
    float4 iv = im[o];
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, b[4] = {iv.x, iv.y, iv.z, iv.w}, n[4] = {nf.x, nf.y, nf.z, nf.w};
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const float lo = (0.01f > a[l]) ? 0.01f : a[l];
      const float cl = (100.0f < lo) ? 100.0f : lo;
      const float u = b[l] * (cl * n[l]);
      b[l] = (g.image_max < u) ? g.image_max : u;
    }
    im[o] = make_float4(b[0], b[1], b[2], b[3]);
  } else if (MODE == 1) {
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, r[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const int z = q * 4 + l;
      r[l] = (z < g.nz && fabsf(a[l]) > g.eps1) ? (1.0f / a[l]) : 0.f;
    }
    reinterpret_cast<float4 *>(nf_inv)[o] = make_float4(r[0], r[1], r[2], r[3]);
  } else {
    float4 *dst = reinterpret_cast<float4 *>(out);
    dst[o] = dst[o] + acc;
  }
}

// ============================================================================
// Rotate-back of the summed partials of every pair (rotateimage2, sbrt:1137-
// 1186) fused with what consumes the correction image:
//   MODE 0: OSEM update pt_cal_updateimage (drv:2018-2059)
//   MODE 1: inverse sensitivity pt_normfac_calculate (drv:1852-1894)
//   MODE 2: corr_out += rotate-back (rotate_image_buf for one view)
// One thread per (FOV column, 4 planes); pairs are added in subset order.
// ============================================================================
template <int MODE>
__global__ void __launch_bounds__(256) rotback_kernel(DevGeom g, const int *__restrict__ pair_views, int npairs,
                                                      const float *__restrict__ bc, const float *__restrict__ br,
                                                      long long vol, float *__restrict__ image,
                                                      float *__restrict__ nf_inv, float *__restrict__ corr_out,
                                                      FrameStrides fr) {
  const int nq = g.zp / 4;
  if (MODE == 0) {
    image += (size_t)(fr.map ? __ldg(fr.map + blockIdx.y) : (int)blockIdx.y) * fr.image;
    bc += (size_t)blockIdx.y * fr.bc;
    if (br != nullptr) br += (size_t)blockIdx.y * fr.bc;
  }
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int col = (int)(t / nq), q = (int)(t - (long long)col * nq);
  if (col >= g.fov_columns) return;
  const short2 xy = g.fov_xy[col];
  const int N = g.nx;
  float4 acc = f4(0.f);
  for (int p = 0; p < npairs; p++) {
    const float2 pos = g.rotpos[(size_t)pair_views[p] * g.fov_columns + col];
    const int ix = (int)pos.x, iy = (int)pos.y;
    if (ix < 0 || ix > N - 2 || iy < 0 || iy > N - 2) continue;
    const float x1 = pos.x - ix, y1 = pos.y - iy;
    const float c1 = (1 - x1) * (1 - y1), c2 = x1 * (1 - y1), c3 = y1 * (1 - x1), c4 = y1 * x1;
    const float4 *Bc = reinterpret_cast<const float4 *>(bc + (size_t)p * vol);
    const size_t i1 = ((size_t)ix * N + iy) * nq + q, i2 = i1 + (size_t)N * nq, i3 = i1 + nq, i4 = i2 + nq;
    float4 b1 = __ldg(Bc + i1), b2 = __ldg(Bc + i2), b3 = __ldg(Bc + i3), b4 = __ldg(Bc + i4);
    if (br != nullptr) {
      const float4 *Br = reinterpret_cast<const float4 *>(br + (size_t)p * vol);
      b1 = b1 + __ldg(Br + i1);
      b2 = b2 + __ldg(Br + i2);
      b3 = b3 + __ldg(Br + i3);
      b4 = b4 + __ldg(Br + i4);
    }
    acc = acc + ((b1 * c1 + b2 * c2) + (b3 * c3 + b4 * c4));
  }
  const size_t o = ((size_t)xy.x * N + xy.y) * nq + q;
  if (MODE == 0) {
    float4 *im = reinterpret_cast<float4 *>(image);
    const float4 nf = reinterpret_cast<const float4 *>(nf_inv)[o];
    float4 iv = im[o];
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, b[4] = {iv.x, iv.y, iv.z, iv.w}, n[4] = {nf.x, nf.y, nf.z, nf.w};
#pragma unroll
    for (int l = 0; l < 4; l++) {
      // _mm_max_ps(0.01, c), _mm_min_ps(100, .), _mm_min_ps(image_max, .):
      // each returns its second operand when either is NaN
      const float lo = (0.01f > a[l]) ? 0.01f : a[l];
      const float cl = (100.0f < lo) ? 100.0f : lo;
      const float u = b[l] * (cl * n[l]);
      b[l] = (g.image_max < u) ? g.image_max : u;
    }
    im[o] = make_float4(b[0], b[1], b[2], b[3]);
  } else if (MODE == 1) {
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, r[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const int z = q * 4 + l;
      r[l] = (z < g.nz && fabsf(a[l]) > g.eps1) ? (1.0f / a[l]) : 0.f;
    }
    reinterpret_cast<float4 *>(nf_inv)[o] = make_float4(r[0], r[1], r[2], r[3]);
  } else if (MODE == 2) {
    float4 *co = reinterpret_cast<float4 *>(corr_out);
    co[o] = co[o] + acc;
  } else {
    reinterpret_cast<float4 *>(corr_out)[o] = acc;
  }
}

// rotate-back sample positions, incremented along y exactly as rotateimage2
// does (sbrt:1148-1184)
__global__ void rotpos_kernel(DevGeom g, float2 *__restrict__ rotpos, const int *__restrict__ row_start) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, vi = blockIdx.y;
  if (X >= g.nx) return;
  const int N = g.nx, h = N / 2;
  const float cosv = g.cos_psi[vi] / 1.0f;
  const float sinv = -g.sin_psi[vi] / 1.0f;
  const float xxx0 = (float)(-N / 2) * cosv + (float)h * sinv + (float)h;
  const float yyy0 = (float)(-N / 2) * sinv - (float)h * cosv + (float)h;
  const int ys = g.cyl0[X], ye = g.cyl1[X];
  float xx0 = xxx0 - (float)ys * sinv + (float)X * cosv;
  float yy0 = yyy0 + (float)ys * cosv + (float)X * sinv;
  float2 *dst = rotpos + (size_t)vi * g.fov_columns + row_start[X];
  for (int y = ys; y < ye; y++) {
    dst[y - ys] = make_float2(xx0, yy0);
    xx0 -= sinv;
    yy0 += cosv;
  }
}

// ============================================================================
// Input preparation + re-layout (prepare_norm/norm_ANW drv:796-1056,
// prepare_osem3dw3 drv:1649-1818, mul/add projection simd_operation.cpp:4-58)
// from the flat file layout into the quad layout.  One thread per (pair,
// quad, run of planes).
// ============================================================================
template <typename PT, typename AT>
__global__ void prep_kernel(DevGeom g, int nbins, const int16_t *__restrict__ prompts,
                            const float *__restrict__ randoms, const float *__restrict__ norm,
                            const float *__restrict__ atten, const float *__restrict__ scatter, int npskip,
                            float eps2, PT *__restrict__ qp, AT *__restrict__ qadd, AT *__restrict__ qmult,
                            int *__restrict__ mask_accum, int planes_per_thread, int plane0, int nplanes,
                            const int *__restrict__ pair_views, long long s_plane, long long s_half,
                            long long s_slot, long long pf_plane, long long pf_half) {
  // Input element of plane gp, lane l: base + (gp - plane0)*s_plane + h*s_half
  // + bin.  Flat-file chunk (pair_views null): pair = blockIdx.z, base =
  // pair*nbins, planes [plane0, plane0 + nplanes).  Pair-major staging: pair =
  // pair_views[blockIdx.z], base = blockIdx.z*s_slot, all planes.  With
  // pf_plane > 0 the prompts are the whole sinogram instead: element
  // gp*pf_plane + pair*nbins + h*pf_half + bin.
  const int x = blockIdx.x * blockDim.x + threadIdx.x;  // quad
  const int vi = pair_views ? pair_views[blockIdx.z] : (int)blockIdx.z;
  const long long base = pair_views ? (long long)blockIdx.z * s_slot : (long long)vi * nbins;
  if (x >= g.nquads) return;
  const int gp0 = plane0 + blockIdx.y * planes_per_thread;
  const int gp1 = min(gp0 + planes_per_thread, plane0 + nplanes);
  const int hl[4] = {0, 0, 1, 1};
  int bins[4] = {x, nbins - x, x, nbins - x};
  bool ok[4];
  for (int l = 0; l < 4; l++) ok[l] = (bins[l] >= 0 && bins[l] < nbins && x > 0);
  int any = 0;
  for (int gp = gp0; gp < gp1; gp++) {
    const int s = g.plane_seg[gp];
    const int segoff = g.poff[s] - 2 * s - 1;
    const int r = gp - segoff, ns = g.ytop[s] - g.ybot[s] + 1;
    const bool kill = (r < npskip || r + npskip >= ns);
    float pv[4], av[4], mv[4];
    for (int l = 0; l < 4; l++) {
      pv[l] = av[l] = mv[l] = 0.f;
      if (!ok[l]) continue;
      const size_t i = (size_t)(base + (long long)(gp - plane0) * s_plane + hl[l] * s_half + bins[l]);
      const float nz = norm ? (kill ? 0.f : __ldg(norm + i)) : 1.0f;
      const float araw = atten ? __ldg(atten + i) : 1.0f;
      const float ac = (araw < 1.0f) ? 1.0f : araw;
      float m;
      if (nz > 0.0f) {
        const float den = nz * ac;
        m = (den > eps2) ? 1.0f / den : 0.0f;
      } else {
        m = nz;
      }
      float a = __ldg(randoms + i) * nz;
      if (scatter) a = a + __ldg(scatter + i);
      a = a * araw;
      const size_t pi = pf_plane > 0 ? (size_t)((long long)gp * pf_plane + (long long)vi * nbins +
                                                hl[l] * pf_half + bins[l])
                                     : i;
      const float p = (nz == 0.0f) ? 0.f : (float)__ldg(prompts + pi);
      if (nz != 0.0f) any = 1;
      pv[l] = p;
      av[l] = a;
      mv[l] = m;
    }
    const size_t o = ((size_t)vi * g.nquads + x) * g.pplanes + g.poff[s] + r;
    if (std::is_same<AT, __half>::value) {
      // fp16 holds magnitudes up to 65504: a larger term is reported, not stored wrapped
      bool over = false;
      for (int l = 0; l < 4; l++) over |= fabsf(av[l]) > 65504.f || fabsf(mv[l]) > 65504.f;
      if (over) atomicOr(g.range_err, 1);
    }
    store_p4(qp, o, pv);
    store_p4(qadd, o, av);
    store_p4(qmult, o, mv);
  }
  if (any) atomicOr(mask_accum + vi * g.nquads + x, 1);
}

__global__ void finish_mask_kernel(DevGeom g, const int *__restrict__ accum, int16_t *__restrict__ nzmask) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (g.nviews / 2) * g.nquads) return;
  const int x = i % g.nquads;
  nzmask[i] = (x == 0) ? 1 : (accum[i] ? 1 : 0);
}

__global__ void init_image_kernel(DevGeom g, float *__restrict__ image) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)g.nx * g.nx * g.zp;
  if (t >= total) return;
  const int z = (int)(t % g.zp);
  const long long xy = t / g.zp;
  const int X = (int)(xy / g.nx), Y = (int)(xy % g.nx);
  const bool fov = g.cyl0[X] != g.cyl1[X] && Y >= g.cyl0[X] && Y < g.cyl1[X];
  image[t] = (fov && z >= g.z_min && z < g.z_max) ? 1.0f : 0.0f;
}

// post-iteration pass (drv:4288-4297) with an FP64 sum, deterministic:
// per-block partial sums, then one block adds them in order.
__global__ void post_iter_kernel(DevGeom g, float *__restrict__ image, double *__restrict__ partial,
                                 FrameStrides fr) {
  __shared__ double red[256];
  image += (size_t)(fr.map ? __ldg(fr.map + blockIdx.y) : (int)blockIdx.y) * fr.image;
  partial += (size_t)blockIdx.y * fr.partial;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nz = g.z_max - g.z_min;
  double s = 0.0;
  if (t < (long long)g.fov_columns * nz) {
    const int col = (int)(t / nz), z = g.z_min + (int)(t % nz);
    const short2 xy = g.fov_xy[col];
    float *p = image + ((size_t)xy.x * g.nx + xy.y) * g.zp + z;
    const float v = *p;
    s = (double)v;
    if ((double)v < 1e-16) *p = 0.f;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}
// One block: each thread sums a contiguous run of partials, then a fixed
// tree adds the runs -- the same order on every call (deterministic).
__global__ void sum_partials_kernel(const double *__restrict__ partial, int n, double *__restrict__ out,
                                    long long frame_stride, const int *__restrict__ map) {
  __shared__ double red[1024];
  partial += (size_t)blockIdx.x * frame_stride;
  out += map ? map[blockIdx.x] : (int)blockIdx.x;
  const int t = threadIdx.x, T = blockDim.x;
  const int per = (n + T - 1) / T, b = t * per, e = min(b + per, n);
  double s = 0.0;
  for (int i = b; i < e; i++) s += partial[i];
  red[t] = s;
  __syncthreads();
  for (int k = T / 2; k > 0; k >>= 1) {
    if (t < k) red[t] += red[t + k];
    __syncthreads();
  }
  if (t == 0) *out = red[0];
}

__global__ void rows_to_quad_kernel(DevGeom g, int nbins, const float *__restrict__ rows, float4 *__restrict__ quad,
                                    int apply_bp_scale) {
  const int gp = blockIdx.y, x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= g.nquads || gp >= g.segmentsize) return;
  const int s = g.plane_seg[gp];
  const int segoff = g.poff[s] - 2 * s - 1;
  const int r = gp - segoff;
  const size_t P = g.segmentsize;
  const int xm = nbins - x;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (x > 0) {
    v[0] = rows[(size_t)gp * nbins + x];
    v[1] = rows[(size_t)gp * nbins + xm];
    v[2] = rows[(P + gp) * nbins + x];
    v[3] = rows[(P + gp) * nbins + xm];
  }
  if (apply_bp_scale) {
    const float bs = g.bp_scale[s];
    for (int l = 0; l < 4; l++) v[l] = v[l] * bs;
  }
  quad[(size_t)x * g.pplanes + g.poff[s] + r] = make_float4(v[0], v[1], v[2], v[3]);
}

__global__ void quad_to_rows_kernel(DevGeom g, int nbins, const float4 *__restrict__ quad,
                                    const QuadWork *__restrict__ work, float *__restrict__ rows) {
  const int gp = blockIdx.x * blockDim.x + threadIdx.x;
  const QuadWork w = work[blockIdx.y];
  if (gp >= g.segmentsize) return;
  const int s = g.plane_seg[gp];
  const int segoff = g.poff[s] - 2 * s - 1;
  const int r = gp - segoff;
  const size_t P = g.segmentsize;
  const int x = w.x, xm = nbins - x;
  const float4 q = quad[(size_t)x * g.pplanes + g.poff[s] + r];
  rows[(size_t)gp * nbins + x] = q.x;
  rows[(size_t)gp * nbins + xm] = q.y;
  rows[(P + gp) * nbins + x] = q.z;
  rows[(P + gp) * nbins + xm] = q.w;
}

__global__ void quad_to_file_kernel(DevGeom g, int nbins, const float4 *__restrict__ quad, long long stride,
                                    const QuadWork *__restrict__ work, float *__restrict__ sino) {
  const int gp = blockIdx.x * blockDim.x + threadIdx.x;
  const QuadWork w = work[blockIdx.y];
  if (gp >= g.segmentsize) return;
  const int s = g.plane_seg[gp];
  const int r = gp - (g.poff[s] - 2 * s - 1);
  const int x = w.x, xm = nbins - x, V = g.nviews;
  const float4 q = quad[(size_t)w.slot * stride + (size_t)x * g.pplanes + g.poff[s] + r];
  const size_t r0 = ((size_t)gp * V + w.view) * nbins, r1 = ((size_t)gp * V + w.view + V / 2) * nbins;
  sino[r0 + x] = q.x;
  sino[r0 + xm] = q.y;
  sino[r1 + x] = q.z;
  sino[r1 + xm] = q.w;
}

__global__ void add_partials_kernel(long long n4, const float4 *__restrict__ a, const float4 *__restrict__ b,
                                    float4 *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n4) out[i] = a[i] + b[i];
}

template <typename T>
__global__ void scale_pairs_kernel(DevGeom g, const T *__restrict__ src, const int *__restrict__ views,
                                   float4 *__restrict__ dst, long long dst_pair_stride) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per = (long long)g.nquads * g.pplanes;
  if (i >= per) return;
  const int slot = blockIdx.y;
  const int pp = (int)(i % g.pplanes);
  const int s = g.pplane_seg[pp];
  const P4 m = load_p4(src, (size_t)views[slot] * per + i);
  float4 o = f4(0.f);
  if (s >= 0) {
    const float bs = g.bp_scale[s];
    o = make_float4(m.v[0] * bs, m.v[1] * bs, m.v[2] * bs, m.v[3] * bs);
  }
  dst[(size_t)slot * dst_pair_stride + i] = o;
}

// Launches a kernel that has `ctas` CTAs resident per SM by its registers; what
// their shared memory leaves of the SM's stays L1, which holds the sampling
// tables the projectors read (the whole SM's memory as shared memory instead:
// adjoint 1200 us a subset at span 9 against 1057, the back projector of that
// build 361 against 343).  The split goes with the launch, and the limit that
// belongs to the kernel itself is always the same: contexts of other sizes may
// launch it from other threads.
template <typename... P, typename... A>
cudaError_t launch_smem(void (*k)(P...), long long grid, int threads, size_t smem, int ctas, cudaStream_t st,
                        A... args) {
  constexpr size_t kSm = 228 * 1024, kReserved = 1024;        // of an SM; of a CTA
  constexpr size_t kMaxDynamic = kSm - kReserved - 512;       // less the kernels' static shared memory
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)std::max(smem, kMaxDynamic));
  if (e != cudaSuccess) return e;
  ctas = (int)std::max<size_t>(1, std::min<size_t>(ctas, kSm / (smem + kReserved)));
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  at.val.sharedMemCarveout = (unsigned)std::min<size_t>(100, (ctas * (smem + kReserved) * 100 + kSm - 1) / kSm);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

template <int MODE, int PL, typename PT, typename AT>
cudaError_t launch_fp_t(const DevGeom &g, const float *samples, const QuadWork *work, int nwork, const void *prompts,
                        const void *add, float *out, long long out_pair_stride, const FrameStrides &fr,
                        cudaStream_t st) {
  const int warps = g.nfptasks / 16 + 1;
  const int ZS = g.zp + kFpZPad;
  const size_t smem = (size_t)(2 * kFpSlots + 1) * ZS * sizeof(float4) + (size_t)kFpSlots * g.groupmax * sizeof(FpMid);
  return launch_smem(fp_kernel<MODE, PL, PT, AT>, (long long)nwork * fr.n, warps * 32, smem, std::max(1, 32 / warps),
                     st, g, reinterpret_cast<const float4 *>(samples), work, (const PT *)prompts, (const AT *)add,
                     reinterpret_cast<float4 *>(out), out_pair_stride / 4, fr);
}

template <int PL>
cudaError_t launch_fp_pl(const DevGeom &g, const float *samples, const QuadWork *work, int nwork, int mode,
                         const void *prompts, const void *add, int storage, float *out, long long stride,
                         const FrameStrides &fr, cudaStream_t st) {
  if (mode == 0)
    return launch_fp_t<0, PL, int16_t, float>(g, samples, work, nwork, nullptr, nullptr, out, stride, fr, st);
  if (storage == 0)
    return launch_fp_t<1, PL, int16_t, float>(g, samples, work, nwork, prompts, add, out, stride, fr, st);
  if (storage == 1)
    return launch_fp_t<1, PL, int16_t, __nv_bfloat16>(g, samples, work, nwork, prompts, add, out, stride, fr,
                                                      st);
  return launch_fp_t<1, PL, int16_t, __half>(g, samples, work, nwork, prompts, add, out, stride, fr, st);
}

}  // namespace

cudaError_t launch_fp(const DevGeom &g, const float *image, float *samples, const int *pair_views, int view0,
                      int npairs, const QuadWork *work, int nwork, int mode, const void *prompts, const void *add,
                      int storage, float *out, long long out_pair_stride, const FrameStrides &fr, cudaStream_t st) {
  if (nwork <= 0 || fr.n <= 0) return cudaSuccess;
  constexpr int T = kSampleTile;
  // the frames go in turns where they would exceed the grid's third dimension
  for (int f0 = 0, per = 65535 / (2 * npairs); f0 < fr.n; f0 += per) {
    FrameStrides part = fr;
    part.n = std::min(per, fr.n - f0);
    if (fr.map) part.map = fr.map + f0;
    // 16 rows a warp, fewer where that leaves less than eight CTAs an SM
    const int nx = (g.c + T - 1) / T, nz = 2 * npairs * part.n;
    int steps = 16;
    while (steps > 1 && (long long)nx * nz * (g.c / (T * steps) + 1) < 8 * 148) steps /= 2;
    fp_sample_kernel<<<dim3(nx, g.c / (T * steps) + 1, nz), T * T * 32, 0, st>>>(
        g, image + (fr.map ? 0 : (size_t)f0 * fr.image), pair_views, view0, npairs,
        reinterpret_cast<float4 *>(samples + (size_t)f0 * fr.samples), part, steps);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  auto f = g.fp_run == kFpRuns[0]   ? launch_fp_pl<kFpRuns[0]>
           : g.fp_run == kFpRuns[1] ? launch_fp_pl<kFpRuns[1]>
           : g.fp_run == kFpRuns[2] ? launch_fp_pl<kFpRuns[2]>
                                    : launch_fp_pl<kFpRuns[3]>;
  return f(g, samples, work, nwork, mode, prompts, add, storage, out, out_pair_stride, fr, st);
}

template <bool ACC, bool MULTI>
cudaError_t launch_bp_t(const DevGeom &g, const float *in, long long in_pair_stride, const QuadWork *work, int nquads,
                        float *bc, float *br, long long vol, const FrameStrides &fr, int view, int x0,
                        cudaStream_t st) {
  const size_t smem = (size_t)4 * g.bp_s4 * sizeof(float4);
  // launches that do not fill the chip share each quad among several CTAs
  const long long quads = (long long)nquads * fr.n;
  const int split = (int)std::max<long long>(1, std::min<long long>(4, (4 * 148 + quads - 1) / quads));
  return launch_smem(bp_kernel<ACC, MULTI>, quads * split, kBpThreads, smem, 2, st, g,
                     reinterpret_cast<const float4 *>(in), in_pair_stride / 4, work, bc, br, vol, fr, view, x0, split);
}

cudaError_t launch_bp(const DevGeom &g, const float *in, long long in_pair_stride, const QuadWork *work, int nwork,
                      float *bc, float *br, long long vol, const FrameStrides &fr, cudaStream_t st) {
  if (nwork <= 0 || fr.n <= 0) return cudaSuccess;
  auto f = fr.n > 1 ? launch_bp_t<false, true> : launch_bp_t<false, false>;
  return f(g, in, in_pair_stride, work, nwork, bc, br, vol, fr, 0, 0, st);
}

cudaError_t launch_adj(const DevGeom &g, const float *in, long long in_pair_stride, const QuadWork *work, int nwork,
                       float *bc, float *br, long long vol, const FrameStrides &fr, cudaStream_t st) {
  if (nwork <= 0 || fr.n <= 0) return cudaSuccess;
  const size_t smem = (size_t)g.bp_splanes * sizeof(float4);
  auto k = g.adj_ends ? adj_kernel<kAdjZ, true> : adj_kernel<kAdjZ, false>;
  return launch_smem(k, (long long)nwork * fr.n, 256, smem, 3, st, g, reinterpret_cast<const float4 *>(in),
                     in_pair_stride / 4, work, bc, br, vol, fr);
}

cudaError_t launch_adj_rotate(const DevGeom &g, const int *pair_views, int npairs, const float *bc, const float *br,
                              long long vol, float *image, float *nf_inv, float *out, int mode,
                              const FrameStrides &fr, cudaStream_t st) {
  if (fr.n <= 0) return cudaSuccess;
  if (mode != 0 && fr.n != 1) return cudaErrorInvalidValue;
  const long long cols = (mode == 2) ? (long long)g.nx * g.nx : (long long)g.fov_columns;
  if (npairs > g.adj_pairs || !g.adj_ent || !g.adj_cnt) return cudaErrorInvalidValue;
  const int threads = 256;
  {
    const long long m = cols * npairs;
    const unsigned cb = (unsigned)((m + threads - 1) / threads);
    if (mode == 2)
      adj_cover_kernel<2><<<cb, threads, 0, st>>>(g, pair_views, npairs);
    else
      adj_cover_kernel<0><<<cb, threads, 0, st>>>(g, pair_views, npairs);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  const long long n = cols * (g.zp / 4);
  const dim3 blocks((unsigned)((n + threads - 1) / threads), fr.n);
  if (mode == 0)
    adj_rotate_kernel<0><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, out, fr);
  else if (mode == 1)
    adj_rotate_kernel<1><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, out, fr);
  else
    adj_rotate_kernel<2><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, out, fr);
  return cudaGetLastError();
}

cudaError_t launch_bp_sum(const DevGeom &g, const float *quad, int view, int x0, int nquads, float *out,
                          cudaStream_t st) {
  if (nquads <= 0) return cudaSuccess;
  return launch_bp_t<true, false>(g, quad, 0, nullptr, nquads, out, nullptr, 0, one_frame(), view, x0, st);
}

cudaError_t launch_rotback(const DevGeom &g, const int *pair_views, int npairs, const float *bc, const float *br,
                           long long vol, float *image, float *nf_inv, float *corr_out, int mode,
                           const FrameStrides &fr, cudaStream_t st) {
  if (fr.n <= 0) return cudaSuccess;
  if (mode != 0 && fr.n != 1) return cudaErrorInvalidValue;
  const long long n = (long long)g.fov_columns * (g.zp / 4);
  const int threads = 256;
  const dim3 blocks((unsigned)((n + threads - 1) / threads), fr.n);
  if (mode == 0)
    rotback_kernel<0><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, corr_out, fr);
  else if (mode == 1)
    rotback_kernel<1><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, corr_out, fr);
  else if (mode == 2)
    rotback_kernel<2><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, corr_out, fr);
  else
    rotback_kernel<3><<<blocks, threads, 0, st>>>(g, pair_views, npairs, bc, br, vol, image, nf_inv, corr_out, fr);
  return cudaGetLastError();
}

cudaError_t launch_rotpos(const DevGeom &g, float2 *rotpos, const int *row_start, cudaStream_t st) {
  dim3 grid((g.nx + 127) / 128, g.nviews / 2);
  rotpos_kernel<<<grid, 128, 0, st>>>(g, rotpos, row_start);
  return cudaGetLastError();
}

cudaError_t launch_prep(const DevGeom &g, int nbins, const int16_t *prompts, const float *randoms, const float *norm,
                        const float *atten, const float *scatter, int npskip, float eps2, int storage, void *q_prompts,
                        void *q_add, void *q_mult, int *quad_mask_accum, int plane0, int nplanes,
                        cudaStream_t st) {
  const int ppt = 16;
  dim3 grid((g.nquads + 127) / 128, (nplanes + ppt - 1) / ppt, g.nviews / 2);
  const long long sp = (long long)g.nviews * nbins, sh = (long long)(g.nviews / 2) * nbins;
  if (storage == 0)
    prep_kernel<int16_t, float><<<grid, 128, 0, st>>>(g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2,
                                                      (int16_t *)q_prompts, (float *)q_add, (float *)q_mult,
                                                      quad_mask_accum, ppt, plane0, nplanes, nullptr, sp, sh, 0, 0, 0);
  else if (storage == 1)
    prep_kernel<int16_t, __nv_bfloat16><<<grid, 128, 0, st>>>(
        g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2, (int16_t *)q_prompts, (__nv_bfloat16 *)q_add,
        (__nv_bfloat16 *)q_mult, quad_mask_accum, ppt, plane0, nplanes, nullptr, sp, sh, 0, 0, 0);
  else
    prep_kernel<int16_t, __half><<<grid, 128, 0, st>>>(
        g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2, (int16_t *)q_prompts, (__half *)q_add,
        (__half *)q_mult, quad_mask_accum, ppt, plane0, nplanes, nullptr, sp, sh, 0, 0, 0);
  return cudaGetLastError();
}

// SaveImage's layout (drv:4020-4043): out[z][y][x] = image[x][y][z] on FOV
// columns, planes < nz; zero elsewhere.  One thread per (z, y, x), x fastest.
__global__ void image_zyx_kernel(DevGeom g, const float *__restrict__ image, float *__restrict__ out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)g.nz * g.nx * g.nx;
  if (t >= n) return;
  const int x = (int)(t % g.nx), y = (int)((t / g.nx) % g.nx), z = (int)(t / ((long long)g.nx * g.nx));
  const bool in = y >= g.cyl0[x] && y < g.cyl1[x];
  out[t] = in ? __ldg(image + ((size_t)x * g.nx + y) * g.zp + z) : 0.f;
}

cudaError_t launch_image_zyx(const DevGeom &g, const float *image, float *out, cudaStream_t st) {
  const long long n = (long long)g.nz * g.nx * g.nx;
  image_zyx_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, image, out);
  return cudaGetLastError();
}

cudaError_t launch_prep_pairs(const DevGeom &g, int nbins, const int16_t *prompts, const float *randoms,
                              const float *norm, const float *atten, const float *scatter, int npskip, float eps2,
                              int storage, void *q_prompts, void *q_add, void *q_mult, int *quad_mask_accum,
                              const int *pair_views, int npairs, cudaStream_t st, bool flat_prompts) {
  const int ppt = 16;
  dim3 grid((g.nquads + 127) / 128, (g.segmentsize + ppt - 1) / ppt, npairs);
  const long long P = g.segmentsize, sp = nbins, sh = P * nbins, ss = 2 * P * nbins;
  const long long fp = flat_prompts ? (long long)g.nviews * nbins : 0, fh = (long long)(g.nviews / 2) * nbins;
  if (storage == 0)
    prep_kernel<int16_t, float><<<grid, 128, 0, st>>>(g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2,
                                                      (int16_t *)q_prompts, (float *)q_add, (float *)q_mult,
                                                      quad_mask_accum, ppt, 0, g.segmentsize, pair_views, sp, sh, ss, fp, fh);
  else if (storage == 1)
    prep_kernel<int16_t, __nv_bfloat16><<<grid, 128, 0, st>>>(
        g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2, (int16_t *)q_prompts, (__nv_bfloat16 *)q_add,
        (__nv_bfloat16 *)q_mult, quad_mask_accum, ppt, 0, g.segmentsize, pair_views, sp, sh, ss, fp, fh);
  else
    prep_kernel<int16_t, __half><<<grid, 128, 0, st>>>(
        g, nbins, prompts, randoms, norm, atten, scatter, npskip, eps2, (int16_t *)q_prompts, (__half *)q_add,
        (__half *)q_mult, quad_mask_accum, ppt, 0, g.segmentsize, pair_views, sp, sh, ss, fp, fh);
  return cudaGetLastError();
}

cudaError_t launch_scale_pairs(const DevGeom &g, const void *src, int storage, const int *views, int npairs,
                               float *dst, long long dst_pair_stride, cudaStream_t st) {
  const long long per = (long long)g.nquads * g.pplanes;
  dim3 grid((unsigned)((per + 255) / 256), npairs);
  if (storage == 0)
    scale_pairs_kernel<float><<<grid, 256, 0, st>>>(g, (const float *)src, views, reinterpret_cast<float4 *>(dst),
                                                    dst_pair_stride / 4);
  else if (storage == 1)
    scale_pairs_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(g, (const __nv_bfloat16 *)src, views,
                                                            reinterpret_cast<float4 *>(dst), dst_pair_stride / 4);
  else
    scale_pairs_kernel<__half><<<grid, 256, 0, st>>>(g, (const __half *)src, views, reinterpret_cast<float4 *>(dst),
                                                     dst_pair_stride / 4);
  return cudaGetLastError();
}

cudaError_t launch_finish_mask(const DevGeom &g, const int *accum, int16_t *nzmask, cudaStream_t st) {
  const int n = (g.nviews / 2) * g.nquads;
  finish_mask_kernel<<<(n + 255) / 256, 256, 0, st>>>(g, accum, nzmask);
  return cudaGetLastError();
}

cudaError_t launch_init_image(const DevGeom &g, float *image, cudaStream_t st) {
  const long long n = (long long)g.nx * g.nx * g.zp;
  init_image_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, image);
  return cudaGetLastError();
}

cudaError_t launch_post_iteration(const DevGeom &g, float *image, double *partial, double *sum,
                                  const FrameStrides &fr, cudaStream_t st) {
  if (fr.n <= 0) return cudaSuccess;
  const long long n = (long long)g.fov_columns * (g.z_max - g.z_min);
  const int blocks = (int)((n + 255) / 256);
  if (fr.n > 1 && fr.partial < blocks) return cudaErrorInvalidValue;
  post_iter_kernel<<<dim3(blocks, fr.n), 256, 0, st>>>(g, image, partial, fr);
  sum_partials_kernel<<<fr.n, 1024, 0, st>>>(partial, blocks, sum, fr.partial, fr.map);
  return cudaGetLastError();
}

int post_iteration_blocks(const DevGeom &g) {
  const long long n = (long long)g.fov_columns * (g.z_max - g.z_min);
  return (int)((n + 255) / 256);
}

cudaError_t launch_rows_to_quad(const DevGeom &g, int nbins, const float *rows, float *quad, int apply_bp_scale,
                                cudaStream_t st) {
  dim3 grid((g.nquads + 127) / 128, g.segmentsize);
  rows_to_quad_kernel<<<grid, 128, 0, st>>>(g, nbins, rows, reinterpret_cast<float4 *>(quad), apply_bp_scale);
  return cudaGetLastError();
}

cudaError_t launch_quad_to_rows(const DevGeom &g, int nbins, const float *quad, const QuadWork *work, int nwork,
                                float *rows, cudaStream_t st) {
  if (nwork <= 0) return cudaSuccess;
  dim3 grid((g.segmentsize + 255) / 256, nwork);
  quad_to_rows_kernel<<<grid, 256, 0, st>>>(g, nbins, reinterpret_cast<const float4 *>(quad), work, rows);
  return cudaGetLastError();
}

cudaError_t launch_quad_to_file(const DevGeom &g, int nbins, const float *quad, long long quad_pair_stride,
                                const QuadWork *work, int nwork, float *sino, cudaStream_t st) {
  if (nwork <= 0) return cudaSuccess;
  dim3 grid((g.segmentsize + 255) / 256, nwork);
  quad_to_file_kernel<<<grid, 256, 0, st>>>(g, nbins, reinterpret_cast<const float4 *>(quad), quad_pair_stride / 4,
                                            work, sino);
  return cudaGetLastError();
}

cudaError_t launch_add_partials(const DevGeom &g, const float *bc, const float *br, float *out, cudaStream_t st) {
  const long long n4 = (long long)g.nx * g.nx * g.zp / 4;
  add_partials_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(n4, reinterpret_cast<const float4 *>(bc),
                                                                     reinterpret_cast<const float4 *>(br),
                                                                     reinterpret_cast<float4 *>(out));
  return cudaGetLastError();
}

// ============================================================================
// PSF resolution modelling (psf.cpp), on the FOV columns of [x][y][zp] images.
// psf_x_kernel is convolvex (psf.cpp:163-206): taps mask in [-h, h) of the
// x kernel over the x positions inside the FOV of row y, the result divided
// by the sum of the taps used unless that sum is 0 or 1.  psf_yz_kernel is
// convolveyz (psf.cpp:350-460): the same along y (its tap sum kept, not
// applied), then along z over the planes [z_min, z_max) -- with the y
// kernel's taps, as the reference's loop reads them -- scaled by
// norm_z[z] / (y tap sum), norm_z the inverse of the z kernel taps that fall
// inside [z_min, z_max) (host-computed).  Sums in tap order, unfused.
// Up to kPsfMaxH taps a side, a CTA takes kPsfRun columns along the pass's
// direction and a thread one plane of each, from a window of kPsfRun + 2H - 1
// inputs in registers; an input outside the FOV reads as 0, whose product adds
// nothing.  (Measured on B200, HRRT span-9 volume, 13 taps: one CTA per column
// with a load and a test per tap took 134 + 174 us, these 53 + 64 us.)  Longer
// filters run one CTA per FOV column, one thread per plane.
// ============================================================================
constexpr int kPsfRun = 8, kPsfMaxH = 8;

template <int H>
__global__ void __launch_bounds__(256) psf_x_run_kernel(DevGeom g, const float *__restrict__ in,
                                                        float *__restrict__ out, const float *__restrict__ filt) {
  const int y = blockIdx.y, z = threadIdx.x, N = g.nx, zp = g.zp;
  const int lo = g.cyl0[y], hi = g.cyl1[y], x0 = lo + blockIdx.x * kPsfRun;
  if (x0 >= hi || z >= zp) return;
  float c[2 * H], w[kPsfRun + 2 * H - 1];
#pragma unroll
  for (int m = 0; m < 2 * H; m++) c[m] = __ldg(filt + m);
#pragma unroll
  for (int k = 0; k < kPsfRun + 2 * H - 1; k++) {
    const int x2 = x0 - H + k;
    w[k] = (x2 >= lo && x2 < hi) ? __ldg(in + ((size_t)x2 * N + y) * zp + z) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kPsfRun; i++) {
    const int x = x0 + i;
    if (x >= hi) break;
    float acc = 0.f, norm = 0.f;
#pragma unroll
    for (int m = 0; m < 2 * H; m++) {
      const int x2 = x - H + m;
      norm = norm + ((x2 >= lo && x2 < hi) ? c[m] : 0.f);
      acc = acc + w[i + m] * c[m];
    }
    if (norm != 1.0f && norm != 0.0f) acc = acc * (1.0f / norm);
    out[((size_t)x * N + y) * zp + z] = acc;
  }
}

template <int H>
__global__ void __launch_bounds__(256) psf_yz_run_kernel(DevGeom g, const float *__restrict__ in,
                                                         float *__restrict__ out, const float *__restrict__ filt,
                                                         const float *__restrict__ normz) {
  extern __shared__ float col[];  // [kPsfRun][H + zp + H]: the y-convolved columns, 0 outside [z_min, z_max)
  const int x = blockIdx.y, z = threadIdx.x, N = g.nx, zp = g.zp, W = zp + 2 * H;
  const int lo = g.cyl0[x], hi = g.cyl1[x], y0 = lo + blockIdx.x * kPsfRun;
  if (y0 >= hi) return;
  for (int i = z; i < kPsfRun * 2 * H; i += blockDim.x) {
    const int k = i % (2 * H);
    col[(i / (2 * H)) * W + (k < H ? k : zp + k)] = 0.f;
  }
  float c[2 * H], norms[kPsfRun];
#pragma unroll
  for (int m = 0; m < 2 * H; m++) c[m] = __ldg(filt + m);
  if (z < zp) {
    float w[kPsfRun + 2 * H - 1];
    const float *src = in + (size_t)x * N * zp + z;
#pragma unroll
    for (int k = 0; k < kPsfRun + 2 * H - 1; k++) {
      const int y2 = y0 - H + k;
      w[k] = (y2 >= lo && y2 < hi) ? __ldg(src + (size_t)y2 * zp) : 0.f;
    }
    const bool inside = z >= g.z_min && z < g.z_max;
#pragma unroll
    for (int i = 0; i < kPsfRun; i++) {
      float acc = 0.f, norm = 0.f;
#pragma unroll
      for (int m = 0; m < 2 * H; m++) {
        const int y2 = y0 + i - H + m;
        norm = norm + ((y2 >= lo && y2 < hi) ? c[m] : 0.f);
        acc = acc + w[i + m] * c[m];
      }
      norms[i] = norm;
      col[i * W + H + z] = inside ? acc : 0.f;
    }
  }
  __syncthreads();
  if (z >= zp) return;
  const float nz = __ldg(normz + z);
#pragma unroll
  for (int i = 0; i < kPsfRun; i++) {
    if (y0 + i >= hi) break;
    float o = 0.f;
    if (norms[i] != 0.0f) {
      if (z < g.nz) {
#pragma unroll
        for (int m = 0; m < 2 * H; m++) o = o + col[i * W + z + m] * c[m];
      }
      o = o * (nz * (1.0f / norms[i]));
    }
    out[((size_t)x * N + y0 + i) * zp + z] = o;
  }
}

__global__ void psf_x_kernel(DevGeom g, const float *__restrict__ in, float *__restrict__ out,
                             const float *__restrict__ filt, int h) {
  const int col = blockIdx.x, z = threadIdx.x;
  if (z >= g.zp) return;
  const short2 xy = g.fov_xy[col];
  const int x = xy.x, y = xy.y, N = g.nx;
  const int lo = g.cyl0[y], hi = g.cyl1[y];
  float acc = 0.f, norm = 0.f;
  for (int mask = -h; mask < h; mask++) {
    const int x2 = x + mask;
    if (x2 < lo || x2 >= hi) continue;
    const float c = __ldg(filt + mask + h);
    norm = norm + c;
    acc = acc + __ldg(in + ((size_t)x2 * N + y) * g.zp + z) * c;
  }
  if (norm != 1.0f && norm != 0.0f) acc = acc * (1.0f / norm);
  out[((size_t)x * N + y) * g.zp + z] = acc;
}

__global__ void psf_yz_kernel(DevGeom g, const float *__restrict__ in, float *__restrict__ out,
                              const float *__restrict__ filty, int h, const float *__restrict__ normz) {
  extern __shared__ float col[];  // [zp] the y-convolved column
  const int c = blockIdx.x, z = threadIdx.x;
  const short2 xy = g.fov_xy[c];
  const int x = xy.x, y = xy.y, N = g.nx, zp = g.zp;
  const int lo = g.cyl0[x], hi = g.cyl1[x];
  float acc = 0.f, norm = 0.f;
  for (int mask = -h; mask < h; mask++) {
    const int y2 = y + mask;
    if (y2 < lo || y2 >= hi) continue;
    const float f = __ldg(filty + mask + h);
    norm = norm + f;
    if (z < zp) acc = acc + __ldg(in + ((size_t)x * N + y2) * zp + z) * f;
  }
  if (z < zp) col[z] = acc;
  __syncthreads();
  if (z >= zp) return;
  float o = 0.f;
  if (norm != 0.0f) {
    for (int mask = -h; mask < h; mask++) {
      const int z2 = z + mask;
      if (z2 < g.z_min || z2 >= g.z_max || z >= g.nz) continue;
      o = o + col[z2] * __ldg(filty + mask + h);
    }
    o = o * (__ldg(normz + z) * (1.0f / norm));
  }
  out[((size_t)x * N + y) * zp + z] = o;
}

// The consumers of the correction image once it is a separate volume (the
// PSF path): MODE 0 the OSEM update, MODE 1 the inverse sensitivity; the
// arithmetic of rotback_kernel's modes 0 and 1.  MODE 2: the MAP update of
// pt_cal_updateimage_mapem (je_hrrt_osem3d/hrrt_osem3d.cpp:2031-2073),
// image = min(image_max, image * min(100, max(0.1, corr / (beta * dpf + 1 / nf_inv))))
// with SSE's min/max rule; the reference's _mm_rcp_ps approximation of
// 1 / nf_inv (relative error up to 1.5 * 2^-12) is the exact reciprocal here.
template <int MODE>
__global__ void __launch_bounds__(256) apply_corr_kernel(DevGeom g, const float *__restrict__ corr,
                                                         float *__restrict__ image, float *__restrict__ nf_inv,
                                                         const float *__restrict__ dpf, float beta) {
  const int nq = g.zp / 4;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int col = (int)(t / nq), q = (int)(t - (long long)col * nq);
  if (col >= g.fov_columns) return;
  const short2 xy = g.fov_xy[col];
  const size_t o = ((size_t)xy.x * g.nx + xy.y) * nq + q;
  const float4 acc = reinterpret_cast<const float4 *>(corr)[o];
  if (MODE == 0) {
    float4 *im = reinterpret_cast<float4 *>(image);
    const float4 nf = reinterpret_cast<const float4 *>(nf_inv)[o];
    float4 iv = im[o];
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, b[4] = {iv.x, iv.y, iv.z, iv.w}, n[4] = {nf.x, nf.y, nf.z, nf.w};
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const float lo = (0.01f > a[l]) ? 0.01f : a[l];
      const float cl = (100.0f < lo) ? 100.0f : lo;
      const float u = b[l] * (cl * n[l]);
      b[l] = (g.image_max < u) ? g.image_max : u;
    }
    im[o] = make_float4(b[0], b[1], b[2], b[3]);
  } else if (MODE == 2) {
    float4 *im = reinterpret_cast<float4 *>(image);
    const float4 nf = reinterpret_cast<const float4 *>(nf_inv)[o];
    const float4 dp = reinterpret_cast<const float4 *>(dpf)[o];
    float4 iv = im[o];
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, b[4] = {iv.x, iv.y, iv.z, iv.w}, n[4] = {nf.x, nf.y, nf.z, nf.w},
          d[4] = {dp.x, dp.y, dp.z, dp.w};
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const float den = __fadd_rn(__fmul_rn(beta, d[l]), __frcp_rn(n[l]));
      const float q = __fdiv_rn(a[l], den);
      const float lo = (0.1f > q) ? 0.1f : q;
      const float cl = (100.0f < lo) ? 100.0f : lo;
      const float u = __fmul_rn(b[l], cl);
      b[l] = (g.image_max < u) ? g.image_max : u;
    }
    im[o] = make_float4(b[0], b[1], b[2], b[3]);
  } else {
    float a[4] = {acc.x, acc.y, acc.z, acc.w}, r[4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const int z = q * 4 + l;
      r[l] = (z < g.nz && fabsf(a[l]) > g.eps1) ? (1.0f / a[l]) : 0.f;
    }
    reinterpret_cast<float4 *>(nf_inv)[o] = make_float4(r[0], r[1], r[2], r[3]);
  }
}

template <int H>
cudaError_t launch_psf_run(const DevGeom &g, const float *in, float *tmp, float *out, const float *filt_x,
                           const float *filt_y, const float *normz, cudaStream_t st) {
  const int threads = ((g.zp + 31) / 32) * 32;
  const dim3 grid((g.nx + kPsfRun - 1) / kPsfRun, g.nx);
  psf_x_run_kernel<H><<<grid, threads, 0, st>>>(g, in, tmp, filt_x);
  psf_yz_run_kernel<H><<<grid, threads, kPsfRun * (g.zp + 2 * H) * sizeof(float), st>>>(g, tmp, out, filt_y, normz);
  return cudaGetLastError();
}

cudaError_t launch_psf(const DevGeom &g, const float *in, float *tmp, float *out, const float *filt_x, int hx,
                       const float *filt_y, int hy, const float *normz, cudaStream_t st) {
  const int threads = ((g.zp + 31) / 32) * 32;
  if (hx == hy && threads <= 256) {
    switch (hx) {
      case 1: return launch_psf_run<1>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 2: return launch_psf_run<2>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 3: return launch_psf_run<3>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 4: return launch_psf_run<4>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 5: return launch_psf_run<5>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 6: return launch_psf_run<6>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case 7: return launch_psf_run<7>(g, in, tmp, out, filt_x, filt_y, normz, st);
      case kPsfMaxH: return launch_psf_run<kPsfMaxH>(g, in, tmp, out, filt_x, filt_y, normz, st);
      default: break;
    }
  }
  psf_x_kernel<<<g.fov_columns, threads, 0, st>>>(g, in, tmp, filt_x, hx);
  psf_yz_kernel<<<g.fov_columns, threads, g.zp * sizeof(float), st>>>(g, tmp, out, filt_y, hy, normz);
  return cudaGetLastError();
}

// ============================================================================
// MAP, technique 1 of je_hrrt_osem3d (-b 1,beta): Green's one-step-late
// prior.  calculate_DPF_image (je_hrrt_osem3d/dpfcalc.c:23-31, :66-85,
// :266-300) and the update pt_cal_updateimage_mapem (hrrt_osem3d.cpp:
// 2031-2073).
//   map_max_kernel : the image maximum over the FOV columns and planes
//                    [0, nz), never below 0 (the float's bits, an unsigned
//                    maximum, order like the values for non-negative floats);
//   map_dpf_kernel : one thread per FOV voxel: delta = (1.2 max) / 20 and,
//                    for 1 <= x < nx-1 and 1 <= z < nz-1, the 6 face and
//                    (times sqrt(0.5)) 12 edge terms tanh((c - n) / delta) =
//                    (e - 1) / (e + 1), e = exp(2 (c - n) / delta), summed in
//                    the source's order in float, combined in double; 0
//                    elsewhere.  e is exp() in double rounded to float, the
//                    correctly rounded value.
//   MAP update     : apply_corr_kernel<2>.
// ============================================================================
__global__ void __launch_bounds__(256) map_max_kernel(DevGeom g, const float *__restrict__ img,
                                                      unsigned int *__restrict__ mx) {
  // a warp takes a column at a time: one
  // atomic per warp of the grid, not per 32 voxels (200 -> 23 us)
  const int ln = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  unsigned int v = 0;
  for (int col = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); col < g.fov_columns; col += warps) {
    const short2 xy = g.fov_xy[col];
    const float *p = img + ((size_t)xy.x * g.nx + xy.y) * g.zp;
    for (int z = ln; z < g.nz; z += 32) {
      const float f = __ldg(p + z);
      if (f > 0.f) v = max(v, __float_as_uint(f));
    }
  }
  v = __reduce_max_sync(0xffffffffu, v);
  if (ln == 0 && v) atomicMax(mx, v);
}

__device__ __forceinline__ float map_tanh(float r, float delta) {
  const float e = __double2float_rn(exp((double)__fdiv_rn(__fmul_rn(2.0f, r), delta)));
  return __fdiv_rn(__fsub_rn(e, 1.0f), __fadd_rn(e, 1.0f));
}

__global__ void __launch_bounds__(256) map_dpf_kernel(DevGeom g, const float *__restrict__ img,
                                                      const unsigned int *__restrict__ mx, float *__restrict__ dpf) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)g.fov_columns * g.zp) return;
  const int col = (int)(t / g.zp), z = (int)(t - (long long)col * g.zp);
  const short2 xy = g.fov_xy[col];
  const int x = xy.x, y = xy.y, N = g.nx, zp = g.zp;
  float out = 0.f;
  if (x >= 1 && x < N - 1 && z >= 1 && z < g.nz - 1) {
    const float maxpet = __double2float_rn(1.2 * (double)__uint_as_float(*mx));
    const float delta = __double2float_rn((double)maxpet / 20.0);
    auto I = [&](int a, int b, int c) { return __ldg(img + ((size_t)a * N + b) * zp + c); };
    const float c = I(x, y, z);
    float a = map_tanh(__fsub_rn(c, I(x, y, z - 1)), delta);
    a = __fadd_rn(a, map_tanh(__fsub_rn(c, I(x, y, z + 1)), delta));
    a = __fadd_rn(a, map_tanh(__fsub_rn(c, I(x - 1, y, z)), delta));
    a = __fadd_rn(a, map_tanh(__fsub_rn(c, I(x + 1, y, z)), delta));
    a = __fadd_rn(a, map_tanh(__fsub_rn(c, I(x, y - 1, z)), delta));
    a = __fadd_rn(a, map_tanh(__fsub_rn(c, I(x, y + 1, z)), delta));
    float b = map_tanh(__fsub_rn(c, I(x - 1, y, z - 1)), delta);
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x, y - 1, z - 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x + 1, y, z - 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x, y + 1, z - 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x - 1, y - 1, z)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x - 1, y + 1, z)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x + 1, y - 1, z)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x + 1, y + 1, z)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x - 1, y, z + 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x, y - 1, z + 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x + 1, y, z + 1)), delta));
    b = __fadd_rn(b, map_tanh(__fsub_rn(c, I(x, y + 1, z + 1)), delta));
    out = __double2float_rn(__dadd_rn((double)a, __dmul_rn(0.70710678118654752440, (double)b)));
  }
  dpf[((size_t)x * N + y) * zp + z] = out;
}

cudaError_t launch_map_prior(const DevGeom &g, const float *image, unsigned int *mx, float *dpf, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(mx, 0, sizeof(unsigned int), st);
  if (e != cudaSuccess) return e;
  const long long n2 = (long long)g.fov_columns * g.zp;
  const int max_blocks = std::min(4 * 148, (g.fov_columns + 7) / 8);
  map_max_kernel<<<max_blocks, 256, 0, st>>>(g, image, mx);
  map_dpf_kernel<<<(unsigned)((n2 + 255) / 256), 256, 0, st>>>(g, image, mx, dpf);
  return cudaGetLastError();
}

cudaError_t launch_apply_corr(const DevGeom &g, const float *corr, float *image, float *nf_inv, int mode,
                              cudaStream_t st, const float *dpf, float beta) {
  const long long n = (long long)g.fov_columns * (g.zp / 4);
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (mode == 0)
    apply_corr_kernel<0><<<blocks, 256, 0, st>>>(g, corr, image, nf_inv, nullptr, 0.f);
  else if (mode == 1)
    apply_corr_kernel<1><<<blocks, 256, 0, st>>>(g, corr, image, nf_inv, nullptr, 0.f);
  else
    apply_corr_kernel<2><<<blocks, 256, 0, st>>>(g, corr, image, nf_inv, dpf, beta);
  return cudaGetLastError();
}

}  // namespace hrrt
