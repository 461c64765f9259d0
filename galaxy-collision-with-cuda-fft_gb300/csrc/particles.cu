// Particle <-> grid kernels of the PM force chain.
//
// Arithmetic follows the reference kernels in src/galaxy_collision/deposit.py
// and integrator.py operation by operation in f32 with explicit
// round-to-nearest intrinsics (no FMA contraction), so the CPU restatement can
// reproduce them bit for bit. The deposit accumulates the reference's per-corner
// contributions m*wx*wy*wz into an int64 fixed-point grid: the partial product
// (m/dx^3*wx)*wy is rounded to f32 as the reference rounds it, and its exact
// product with wz is rounded once to the nearest quantum (one fused
// multiply-add). Integer addition is associative, so the density is
// bit-identical whatever the particle order or atomic interleaving.
#include "common.cuh"
#include "umma.cuh"

#include <math.h>

#include <cmath>
#include <cstdint>

// ------------------------------------------------------------------------------
// fixed-point set-up: total density-mass and quantum exponent
// ------------------------------------------------------------------------------
// The quantum must not depend on the particle order (sorting permutes the
// particles), so the total S = sum m/dx^3 is formed exactly: every positive
// finite term is truncated to an integer multiple of 2^-s, with s chosen from
// the largest term (an order-independent maximum) so that the integer sum of
// all n terms stays below 2^62, and the integers are summed exactly.
__global__ void __launch_bounds__(256) k_mass_max(const float *__restrict__ m, long long n, float inv_vol,
                                                  unsigned *__restrict__ maxbits) {
  gc_after();
  unsigned best = 0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const float mm = __fmul_rn(m[p], inv_vol);
    if (isfinite(mm) && mm > 0.0f) best = max(best, __float_as_uint(mm));
  }
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31) == 0 && best) atomicMax(maxbits, best);
}

__device__ __forceinline__ int mass_shift(unsigned maxbits, int log2n) {
  const int emax = (int)((maxbits >> 23) & 0xffu) - 127;  // max term < 2^(emax+1)
  return 62 - log2n - (emax + 1);
}

__global__ void __launch_bounds__(256) k_mass_isum(const float *__restrict__ m, long long n, float inv_vol,
                                                   const unsigned *__restrict__ maxbits, int log2n,
                                                   unsigned long long *__restrict__ isum) {
  gc_after();
  const int s = mass_shift(*maxbits, log2n);
  unsigned long long acc = 0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const float mm = __fmul_rn(m[p], inv_vol);
    if (isfinite(mm) && mm > 0.0f) {  // floor(mm * 2^s) from the float bits (no FP64)
      const unsigned u = __float_as_uint(mm);
      int ex = (int)((u >> 23) & 0xffu);
      const unsigned long long mant = (u & 0x7fffffu) | (ex ? 0x800000u : 0u);
      if (ex == 0) ex = 1;
      const int e2 = ex - 150 + s;
      acc += e2 >= 0 ? (mant << e2) : (e2 > -64 ? (mant >> -e2) : 0ull);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(isum, acc);
}

// E = exponent(S) - bits so that the whole mass is at most 2^bits quanta.
__global__ void k_qexp(const unsigned *__restrict__ maxbits, const unsigned long long *__restrict__ isum, int log2n,
                       double *__restrict__ small, int mass_slot, int exp_slot, int bits) {
  gc_after();
  if (threadIdx.x != 0) return;
  double S = 0.0;
  if (*maxbits) S = ldexp((double)(*isum), -mass_shift(*maxbits, log2n));
  int ex = 0;
  if (S > 0.0) frexp(S, &ex);  // S = f * 2^ex, f in [0.5, 1)
  int E = ex - bits;
  if (E < -120) E = -120;      // keep 2^-E a normal f32
  if (E > 120) E = 120;
  small[mass_slot] = S;
  small[exp_slot] = (double)E;
}

// Quanta of the mean particle, 1 to 2 times this; where it lies between 2^20 and 2^22 and
// the particles are many, their masses decide which pass of the deposit takes them (see
// gc_deposit_q).
#define HEAVY_MIN (1 << 20)
static double mean_quanta(int bits, int64_t n) { return std::ldexp(1.0, bits - 1) / (double)n; }
static bool quanta_undecided(int bits, int64_t n) {
  const double q = mean_quanta(bits, n);
  return n >= HEAVY_MIN && q >= 1048576.0 && q < 4194304.0;
}

// Whether at least 1/32 of 1024 masses, spread over the array, reach 2^22 quanta.
__global__ void __launch_bounds__(1024)
    k_mass_heavy(const float *__restrict__ m, long long n, float inv_vol, const double *__restrict__ qexp,
                 int *__restrict__ heavy) {
  gc_after();
  const float mm = __fmul_rn(__ldg(m + (n - 1) * (long long)threadIdx.x / 1023), inv_vol);
  const int c = __syncthreads_count(!(fabsf(__fmul_rn(mm, ldexpf(1.0f, -(int)*qexp))) < 4194304.0f));
  if (threadIdx.x == 0) *heavy = c >= 32;
}

static int ceil_log2(long long n) {
  int L = 0;
  while ((1LL << L) < n) ++L;
  return L;
}

int gc_fixed_point_setup(gc_ctx *ctx, const float *m, int64_t n, int bits, int mass_slot, int exp_slot) {
  const float dxf = (float)ctx->dx;
  const float inv_vol = 1.0f / ((dxf * dxf) * dxf);
  // two integer scratch words live in the reduction buffer
  int s = gc_ensure_red(ctx, 4);
  if (s) return s;
  unsigned *maxbits = (unsigned *)ctx->red;
  unsigned long long *isum = (unsigned long long *)(ctx->red + 1);
  GC_CUDA(ctx, cudaMemsetAsync(ctx->red, 0, 2 * sizeof(double), ctx->stream));
  unsigned nb = gc_blocks(n, 256);
  if (nb > gc_sms() * 8u) nb = gc_sms() * 8u;
  const int L = ceil_log2((long long)n);
  gc_launch_after(ctx, GK_MASS, k_mass_max, dim3(nb), dim3(256), 0, m, (long long)n, inv_vol, maxbits);
  gc_launch_after(ctx, GK_MASS, k_mass_isum, dim3(nb), dim3(256), 0, m, (long long)n, inv_vol, maxbits, L, isum);
  gc_launch_after(ctx, GK_MASS, k_qexp, dim3(1), dim3(32), 0, maxbits, isum, L, ctx->dsmall, mass_slot, exp_slot, bits);
  if (quanta_undecided(bits, n))
    gc_launch_after(ctx, GK_MASS, k_mass_heavy, dim3(1), dim3(1024), 0, m, (long long)n, inv_vol,
                    (const double *)(ctx->dsmall + exp_slot), reinterpret_cast<int *>(ctx->dsmall + exp_slot + 1));
  GC_LAUNCH_CHECK(ctx, "fixed-point set-up");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// deposit (deposit.py:47-82)
// ------------------------------------------------------------------------------
// RNE(a * b * 2^k) as an int64, for finite a, b and |a * b * 2^k| < 2^62: the
// product of the two 24-bit significands is exact in 64 bits, so the rounding
// is the single rounding of the exact product (integer ALUs only).
__device__ __forceinline__ long long prod_to_i64_rn(float a, float b, int k) {
  const unsigned ua = __float_as_uint(a), ub = __float_as_uint(b);
  int ea = (int)((ua >> 23) & 0xffu), eb = (int)((ub >> 23) & 0xffu);
  const unsigned long long ma = (ua & 0x7fffffu) | (ea ? 0x800000u : 0u);
  const unsigned long long mb = (ub & 0x7fffffu) | (eb ? 0x800000u : 0u);
  if (ea == 0) ea = 1;
  if (eb == 0) eb = 1;
  const unsigned long long prod = ma * mb;  // < 2^48
  const int sh = ea + eb - 300 + k;          // |a * b * 2^k| = prod * 2^sh
  long long r;
  if (sh >= 0) {
    r = (long long)(prod << sh);
  } else if (sh <= -49) {
    r = 0;  // below 1/2
  } else {
    const int rs = -sh;
    unsigned long long q = prod >> rs;
    const unsigned long long rem = prod & ((1ull << rs) - 1ull), half = 1ull << (rs - 1);
    if (rem > half || (rem == half && (q & 1ull))) q += 1ull;
    r = (long long)q;
  }
  return ((ua ^ ub) >> 31) ? -r : r;
}

// The exponent k of a power of two 2^k held in a normal f32.
__device__ __forceinline__ int pow2_exponent(float p) { return (int)((__float_as_uint(p) >> 23) & 0xffu) - 127; }

// Per-corner int64 contributions of one particle; corners outside the box are 0.
// Returns false when the particle deposits nothing.
__device__ __forceinline__ bool cic_contrib(float x, float y, float z, float mass, const DepCtx &d, float qscale,
                                            CellPos &c, long long (&q)[8]) {
  if (!gc_cell_of(x, y, z, d.dx, d.G, c)) return false;
  const float mm = __fmul_rn(mass, d.inv_vol);
  const int qk = pow2_exponent(qscale);
  const float wx[2] = {__fsub_rn(1.0f, c.fx), c.fx};
  const float wy[2] = {__fsub_rn(1.0f, c.fy), c.fy};
  const float wz[2] = {__fsub_rn(1.0f, c.fz), c.fz};
#pragma unroll
  for (int cx = 0; cx < 2; ++cx)
#pragma unroll
    for (int cy = 0; cy < 2; ++cy)
#pragma unroll
      for (int cz = 0; cz < 2; ++cz) {
        const int jx = c.ix + cx, jy = c.iy + cy, jz = c.iz + cz;
        const bool in = (unsigned)jx < (unsigned)d.G && (unsigned)jy < (unsigned)d.G && (unsigned)jz < (unsigned)d.G;
        const float b = __fmul_rn(__fmul_rn(mm, wx[cx]), wy[cy]);
        q[(cx * 2 + cy) * 2 + cz] = in ? prod_to_i64_rn(b, wz[cz], qk) : 0LL;
      }
  return true;
}

__device__ __forceinline__ void flush_corners(long long *__restrict__ qg, int ix, int iy, int iz, int G,
                                              const long long (&q)[8]) {
#pragma unroll
  for (int cx = 0; cx < 2; ++cx)
#pragma unroll
    for (int cy = 0; cy < 2; ++cy)
#pragma unroll
      for (int cz = 0; cz < 2; ++cz) {
        const long long v = q[(cx * 2 + cy) * 2 + cz];
        const int jx = ix + cx, jy = iy + cy, jz = iz + cz;
        if (v != 0 && (unsigned)jx < (unsigned)G && (unsigned)jy < (unsigned)G && (unsigned)jz < (unsigned)G) {
          const size_t idx = ((size_t)jx * G + jy) * G + jz;
          atomicAdd((unsigned long long *)(qg + idx), (unsigned long long)v);
        }
      }
}

// One particle per thread; when a whole warp shares one cell its 8 corner sums
// are reduced in registers and flushed by one lane.
__global__ void __launch_bounds__(256)
    k_deposit(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
              const float *__restrict__ m, long long n, DepCtx d, const double *__restrict__ qexp,
              long long *__restrict__ qg, unsigned *__restrict__ status) {
  const float qscale = ldexpf(1.0f, -(int)(*qexp));
  const int lane = threadIdx.x & 31;
  const long long warp0 = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31));
  const long long wstride = (long long)gridDim.x * blockDim.x;
  for (long long base = warp0; base < n; base += wstride) {
    const long long p = base + lane;
    CellPos c;
    long long q[8];
    bool ok = false;
    if (p < n) {
      const float px = x[p], py = y[p], pz = z[p];
      if (!gc_finite3(px, py, pz)) atomicOr(status, GC_FLAG_NONFINITE_POS);
      ok = cic_contrib(px, py, pz, m[p], d, qscale, c, q);
    }
    const unsigned key = ok ? (unsigned)(((c.ix + 1) * (d.G + 1) + (c.iy + 1)) * (d.G + 1) + (c.iz + 1))
                            : (0x80000000u | (unsigned)lane);
    int all_same = 0;
    __match_all_sync(0xffffffffu, key, &all_same);
    if (all_same) {
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        long long v = q[t];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        q[t] = v;
      }
      if (lane == 0) flush_corners(qg, c.ix, c.iy, c.iz, d.G, q);
    } else if (ok) {
      flush_corners(qg, c.ix, c.iy, c.iz, d.G, q);
    }
  }
}

// Cell-sorted particles, warp-contiguous. Lane L of warp w takes the particles
// t0 + 256 w + 32 j + L (j = 0..7) of the CTA's tile of 2048, so the 32
// particles a warp handles at once are adjacent in the array: after the cell
// sort they share one or two cells, and the particles that drifted into a
// neighbouring cell since the sort are scattered among them.
//
// Per particle the 8 corner contributions are the reference's products
// m/dx^3 * wx * wy * wz (deposit.py:69-82) scaled by the quantum (a power of
// two: exact) and rounded to the nearest integer (dep_corners: the last
// multiplication fused with the rounding, two corners per packed f32x2
// instruction). The bias of the rounding is subtracted in integer arithmetic,
// and the corner values are summed in int32, which is exact because every
// partial sum fits.
//
// Into the shared-memory box (below) the warp keeps a run cell (dep_warp_runs):
// lanes in it add their corners in registers, and the run is reduced across the
// warp with one redux.sync per corner when the warp leaves the cell. Lanes in any
// other cell (drifted particles) add their own corners. A redux.sync over the full
// warp costs the same whatever the keys, unlike one per group of equal keys,
// which serialises over the groups. (dep_warp_pass, of the particle pass that
// deposits too, reduces the cells of lane 0 and lane 31 instead.)
//
// Each warp owns an int32 box of nodes in shared memory (no block-wide
// barriers: warps never wait for each other). Corners go to it when the cells
// of the warp's 256 particles fit the box (it is the cell range of
// their coordinate range: x/dx is monotone) and their total quanta bound every
// node below 2^31; the box is added to the int64 grid with one atomic per
// nonzero node when the warp moves on. Otherwise every lane's corners go to the
// grid directly (dep_warp_direct). Particles whose contribution reaches 2^22 quanta (point masses) are
// deposited out of line at the end of the tile with the general int64
// rounding. Correct for any particle order;
// the sort makes it fast.
//
// WIDE is the same pass for fine quanta, where ordinary particles reach 2^22 of
// them (2^52 quanta in all, the default, below 2^30 particles): a corner value
// up to 2^41 quanta is split as h 2^20 + l with |l| <= 2^19 by two fused
// multiply-adds (dep_corners_wide), and h and l are summed separately in
// int32, each with its own half of the box. One particle per thread went to the
// grid with eight int64 atomics before. Measured, 1.5M particles sorted on a
// 100^3 grid at 2^-52 of the mass: 327 us before, 21 us now.
#define DEP_NONE 0xffffffffu
#define DEP_PER 8
#define DEP_WTILE (32 * DEP_PER)  // particles of one warp
template <bool WIDE>
struct DepW {
  static constexpr int box = WIDE ? 768 : 1024;         // nodes of one warp's box
  static constexpr float limit = WIDE ? 2199023255552.0f : 4194304.0f;  // 2^41, 2^22: largest quanta in the pass
  static constexpr int words = WIDE ? 2 * box : box;    // shared memory of a warp (int32)
};
static_assert(DepW<false>::box <= 1024 && DepW<true>::box <= 1024,
              "the box flush's reciprocal quotients are exact below 2^10 nodes");
#define DEP_BIAS 0x4B400000u
#define DEP_BIAS_H 0x55400000u  // the bits of 1.5 * 2^43

// Packed f32x2 arithmetic (two lanes of a 64-bit register, IEEE round to
// nearest per lane).
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 A, B, D;\n\tmov.b64 A, {%2, %3};\n\tmov.b64 B, {%4, %5};\n\t"
      "mul.rn.f32x2 D, A, B;\n\tmov.b64 {%0, %1}, D;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 A, B, C, D;\n\tmov.b64 A, {%2, %3};\n\tmov.b64 B, {%4, %5};\n\tmov.b64 C, {%6, %7};\n\t"
      "fma.rn.f32x2 D, A, B, C;\n\tmov.b64 {%0, %1}, D;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// The 8 corner values of a particle of s quanta (|s| < 2^22) with weights
// (wx0, fx), (wy0, fy), (wz0, fz), as the bits of 1.5 * 2^23 + RNE(b * wz)
// (corner order (cx, cy, cz)): the partial products a = s*wx and b = a*wy are
// rounded to f32, and b * wz + 1.5 * 2^23 is one fused multiply-add, whose single
// rounding (spacing 1 in [2^23, 2^24)) is the rounding of the exact product to
// the nearest integer. Two corners per packed instruction.
__device__ __forceinline__ void dep_corners(float s, float wx0, float fx, float wy0, float fy, float wz0, float fz,
                                            unsigned (&r)[8]) {
  const float2 a = f2_mul(make_float2(s, s), make_float2(wx0, fx));
  const float2 wy = make_float2(wy0, fy), wz = make_float2(wz0, fz), M = make_float2(12582912.0f, 12582912.0f);
  const float2 b0 = f2_mul(make_float2(a.x, a.x), wy), b1 = f2_mul(make_float2(a.y, a.y), wy);
  const float2 r01 = f2_fma(make_float2(b0.x, b0.x), wz, M), r23 = f2_fma(make_float2(b0.y, b0.y), wz, M);
  const float2 r45 = f2_fma(make_float2(b1.x, b1.x), wz, M), r67 = f2_fma(make_float2(b1.y, b1.y), wz, M);
  r[0] = __float_as_uint(r01.x); r[1] = __float_as_uint(r01.y);
  r[2] = __float_as_uint(r23.x); r[3] = __float_as_uint(r23.y);
  r[4] = __float_as_uint(r45.x); r[5] = __float_as_uint(r45.y);
  r[6] = __float_as_uint(r67.x); r[7] = __float_as_uint(r67.y);
}

// The same corner values for |s| < 2^41 quanta, as h 2^20 + l: F = b * wz + 1.5 * 2^43
// has spacing 2^20, so h = (F - 1.5 * 2^43) / 2^20 is the product rounded to a
// multiple of 2^20; 1.5 * 2^23 - h 2^20 = (1.5 * 2^43 + 1.5 * 2^23) - F is exact (a
// multiple of 2^20 below 2^44), and b * wz plus it is one fused multiply-add
// of spacing 1 around 1.5 * 2^23: l is the exact remainder rounded to the nearest
// integer (ties to even, as of the whole product: h 2^20 is even). So h 2^20 + l is
// the exact product rounded once.
__device__ __forceinline__ void dep_corners_wide(float s, float wx0, float fx, float wy0, float fy, float wz0,
                                                 float fz, int (&h)[8], int (&l)[8]) {
  const float2 a = f2_mul(make_float2(s, s), make_float2(wx0, fx));
  const float2 wy = make_float2(wy0, fy), wz = make_float2(wz0, fz);
  const float2 b[2] = {f2_mul(make_float2(a.x, a.x), wy), f2_mul(make_float2(a.y, a.y), wy)};
  const float2 M = make_float2(13194139533312.0f, 13194139533312.0f);  // 1.5 * 2^43
  const float2 K = make_float2(13194152116224.0f, 13194152116224.0f);  // ... + 1.5 * 2^23
  const float2 neg = make_float2(-1.0f, -1.0f);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float bv = (p & 1) ? b[p >> 1].y : b[p >> 1].x;
    const float2 bb = make_float2(bv, bv);
    const float2 F = f2_fma(bb, wz, M);
    const float2 L = f2_fma(bb, wz, f2_fma(F, neg, K));
    h[2 * p] = (int)(__float_as_uint(F.x) - DEP_BIAS_H);
    h[2 * p + 1] = (int)(__float_as_uint(F.y) - DEP_BIAS_H);
    l[2 * p] = (int)(__float_as_uint(L.x) - DEP_BIAS);
    l[2 * p + 1] = (int)(__float_as_uint(L.y) - DEP_BIAS);
  }
}

// Corner contributions of a particle whose mass exceeds 2^22 quanta.
__device__ __forceinline__ void cic_q_large(float mm, float fx, float fy, float fz, float qscale, long long (&q)[8]) {
  const float wx[2] = {__fsub_rn(1.0f, fx), fx};
  const float wy[2] = {__fsub_rn(1.0f, fy), fy};
  const float wz[2] = {__fsub_rn(1.0f, fz), fz};
  const int qk = pow2_exponent(qscale);
#pragma unroll
  for (int c = 0; c < 8; ++c)
    q[c] = prod_to_i64_rn(__fmul_rn(__fmul_rn(mm, wx[c >> 2]), wy[(c >> 1) & 1]), wz[c & 1], qk);
}

// Add 8 corner values to the int64 grid, dropping corners outside it.
__device__ __forceinline__ void corners_to_grid(long long *__restrict__ qg, int G, int ix, int iy, int iz,
                                                const long long (&q)[8]) {
  const bool interior = ix >= 0 && iy >= 0 && iz >= 0 && ix + 1 < G && iy + 1 < G && iz + 1 < G;
  if (interior) {
    const int base = (ix * G + iy) * G + iz;  // G^3 < 2^31
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (q[c] != 0)
        atomicAdd((unsigned long long *)(qg + base + ((c >> 2) * G + ((c >> 1) & 1)) * G + (c & 1)),
                  (unsigned long long)q[c]);
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int jx = ix + (c >> 2), jy = iy + ((c >> 1) & 1), jz = iz + (c & 1);
      if (q[c] != 0 && (unsigned)jx < (unsigned)G && (unsigned)jy < (unsigned)G && (unsigned)jz < (unsigned)G)
        atomicAdd((unsigned long long *)(qg + ((size_t)jx * G + jy) * G + jz), (unsigned long long)q[c]);
    }
  }
}

// A particle whose contribution reaches 2^22 quanta goes to the grid on its own.
__device__ __noinline__ void large_to_grid(long long *__restrict__ qg, int G, int ix, int iy, int iz, float mm,
                                           float fx, float fy, float fz, float qscale) {
  long long q[8];
  cic_q_large(mm, fx, fy, fz, qscale, q);
  corners_to_grid(qg, G, ix, iy, iz, q);
}

// The tile's box of nodes [x0, x0+nx) x [y0, y0+ny) x [z0, z0+nz) in shared memory.
struct DepBox {
  int *b;
  int x0, y0, z0, ny, nz, nyz;
};

template <bool BOX>
__device__ __forceinline__ void dep_out(const DepBox &bx, long long *__restrict__ qg, int G, int ix, int iy, int iz,
                                        const int (&t)[8]) {
  if (BOX) {
    int *b = bx.b + ((ix - bx.x0) * bx.ny + (iy - bx.y0)) * bx.nz + (iz - bx.z0);
    const int nz = bx.nz, nyz = bx.nyz;
    atomicAdd(b, t[0]); atomicAdd(b + 1, t[1]); atomicAdd(b + nz, t[2]); atomicAdd(b + nz + 1, t[3]);
    atomicAdd(b + nyz, t[4]); atomicAdd(b + nyz + 1, t[5]); atomicAdd(b + nyz + nz, t[6]);
    atomicAdd(b + nyz + nz + 1, t[7]);
  } else {
    const long long q[8] = {t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]};
    corners_to_grid(qg, G, ix, iy, iz, q);
  }
}

// dep_out with the lane's box node already located.
template <bool BOX>
__device__ __forceinline__ void dep_put(int bo, const DepBox &bx, long long *__restrict__ qg, int G, int ix, int iy,
                                        int iz, const int (&t)[8]) {
  if (BOX) {
    int *bp = bx.b + bo;
    const int nz = bx.nz, nyz = bx.nyz;
    atomicAdd(bp, t[0]); atomicAdd(bp + 1, t[1]); atomicAdd(bp + nz, t[2]); atomicAdd(bp + nz + 1, t[3]);
    atomicAdd(bp + nyz, t[4]); atomicAdd(bp + nyz + 1, t[5]); atomicAdd(bp + nyz + nz, t[6]);
    atomicAdd(bp + nyz + nz + 1, t[7]);
  } else {
    const long long q[8] = {t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]};
    corners_to_grid(qg, G, ix, iy, iz, q);
  }
}

// The DEP_PER particles of one lane (registers), 32 adjacent particles of the
// warp at a time. Sets bit j of `large` for particles left to the out-of-line pass.
template <bool POW2, bool BOX, int NJ = DEP_PER>
__device__ __forceinline__ void dep_warp_pass(const float (&px)[NJ], const float (&py)[NJ],
                                              const float (&pz)[NJ], const float (&pm)[NJ], long long nrem,
                                              const DepCtx &d, float inv_dx, float qscale, const DepBox &bx,
                                              long long *__restrict__ qg, unsigned *__restrict__ status, int lane,
                                              unsigned &large) {
  const int G1 = d.G + 1;
  const float hi = (float)d.G;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float gx, gy, gz;
    if (POW2) {  // x / dx == x * (1/dx) exactly when dx is a power of two
      gx = __fmul_rn(px[j], inv_dx); gy = __fmul_rn(py[j], inv_dx); gz = __fmul_rn(pz[j], inv_dx);
    } else {
      gx = __fdiv_rn(px[j], d.dx); gy = __fdiv_rn(py[j], d.dx); gz = __fdiv_rn(pz[j], d.dx);
    }
    const bool inr = gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi;
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    const float fx = __fsub_rn(gx, __int2float_rn(ix)), fy = __fsub_rn(gy, __int2float_rn(iy)),
                fz = __fsub_rn(gz, __int2float_rn(iz));
    const float mmq = __fmul_rn(__fmul_rn(pm[j], d.inv_vol), qscale);
    const bool small = fabsf(mmq) < 4194304.0f;
    if (!inr && 32 * j < nrem && !gc_finite3(px[j], py[j], pz[j])) atomicOr(status, GC_FLAG_NONFINITE_POS);
    if (inr && !small) large |= 1u << j;
    const bool ok = inr && small;
    const float s = ok ? mmq : 0.0f;
    const float wx0 = __fsub_rn(1.0f, fx), wy0 = __fsub_rn(1.0f, fy), wz0 = __fsub_rn(1.0f, fz);
    unsigned r[8];
    dep_corners(s, wx0, fx, wy0, fy, wz0, fz, r);
    const unsigned key = ok ? (unsigned)(((ix + 1) * G1 + (iy + 1)) * G1 + (iz + 1)) : DEP_NONE;
    const unsigned kA = __shfl_sync(0xffffffffu, key, 0), kB = __shfl_sync(0xffffffffu, key, 31);
    const bool inA = key == kA, inB = key == kB;
    // the lane's corner values, unbiased once for every use below (lanes without
    // a key are never summed into an output: their products may be NaN)
    int v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = (int)(r[c] - DEP_BIAS);
    // the lane's node in the box, shared by the three outputs (unsigned: a lane
    // without a key may hold any cell)
    const int bo = BOX ? (int)((((unsigned)ix - (unsigned)bx.x0) * (unsigned)bx.ny + ((unsigned)iy - (unsigned)bx.y0)) *
                                   (unsigned)bx.nz +
                               ((unsigned)iz - (unsigned)bx.z0))
                       : 0;
    int t[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) t[c] = __reduce_add_sync(0xffffffffu, inA ? v[c] : 0);
    if (lane == 0 && kA != DEP_NONE) dep_put<BOX>(bo, bx, qg, d.G, ix, iy, iz, t);
    if (kB != kA) {
#pragma unroll
      for (int c = 0; c < 8; ++c) t[c] = __reduce_add_sync(0xffffffffu, inB ? v[c] : 0);
      if (lane == 31 && kB != DEP_NONE) dep_put<BOX>(bo, bx, qg, d.G, ix, iy, iz, t);
    }
    if (!inA && !inB && key != DEP_NONE) dep_put<BOX>(bo, bx, qg, d.G, ix, iy, iz, v);
  }
}

// The box path with warp runs: after the cell sort the warp's 32 particles
// of one step mostly share one cell with those of the next steps, so the warp
// keeps a run cell K (warp-uniform) and each lane adds its corner values for K
// in registers; the run's 8 sums are reduced across the warp (redux.sync) and
// added to the box only when no lane is in K any more, and at the end. Lane 31's
// cell, when it differs from K (the warp reaching the next cell), is reduced at
// once; particles in any other cell (drifted since the sort) add their own
// corners. The sums are those of dep_warp_pass regrouped: integer, exact
// (every partial sum of the warp's 256 particles is below 2^30 on this path).
template <bool POW2, int NJ = DEP_PER>
__device__ __forceinline__ void dep_warp_runs(const float (&px)[NJ], const float (&py)[NJ], const float (&pz)[NJ],
                                              const float (&pm)[NJ], long long nrem, const DepCtx &d, float inv_dx,
                                              float qscale, const DepBox &bx, unsigned *__restrict__ status, int lane,
                                              unsigned &large) {
  const int G1 = d.G + 1;
  const float hi = (float)d.G;
  unsigned K = DEP_NONE;  // the run's cell (warp-uniform) ...
  int Kbo = 0;            // ... and its node in the box
  int acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = 0;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float gx, gy, gz;
    if (POW2) {  // x / dx == x * (1/dx) exactly when dx is a power of two
      gx = __fmul_rn(px[j], inv_dx); gy = __fmul_rn(py[j], inv_dx); gz = __fmul_rn(pz[j], inv_dx);
    } else {
      gx = __fdiv_rn(px[j], d.dx); gy = __fdiv_rn(py[j], d.dx); gz = __fdiv_rn(pz[j], d.dx);
    }
    const bool inr = gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi;
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    const float fx = __fsub_rn(gx, __int2float_rn(ix)), fy = __fsub_rn(gy, __int2float_rn(iy)),
                fz = __fsub_rn(gz, __int2float_rn(iz));
    const float mmq = __fmul_rn(__fmul_rn(pm[j], d.inv_vol), qscale);
    const bool small = fabsf(mmq) < 4194304.0f;
    if (!inr && 32 * j < nrem && !gc_finite3(px[j], py[j], pz[j])) atomicOr(status, GC_FLAG_NONFINITE_POS);
    if (inr && !small) large |= 1u << j;
    const bool ok = inr && small;
    const float s = ok ? mmq : 0.0f;
    const float wx0 = __fsub_rn(1.0f, fx), wy0 = __fsub_rn(1.0f, fy), wz0 = __fsub_rn(1.0f, fz);
    unsigned r[8];
    dep_corners(s, wx0, fx, wy0, fy, wz0, fz, r);
    int v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = (int)(r[c] - DEP_BIAS);
    const unsigned key = ok ? (unsigned)(((ix + 1) * G1 + (iy + 1)) * G1 + (iz + 1)) : DEP_NONE;
    // the lane's node in the box (unsigned: a lane without a key may hold any cell)
    const int bo = (int)((((unsigned)ix - (unsigned)bx.x0) * (unsigned)bx.ny + ((unsigned)iy - (unsigned)bx.y0)) *
                             (unsigned)bx.nz +
                         ((unsigned)iz - (unsigned)bx.z0));
    if (!__any_sync(0xffffffffu, K != DEP_NONE && key == K)) {  // the run has ended (warp-uniform)
      if (K != DEP_NONE) {
        int t[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) t[c] = __reduce_add_sync(0xffffffffu, acc[c]);
        if (lane == 0) dep_put<true>(Kbo, bx, nullptr, d.G, 0, 0, 0, t);
      }
      const unsigned have = __ballot_sync(0xffffffffu, key != DEP_NONE);
      const int src = have ? __ffs(have) - 1 : 0;
      K = have ? __shfl_sync(0xffffffffu, key, src) : DEP_NONE;
      Kbo = __shfl_sync(0xffffffffu, bo, src);
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = 0;
    }
    const bool inK = K != DEP_NONE && key == K;
    if (inK) {
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] += v[c];
    }
    const unsigned kB = __shfl_sync(0xffffffffu, key, 31);
    const bool bnext = kB != K && kB != DEP_NONE;  // lane 31 already in another cell (warp-uniform)
    const bool inB = bnext && key == kB;
    if (bnext) {
      int t[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) t[c] = __reduce_add_sync(0xffffffffu, inB ? v[c] : 0);
      if (lane == 31) dep_put<true>(bo, bx, nullptr, d.G, 0, 0, 0, t);
    }
    if (key != DEP_NONE && !inK && !inB) dep_put<true>(bo, bx, nullptr, d.G, 0, 0, 0, v);
  }
  if (K != DEP_NONE) {
    int t[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) t[c] = __reduce_add_sync(0xffffffffu, acc[c]);
    if (lane == 0) dep_put<true>(Kbo, bx, nullptr, d.G, 0, 0, 0, t);
  }
}

// The same for fine quanta, the two halves of the corner values side by side.
__device__ __forceinline__ void dep_box_add_wide(int *bp, const DepBox &bx, const int (&l)[8], const int (&h)[8]) {
  const int nz = bx.nz, nyz = bx.nyz;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    int *q = bp + (c >> 2) * nyz + ((c >> 1) & 1) * nz + (c & 1);
    atomicAdd(q, l[c]);
    atomicAdd(q + DepW<true>::box, h[c]);
  }
}

template <bool POW2, int NJ = DEP_PER>
__device__ __forceinline__ void dep_warp_runs_wide(const float (&px)[NJ], const float (&py)[NJ], const float (&pz)[NJ],
                                              const float (&pm)[NJ], long long nrem, const DepCtx &d, float inv_dx,
                                              float qscale, const DepBox &bx, unsigned *__restrict__ status, int lane,
                                              unsigned &large) {
  const int G1 = d.G + 1;
  const float hi = (float)d.G;
  unsigned K = DEP_NONE;  // the run's cell (warp-uniform) ...
  int Kbo = 0;            // ... and its node in the box
  int acc[8], acch[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = acch[c] = 0;
  // one lane's sums of the warp, into the box
  auto reduce_put = [&](bool mine, int bo, bool in, const int (&l)[8], const int (&h)[8]) {
    int t[8], th[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      t[c] = __reduce_add_sync(0xffffffffu, in ? l[c] : 0);
      th[c] = __reduce_add_sync(0xffffffffu, in ? h[c] : 0);
    }
    if (mine) dep_box_add_wide(bx.b + bo, bx, t, th);
  };
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float gx, gy, gz;
    if (POW2) {  // x / dx == x * (1/dx) exactly when dx is a power of two
      gx = __fmul_rn(px[j], inv_dx); gy = __fmul_rn(py[j], inv_dx); gz = __fmul_rn(pz[j], inv_dx);
    } else {
      gx = __fdiv_rn(px[j], d.dx); gy = __fdiv_rn(py[j], d.dx); gz = __fdiv_rn(pz[j], d.dx);
    }
    const bool inr = gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi;
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    const float fx = __fsub_rn(gx, __int2float_rn(ix)), fy = __fsub_rn(gy, __int2float_rn(iy)),
                fz = __fsub_rn(gz, __int2float_rn(iz));
    const float mmq = __fmul_rn(__fmul_rn(pm[j], d.inv_vol), qscale);
    const bool small = fabsf(mmq) < DepW<true>::limit;
    if (!inr && 32 * j < nrem && !gc_finite3(px[j], py[j], pz[j])) atomicOr(status, GC_FLAG_NONFINITE_POS);
    if (inr && !small) large |= 1u << j;
    const bool ok = inr && small;
    const float s = ok ? mmq : 0.0f;
    const float wx0 = __fsub_rn(1.0f, fx), wy0 = __fsub_rn(1.0f, fy), wz0 = __fsub_rn(1.0f, fz);
    int v[8], vh[8];
    dep_corners_wide(s, wx0, fx, wy0, fy, wz0, fz, vh, v);
    const unsigned key = ok ? (unsigned)(((ix + 1) * G1 + (iy + 1)) * G1 + (iz + 1)) : DEP_NONE;
    // the lane's node in the box (unsigned: a lane without a key may hold any cell)
    const int bo = (int)((((unsigned)ix - (unsigned)bx.x0) * (unsigned)bx.ny + ((unsigned)iy - (unsigned)bx.y0)) *
                             (unsigned)bx.nz +
                         ((unsigned)iz - (unsigned)bx.z0));
    if (!__any_sync(0xffffffffu, K != DEP_NONE && key == K)) {  // the run has ended (warp-uniform)
      if (K != DEP_NONE) reduce_put(lane == 0, Kbo, true, acc, acch);
      const unsigned have = __ballot_sync(0xffffffffu, key != DEP_NONE);
      const int src = have ? __ffs(have) - 1 : 0;
      K = have ? __shfl_sync(0xffffffffu, key, src) : DEP_NONE;
      Kbo = __shfl_sync(0xffffffffu, bo, src);
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = acch[c] = 0;
    }
    const bool inK = K != DEP_NONE && key == K;
    if (inK) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        acc[c] += v[c];
        acch[c] += vh[c];
      }
    }
    const unsigned kB = __shfl_sync(0xffffffffu, key, 31);
    const bool bnext = kB != K && kB != DEP_NONE;  // lane 31 already in another cell (warp-uniform)
    const bool inB = bnext && key == kB;
    if (bnext) reduce_put(lane == 31, bo, inB, v, vh);
    if (key != DEP_NONE && !inK && !inB) dep_box_add_wide(bx.b + bo, bx, v, vh);
  }
  if (K != DEP_NONE) reduce_put(lane == 0, Kbo, true, acc, acch);
}

// The warp's particles straight into the grid (a tile whose cells do not fit the
// box: sparse regions, where hardly two lanes share a cell): every lane adds its
// own corners, up to 2^41 quanta. Out of line, reloading the particles, so that
// the registers of the box path are not shaped by this rare one. Returns the
// `large` bits. (Reducing the cells of lanes 0 and 31 across the warp first, as
// dep_warp_pass does, cost more than it merged: the deposit of 1.9M particles on
// 128^3 took 33 us with it, 19 without; of 10M on 256^3 75 and 64 us.)
template <bool POW2>
__device__ __noinline__ unsigned dep_warp_direct(const float *__restrict__ x, const float *__restrict__ y,
                                                      const float *__restrict__ z, const float *__restrict__ m,
                                                      long long wb, long long nrem, const DepCtx d, float inv_dx,
                                                      float qscale, long long *__restrict__ qg,
                                                      unsigned *__restrict__ status) {
  unsigned large = 0;
#pragma unroll 2
  for (int j = 0; j < DEP_PER; ++j) {
    if (32 * j >= nrem) break;
    const float px = __ldg(x + wb + 32 * j), py = __ldg(y + wb + 32 * j), pz = __ldg(z + wb + 32 * j);
    const float mmq = __fmul_rn(__fmul_rn(__ldg(m + wb + 32 * j), d.inv_vol), qscale);
    const float gx = POW2 ? __fmul_rn(px, inv_dx) : __fdiv_rn(px, d.dx);
    const float gy = POW2 ? __fmul_rn(py, inv_dx) : __fdiv_rn(py, d.dx);
    const float gz = POW2 ? __fmul_rn(pz, inv_dx) : __fdiv_rn(pz, d.dx);
    const float hi = (float)d.G;
    if (!(gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi)) {
      if (!gc_finite3(px, py, pz)) atomicOr(status, GC_FLAG_NONFINITE_POS);
      continue;
    }
    if (!(fabsf(mmq) < DepW<true>::limit)) {
      large |= 1u << j;
      continue;
    }
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    const float fx = __fsub_rn(gx, __int2float_rn(ix)), fy = __fsub_rn(gy, __int2float_rn(iy)),
                fz = __fsub_rn(gz, __int2float_rn(iz));
    int h[8], l[8];
    dep_corners_wide(mmq, __fsub_rn(1.0f, fx), fx, __fsub_rn(1.0f, fy), fy, __fsub_rn(1.0f, fz), fz, h, l);
    long long q[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) q[c] = (long long)h[c] * 1048576LL + l[c];
    corners_to_grid(qg, d.G, ix, iy, iz, q);
  }
  return large;
}

template <bool POW2, bool WIDE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, (WIDE ? 3 : 4) * (8 / WARPS))
    k_deposit_sorted(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                     const float *__restrict__ m, long long n, DepCtx d, float inv_dx,
                     const double *__restrict__ qexp, long long *__restrict__ qg, unsigned *__restrict__ status,
                     const int *__restrict__ skip, const int *__restrict__ heavy) {
  gc_after();
  __shared__ int dep_box[WARPS * DepW<WIDE>::words];
  if (heavy && (*heavy != 0) != WIDE) return;  // the other form takes the particles
  if (skip && *skip) return;                   // scattered particles: the binned passes take them
  const float qscale = ldexpf(1.0f, -(int)(*qexp));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int tile = WARPS * DEP_WTILE;
  int *wbox = dep_box + warp * DepW<WIDE>::words;  // each warp owns a box: no block-wide barriers
  for (int i = lane; i < DepW<WIDE>::words; i += 32) wbox[i] = 0;  // every flush zeroes what it read
  __syncwarp();
  for (long long t0 = (long long)blockIdx.x * tile; t0 < n; t0 += (long long)gridDim.x * tile) {
    const long long wb = t0 + warp * DEP_WTILE + lane;
    const long long nrem = n - wb;  // particle j of this lane exists when 32 j < nrem
    if (nrem + lane <= 0) continue;  // this warp's part of the last tile is empty (warp-uniform)
    float px[DEP_PER], py[DEP_PER], pz[DEP_PER], pm[DEP_PER];
#pragma unroll
    for (int j = 0; j < DEP_PER; ++j) {
      if (32 * j < nrem) {
        px[j] = __ldg(x + wb + 32 * j); py[j] = __ldg(y + wb + 32 * j); pz[j] = __ldg(z + wb + 32 * j);
        pm[j] = __ldg(m + wb + 32 * j);
      } else {  // missing: NaN position (ignored by the bounds, deposits nothing), zero mass
        px[j] = py[j] = pz[j] = __int_as_float(0x7fc00000);
        pm[j] = 0.0f;
      }
    }
    // the warp's cell range from its coordinate range (fminf/fmaxf skip NaN),
    // clamped to the cells -1 .. G-1 that receive mass, and its largest |m|
    DepBox bx;
    bx.b = wbox;
    bool use_box;
    int nx;
    {
      float xl = 3.0e38f, yl = 3.0e38f, zl = 3.0e38f, xh = -3.0e38f, yh = -3.0e38f, zh = -3.0e38f;
      unsigned mb = 0;
#pragma unroll
      for (int j = 0; j < DEP_PER; ++j) {
        xl = fminf(xl, px[j]); xh = fmaxf(xh, px[j]);
        yl = fminf(yl, py[j]); yh = fmaxf(yh, py[j]);
        zl = fminf(zl, pz[j]); zh = fmaxf(zh, pz[j]);
        mb = max(mb, __float_as_uint(pm[j]) & 0x7fffffffu);
      }
      const float gl = -1.0f, gh = (float)d.G - 1.0f;
      const float cl[3] = {xl, yl, zl}, ch[3] = {xh, yh, zh};
      int lo[3], hi[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float l = POW2 ? __fmul_rn(cl[a], inv_dx) : __fdiv_rn(cl[a], d.dx);
        float h = POW2 ? __fmul_rn(ch[a], inv_dx) : __fdiv_rn(ch[a], d.dx);
        l = fminf(fmaxf(floorf(l), gl), gh);
        h = fminf(fmaxf(floorf(h), gl), gh);
        const bool any_pt = cl[a] <= ch[a];
        lo[a] = __reduce_min_sync(0xffffffffu, any_pt ? (int)l : 0x7fffffff);
        hi[a] = __reduce_max_sync(0xffffffffu, any_pt ? (int)h : -0x7fffffff);
      }
      mb = __reduce_max_sync(0xffffffffu, mb);
      bx.x0 = lo[0]; bx.y0 = lo[1]; bx.z0 = lo[2];
      nx = hi[0] - lo[0] + 2;
      bx.ny = hi[1] - lo[1] + 2;
      bx.nz = hi[2] - lo[2] + 2;
      bx.nyz = bx.ny * bx.nz;
      // every small corner is at most min(largest |m| in quanta, 2^22) + 1/2; a wide
      // one's halves are at most 2^21 and 2^19, so 256 of them stay below 2^30
      const float mq = __fmul_rn(__fmul_rn(__uint_as_float(mb), d.inv_vol), qscale);
      use_box = hi[0] >= lo[0] && (long long)nx * bx.nyz <= DepW<WIDE>::box &&
                (WIDE || __fmul_rn(fminf(mq, 4194304.0f) + 1.0f, (float)DEP_WTILE) < 1073741824.0f);
    }
    unsigned large = 0;
    if (use_box)
      WIDE ? dep_warp_runs_wide<POW2>(px, py, pz, pm, nrem, d, inv_dx, qscale, bx, status, lane, large)
           : dep_warp_runs<POW2>(px, py, pz, pm, nrem, d, inv_dx, qscale, bx, status, lane, large);
    else
      large = dep_warp_direct<POW2>(x, y, z, m, wb, nrem, d, inv_dx, qscale, qg, status);
    while (large) {  // rare: point masses
      const int j = __ffs(large) - 1;
      large &= large - 1;
      const long long p = wb + 32 * j;
      const float gx = POW2 ? __fmul_rn(x[p], inv_dx) : __fdiv_rn(x[p], d.dx);
      const float gy = POW2 ? __fmul_rn(y[p], inv_dx) : __fdiv_rn(y[p], d.dx);
      const float gz = POW2 ? __fmul_rn(z[p], inv_dx) : __fdiv_rn(z[p], d.dx);
      const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
      large_to_grid(qg, d.G, ix, iy, iz, __fmul_rn(m[p], d.inv_vol), __fsub_rn(gx, __int2float_rn(ix)),
                    __fsub_rn(gy, __int2float_rn(iy)), __fsub_rn(gz, __int2float_rn(iz)), qscale);
    }
    if (use_box) {
      __syncwarp();
      // the warp's box to the grid, one atomic per nonzero node; zeroed as read.
      // Node coordinates by correctly rounded reciprocals instead of integer
      // divisions: for i < 2^10 the product (i + 1/2) * (1/nyz) is off by less
      // than the distance to the next integer, so truncating it is the quotient.
      const int vol = nx * bx.nyz;
      const float inv_nyz = __frcp_rn((float)bx.nyz), inv_nz = __frcp_rn((float)bx.nz);
      for (int i = lane; i < vol; i += 32) {
        const int v = wbox[i], vh = WIDE ? wbox[DepW<WIDE>::box + i] : 0;
        if ((v | vh) == 0) continue;
        wbox[i] = 0;
        if (WIDE) wbox[DepW<WIDE>::box + i] = 0;
        const int rx = (int)(((float)i + 0.5f) * inv_nyz), rem = i - rx * bx.nyz;
        const int ry = (int)(((float)rem + 0.5f) * inv_nz), rz = rem - ry * bx.nz;
        const int jx = bx.x0 + rx, jy = bx.y0 + ry, jz = bx.z0 + rz;
        if ((unsigned)jx < (unsigned)d.G && (unsigned)jy < (unsigned)d.G && (unsigned)jz < (unsigned)d.G)
          atomicAdd((unsigned long long *)(qg + ((size_t)jx * d.G + jy) * d.G + jz), (unsigned long long)((long long)vh * 1048576LL + v));
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------------------
// particles in no order: bin by tiles of the grid, then deposit tile by tile
// ------------------------------------------------------------------------------
// k_deposit_sorted adds scattered particles to the grid one corner at a time, and the L2
// adds 116 G corners a second (10M particles: 690 us). Here the particles are first
// counted and copied by tiles of 8 x 16 x 32 cells (the nodes of a tile, 9 x 17 x 33, fit
// shared memory as two 32-bit halves), and every tile is then summed on chip and added
// to the grid once per 8192 particles: integer sums, the same grid. 10M particles at
// 256^3 (two disks): count 48, copy 75, deposit 100 us, 232 in all against 690; 250k at
// 64^3 (a Plummer sphere) 32 against 65. Bound by the shared-memory atomics (16 a particle)
// and, where a tile has few particles, by its flush of 5049 nodes.
// An early form of k_bin_deposit gave wrong sums, and a variant of it a bad address, on
// inputs that this form and one with every index checked take exactly; the cause was not
// found in their source. So the indexes stay checked: a particle's place among the copies, an
// item's tile and range, a node's place in its tile. What fails is left out, or held to the
// tile, and raises GC_FLAG_INDEX (10M particles on 256^3, the whole call: 450.5 us without,
// 451.6 so).
#define BIN_X 8
#define BIN_Y 16
#define BIN_Z 32
#define BIN_MIN 200000      // particles, and at least an eighth of the nodes
#define BIN_MAX 4096        // tiles: grids up to 256^3
#define BIN_MAX_GRID 256
#define BIN_CHUNK (1 << 25) // particles that the passes take at a time: bounds their scratch (671 MB) and places
#define BIN_ITEM 8192       // most particles per flush
#define BIN_SUB 2048        // particles between carries: low halves of at most 2^19 each stay below 2^30
#define BIN_NY (BIN_Y + 1)
#define BIN_NZ (BIN_Z + 1)
#define BIN_NODES ((BIN_X + 1) * BIN_NY * BIN_NZ)
#define BIN_LAST (((BIN_X - 1) * BIN_NY + BIN_Y - 1) * BIN_NZ + BIN_Z - 1)  // the last cell's first node
// Largest particle: halves h of at most 2^18 - 1, so that BIN_ITEM of them stay below 2^31.
#define BIN_LIMIT 2.7487685e11f  // 2^38 - 2^20

// Scratch of the binned passes (ctx->bin): all counters are zero between calls.
struct BinScratch {
  int scattered, nitems, nrare;
  unsigned ticket;
  int count[BIN_MAX], start[BIN_MAX + 1], cursor[BIN_MAX];
};

struct BinGeo {
  int ny, nz, n;  // tiles along y and z, all tiles
};
__host__ __device__ inline BinGeo bin_geo(int G) {
  BinGeo b;
  b.ny = (G + BIN_Y - 1) / BIN_Y;
  b.nz = (G + BIN_Z - 1) / BIN_Z;
  b.n = (G + BIN_X - 1) / BIN_X * b.ny * b.nz;
  return b;
}

// The tile of a position, -1 where nothing is deposited, and its grid coordinates. Cells
// -1 belong to the first tile.
template <bool POW2>
__device__ __forceinline__ int bin_of(float px, float py, float pz, const DepCtx &d, float inv_dx, const BinGeo &b,
                                      float &gx, float &gy, float &gz) {
  gx = POW2 ? __fmul_rn(px, inv_dx) : __fdiv_rn(px, d.dx);
  gy = POW2 ? __fmul_rn(py, inv_dx) : __fdiv_rn(py, d.dx);
  gz = POW2 ? __fmul_rn(pz, inv_dx) : __fdiv_rn(pz, d.dx);
  const float hi = (float)d.G;
  if (!(gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi)) return -1;
  const int ix = max(__float2int_rd(gx), 0), iy = max(__float2int_rd(gy), 0), iz = max(__float2int_rd(gz), 0);
  return ((ix / BIN_X) * b.ny + iy / BIN_Y) * b.nz + iz / BIN_Z;
}

// Pairs of neighbours among 32 particles that lie in about the same column of cells.
__device__ __forceinline__ int near_pairs(float px, float py, float pz, float dx) {
  const float ex = px - __shfl_down_sync(0xffffffffu, px, 1), ey = py - __shfl_down_sync(0xffffffffu, py, 1),
              ez = pz - __shfl_down_sync(0xffffffffu, pz, 1);
  const bool near = (threadIdx.x & 31) < 31 && fabsf(ex) < dx && fabsf(ey) < dx && fabsf(ez) < 4.0f * dx;
  return __popc(__ballot_sync(0xffffffffu, near));
}

// Whether the particles come scattered: of 32 stretches of DEP_WTILE, spread over the
// array, most span more cells than a warp's box of k_deposit_sorted, and fewer than half
// of the neighbours among the first 64 of each lie near each other. (Few particles in the order of their cells do the
// first, and yet their corners share sectors of the grid: 4.3M on 256^3 172 us one by one,
// 305 binned; drifted by a third of a cell 211 and 278, by a whole one 264 and 272, 8M so
// 409 and 341.)
__global__ void __launch_bounds__(1024)
    k_bin_probe(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z, long long n,
                float dx, int G, int box, int *__restrict__ scattered) {
  gc_after();
  __shared__ int fit[32], near[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long p0 = (n - DEP_WTILE) * warp / 31;
  float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
  int pairs = 0;
#pragma unroll
  for (int j = 0; j < DEP_WTILE / 32; ++j) {
    const long long p = p0 + 32 * j + lane;
    const float c[3] = {x[p], y[p], z[p]};
    if (j < 2) pairs += near_pairs(c[0], c[1], c[2], dx);
#pragma unroll
    for (int a = 0; a < 3; ++a) { lo[a] = fminf(lo[a], c[a]); hi[a] = fmaxf(hi[a], c[a]); }
  }
  float vol = 1.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
    const float l = fminf(fmaxf(floorf(lo[a] / dx), -1.0f), (float)G - 1.0f);
    const float h = fminf(fmaxf(floorf(hi[a] / dx), -1.0f), (float)G - 1.0f);
    vol *= fmaxf(h - l + 2.0f, 2.0f);
  }
  if (lane == 0) {
    fit[warp] = vol <= (float)box;
    near[warp] = pairs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0, q = 0;
    for (int w = 0; w < 32; ++w) {
      t += fit[w];
      q += near[w];
    }
    *scattered = t < 16 && q < 32 * 2 * 31 / 2;
  }
}

// Particles per tile; the last block turns the counts into places and items (item =
// (tile, first particle) of at most `per` particles).
template <bool POW2>
__global__ void __launch_bounds__(512)
    k_bin_count(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z, long long n,
                DepCtx d, float inv_dx, int per, BinScratch *__restrict__ sc, int2 *__restrict__ items,
                unsigned *__restrict__ status) {
  gc_after();
  __shared__ int hist[BIN_MAX];
  __shared__ int wsum[2][16];
  __shared__ bool last_s;
  if (!sc->scattered) return;
  const BinGeo b = bin_geo(d.G);
  const int tid = threadIdx.x;
  for (int i = tid; i < b.n; i += 512) hist[i] = 0;
  __syncthreads();
  const long long step = (long long)gridDim.x * 512;
  for (long long p0 = blockIdx.x * 512LL + tid; p0 < n; p0 += 4 * step) {
    float px[4], py[4], pz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long p = p0 + j * step;
      const bool in = p < n;
      px[j] = in ? __ldg(x + p) : 4.0e38f; py[j] = in ? __ldg(y + p) : 0.0f; pz[j] = in ? __ldg(z + p) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float gx, gy, gz;
      const int bin = bin_of<POW2>(px[j], py[j], pz[j], d, inv_dx, b, gx, gy, gz);
      if (bin >= 0)
        atomicAdd(&hist[bin], 1);
      else if (p0 + j * step < n && !gc_finite3(px[j], py[j], pz[j]))
        atomicOr(status, GC_FLAG_NONFINITE_POS);
    }
  }
  __syncthreads();
  for (int i = tid; i < b.n; i += 512)
    if (hist[i]) atomicAdd(&sc->count[i], hist[i]);
  __threadfence();
  __syncthreads();
  if (tid == 0) last_s = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  // 512 threads, BIN_MAX / 512 tiles each
  constexpr int PER = BIN_MAX / 512;
  int cnt[PER], c = 0, it = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = PER * tid + k;
    cnt[k] = i < b.n ? __ldcg(&sc->count[i]) : 0;
    if (i < b.n) sc->count[i] = 0;
    c += cnt[k];
    it += (cnt[k] + per - 1) / per;
  }
  const int lane = tid & 31, warp = tid >> 5;
  int ci = c, ii = it;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, ci, o), e = __shfl_up_sync(0xffffffffu, ii, o);
    if (lane >= o) { ci += a; ii += e; }
  }
  if (lane == 31) { wsum[0][warp] = ci; wsum[1][warp] = ii; }
  __syncthreads();
  int cb = ci - c, ib = ii - it;
  for (int w = 0; w < warp; ++w) { cb += wsum[0][w]; ib += wsum[1][w]; }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = PER * tid + k;
    if (i >= b.n) break;
    sc->start[i] = cb;
    sc->cursor[i] = cb;
    for (int q = 0; q < cnt[k]; q += per) items[ib++] = make_int2(i, cb + q);
    cb += cnt[k];
  }
  if (tid == 511) {
    sc->start[b.n] = cb;
    sc->nitems = ib;
    sc->nrare = 0;
    sc->ticket = 0u;
  }
}

// Particles to their tiles, 2048 a time: ranks within the block by shared-memory
// counters, one place in the tile for all of a block's particles of it. The copies hold
// grid coordinates and quanta. Point masses and particles of cells -1 leave a massless
// copy and go to a list of their own.
template <bool POW2>
__global__ void __launch_bounds__(512, 2)
    k_bin_scatter(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                  const float *__restrict__ m, long long n, DepCtx d, float inv_dx, const double *__restrict__ qexp,
                  BinScratch *__restrict__ sc, float4 *__restrict__ out, int *__restrict__ rare,
                  unsigned *__restrict__ status) {
  gc_after();
  __shared__ int hist[BIN_MAX];
  if (!sc->scattered) return;
  const float qscale = ldexpf(1.0f, -(int)(*qexp));
  const BinGeo b = bin_geo(d.G);
  const int tid = threadIdx.x;
  for (int i = tid; i < b.n; i += 512) hist[i] = 0;
  for (long long c0 = blockIdx.x * 2048LL; c0 < n; c0 += gridDim.x * 2048LL) {
    float4 v[4];
    int bin[4], rank[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long p = c0 + 512 * j + tid;
      const bool in = p < n;
      v[j] = in ? make_float4(__ldg(x + p), __ldg(y + p), __ldg(z + p), __ldg(m + p)) : make_float4(4.0e38f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 c;
      bin[j] = bin_of<POW2>(v[j].x, v[j].y, v[j].z, d, inv_dx, b, c.x, c.y, c.z);
      c.w = __fmul_rn(__fmul_rn(v[j].w, d.inv_vol), qscale);
      v[j] = c;
      rank[j] = bin[j] >= 0 ? atomicAdd(&hist[bin[j]], 1) : 0;
    }
    __syncthreads();
    for (int i = tid; i < b.n; i += 512) {
      const int c = hist[i];
      if (c) hist[i] = atomicAdd(&sc->cursor[i], c);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (bin[j] < 0) continue;
      if (v[j].x < 0.0f || v[j].y < 0.0f || v[j].z < 0.0f || !(fabsf(v[j].w) < BIN_LIMIT)) {
        rare[atomicAdd(&sc->nrare, 1)] = (int)(c0 + 512 * j + tid);
        v[j] = make_float4(fmaxf(v[j].x, 0.0f), fmaxf(v[j].y, 0.0f), fmaxf(v[j].z, 0.0f), 0.0f);
      }
      const int place = hist[bin[j]] + rank[j];
      if ((unsigned)place < (unsigned)n)
        out[place] = v[j];
      else
        atomicOr(status, GC_FLAG_INDEX);
    }
    __syncthreads();
    for (int i = tid; i < b.n; i += 512) hist[i] = 0;
  }
}

// One item at a time: corners into the tile's nodes (halves h 2^20 + l), then the nodes to
// the grid.
__global__ void __launch_bounds__(256)
    k_bin_deposit(const float4 *__restrict__ part, int n, int G, int per, const BinScratch *__restrict__ sc,
                  const int2 *__restrict__ items, long long *__restrict__ qg, unsigned *__restrict__ status) {
  gc_after();
  __shared__ int lo[BIN_NODES], hi[BIN_NODES];
  __shared__ int4 cur;  // the item: first and last particle, tile
  if (!sc->scattered) return;
  const BinGeo b = bin_geo(G);
  const int tid = threadIdx.x, nitems = sc->nitems;
  unsigned worst = 0;  // largest node met
  for (int i = tid; i < BIN_NODES; i += 256) lo[i] = hi[i] = 0;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    __syncthreads();  // the last item's nodes are flushed
    if (tid == 0) {
      const int2 it = items[item];
      int4 c = make_int4(0, 0, 0, 0);
      if ((unsigned)it.x < (unsigned)b.n) c = make_int4(it.y, min(sc->start[it.x + 1], it.y + per), it.x, 0);
      if (c.x < 0 || c.x >= c.y || c.y > n) {
        c = make_int4(0, 0, 0, 0);
        atomicOr(status, GC_FLAG_INDEX);
      }
      cur = c;
    }
    __syncthreads();
    const int end = cur.y, tile = cur.z;
    const int tz = tile % b.nz, txy = tile / b.nz, ty = txy % b.ny, tx = txy / b.ny;
    const int x0 = tx * BIN_X, y0 = ty * BIN_Y, z0 = tz * BIN_Z;
    for (int s0 = cur.x; s0 < end; s0 += BIN_SUB) {
      const int s1 = min(end, s0 + BIN_SUB);
#pragma unroll 2
      for (int p = s0 + tid; p < s1; p += 256) {
        const float4 v = __ldcs(part + p);
        const int ix = __float2int_rd(v.x), iy = __float2int_rd(v.y), iz = __float2int_rd(v.z);
        const float fx = __fsub_rn(v.x, __int2float_rn(ix)), fy = __fsub_rn(v.y, __int2float_rn(iy)),
                    fz = __fsub_rn(v.z, __int2float_rn(iz));
        int h[8], l[8];
        dep_corners_wide(v.w, __fsub_rn(1.0f, fx), fx, __fsub_rn(1.0f, fy), fy, __fsub_rn(1.0f, fz), fz, h, l);
        const unsigned at = (unsigned)(((ix - x0) * BIN_NY + (iy - y0)) * BIN_NZ + (iz - z0));
        worst = max(worst, at);
        const int node = (int)min(at, (unsigned)BIN_LAST);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int q = node + (c >> 2) * (BIN_NY * BIN_NZ) + ((c >> 1) & 1) * BIN_NZ + (c & 1);
          atomicAdd(&lo[q], l[c]);
          atomicAdd(&hi[q], h[c]);
        }
      }
      __syncthreads();
      if (s1 < end) {  // carry, so that the low halves stay below 2^31
        for (int i = tid; i < BIN_NODES; i += 256) {
          const int v = lo[i];
          hi[i] += v >> 20;
          lo[i] = v & 0xfffff;
        }
        __syncthreads();
      }
    }
    for (int i = tid; i < BIN_NODES; i += 256) {
      const int l = lo[i], h = hi[i];
      if ((l | h) == 0) continue;
      lo[i] = hi[i] = 0;
      const int rx = i / (BIN_NY * BIN_NZ), rem = i - rx * (BIN_NY * BIN_NZ), ry = rem / BIN_NZ, rz = rem - ry * BIN_NZ;
      const int jx = x0 + rx, jy = y0 + ry, jz = z0 + rz;
      const long long v = (long long)h * 1048576LL + l;
      if (v != 0 && jx < G && jy < G && jz < G)
        atomicAdd((unsigned long long *)(qg + ((size_t)jx * G + jy) * G + jz), (unsigned long long)v);
    }
  }
  if (worst > BIN_LAST) atomicOr(status, GC_FLAG_INDEX);
}

// The particles that no tile takes, one by one.
template <bool POW2>
__global__ void __launch_bounds__(256)
    k_bin_rare(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
               const float *__restrict__ m, DepCtx d, float inv_dx, const double *__restrict__ qexp,
               const BinScratch *__restrict__ sc, const int *__restrict__ rare, long long *__restrict__ qg) {
  gc_after();
  if (!sc->scattered) return;
  const float qscale = ldexpf(1.0f, -(int)(*qexp));
  const int n = sc->nrare;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const int p = rare[i];
    const float gx = POW2 ? __fmul_rn(x[p], inv_dx) : __fdiv_rn(x[p], d.dx);
    const float gy = POW2 ? __fmul_rn(y[p], inv_dx) : __fdiv_rn(y[p], d.dx);
    const float gz = POW2 ? __fmul_rn(z[p], inv_dx) : __fdiv_rn(z[p], d.dx);
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    large_to_grid(qg, d.G, ix, iy, iz, __fmul_rn(m[p], d.inv_vol), __fsub_rn(gx, __int2float_rn(ix)),
                  __fsub_rn(gy, __int2float_rn(iy)), __fsub_rn(gz, __int2float_rn(iz)), qscale);
  }
}

// The binned passes' scratch for n <= BIN_CHUNK particles, grown as needed and kept by the context:
// counters, items, copies, list. False where it cannot be had (device memory) and for a
// stream under capture, whose recorded kernels would go on using a block that a larger
// deposit has replaced: the particles are then deposited one by one.
//
// Particles per item: BIN_ITEM where that leaves two items for every SM, else BIN_SUB (250k
// particles on 64^3: the tiles take 42 us with 8192, 14 with 2048).
static int bin_item(int64_t n) { return n >= (int64_t)gc_sms() * 2 * BIN_ITEM ? BIN_ITEM : BIN_SUB; }
static bool bin_scratch(gc_ctx *ctx, int64_t n) {
  const size_t items = (size_t)BIN_MAX + (size_t)(n / bin_item(n)) + 1;
  const size_t head = (sizeof(BinScratch) + 255) & ~(size_t)255, ib = (items * sizeof(int2) + 255) & ~(size_t)255;
  const size_t need = head + ib + (size_t)n * (sizeof(float4) + sizeof(int));
  if (gc_stream_capturing(ctx)) return false;
  if (ctx->bin && ctx->bin_cap >= need) return true;
  if (ctx->bin) cudaFree(ctx->bin);  // (waits for the work that uses it)
  ctx->bin = nullptr;
  ctx->bin_cap = 0;
  if (cudaMalloc(&ctx->bin, need) != cudaSuccess) {
    cudaGetLastError();
    ctx->bin = nullptr;
    return false;
  }
  if (cudaMemsetAsync(ctx->bin, 0, head, ctx->stream) != cudaSuccess) return false;
  ctx->bin_cap = need;
  return true;
}

int gc_deposit_q(gc_ctx *ctx, const float *x, const float *y, const float *z, const float *m, int64_t n, int bits,
                 const double *qexp, bool any_order) {
  if (n <= 0) return GC_OK;
  DepCtx d;
  d.dx = (float)ctx->dx;
  d.inv_vol = 1.0f / ((d.dx * d.dx) * d.dx);
  d.G = ctx->G;
  int fe = 0;
  const bool pow2 = std::frexp(d.dx, &fe) == 0.5f;
  const float inv_dx = pow2 ? std::ldexp(1.0f, 1 - fe) : 0.0f;
  // The narrow pass takes particles below 2^22 quanta, the wide one below 2^41; both
  // leave the rest to the out-of-line rounding, so the choice changes only speed. Where
  // the particles fit it, the narrow pass has half the sums (8M on 64^3 in the order of their
  // cells at 2^-44 of the mass: a deposit 91 us narrow, 127 wide; drifted by a third of a
  // cell 126 and 204); beyond 2^22 quanta its out-of-line particles take thirty times as long
  // (1.5M at 2^-52: 327 us narrow, 21 wide). The mean particle has 1 to 2 times mean_quanta:
  // narrow below 2^20, where particles of a few times the mean still fit, wide from 2^22 on.
  // Between them both are launched and a sample of the masses (k_mass_heavy) tells the one
  // whose particles they are not to return (4 us in all), from HEAVY_MIN particles on, below
  // which the passes differ by less (600k on 32^3: 38 and 44 us).
  const bool both = quanta_undecided(bits, n), wide = mean_quanta(bits, n) >= 1048576.0;
  const int *heavy = both ? reinterpret_cast<const int *>(qexp + 1) : nullptr;
  // CTAs of eight warps; of two while eight would leave SMs without one (131072
  // particles: 20.4 us with eight, 18.5 with two)
  const bool few = n < (int64_t)gc_sms() * 8 * DEP_WTILE;
  const int warps = few ? 2 : 8;
  const long long tile = (long long)warps * DEP_WTILE;
  const long long ntiles = (n + tile - 1) / tile;
  // Callers that cannot say how their particles are ordered: a probe on the device
  // chooses between this kernel and the binned passes, and the one not chosen returns at
  // once (10 us of launches for sorted particles). The passes win from some 500 particles a
  // tile on: 2M in a Gaussian on 128^3 104 us one by one, 68 binned, on 256^3 114 and 102,
  // 10M 465 and 335; but 500k on 128^3 34 and 35, on 256^3 45 and 54.
  const bool bins = any_order && n >= BIN_MIN && n >= (int64_t)ctx->G * ctx->G * ctx->G / 8 && ctx->G <= BIN_MAX_GRID &&
                    bin_scratch(ctx, std::min<int64_t>(n, BIN_CHUNK));
  BinScratch *sc = bins ? (BinScratch *)ctx->bin : nullptr;
  if (bins)
    gc_launch_after(ctx, GK_DEPOSIT_RUNS, k_bin_probe, dim3(1), dim3(1024), 0, x, y, z, (long long)n, d.dx, ctx->G,
              wide ? (int)DepW<true>::box : (int)DepW<false>::box, &sc->scattered);
  for (int w = 0; w < 2; ++w) {
    if (!both && (w != 0) != wide) continue;
    auto k = few ? (w ? (pow2 ? k_deposit_sorted<true, true, 2> : k_deposit_sorted<false, true, 2>)
                      : (pow2 ? k_deposit_sorted<true, false, 2> : k_deposit_sorted<false, false, 2>))
                 : (w ? (pow2 ? k_deposit_sorted<true, true, 8> : k_deposit_sorted<false, true, 8>)
                      : (pow2 ? k_deposit_sorted<true, false, 8> : k_deposit_sorted<false, false, 8>));
    const long long most = (long long)gc_sms() * (w ? 3 : 4) * (8 / warps);  // resident CTAs: persistent
    const unsigned nb = (unsigned)(ntiles < most ? ntiles : most);
    gc_launch_after(ctx, GK_DEPOSIT_RUNS, k, dim3(nb), dim3(32 * warps), 0, x, y, z, m, (long long)n, d, inv_dx, qexp, ctx->q,
              ctx->dstatus, bins ? (const int *)&sc->scattered : (const int *)nullptr, heavy);
  }
  if (bins) {
    const int64_t most_c = std::min<int64_t>(n, BIN_CHUNK);
    const size_t head = (sizeof(BinScratch) + 255) & ~(size_t)255;
    const int per = bin_item(most_c);
    const size_t ib = (((size_t)BIN_MAX + (size_t)(most_c / per) + 1) * sizeof(int2) + 255) & ~(size_t)255;
    int2 *items = (int2 *)((char *)ctx->bin + head);
    float4 *copy = (float4 *)((char *)ctx->bin + head + ib);
    int *rare = (int *)(copy + most_c);
    const unsigned sms = (unsigned)gc_sms();
    auto k1 = pow2 ? k_bin_count<true> : k_bin_count<false>;
    auto k2 = pow2 ? k_bin_scatter<true> : k_bin_scatter<false>;
    auto k4 = pow2 ? k_bin_rare<true> : k_bin_rare<false>;
    for (int64_t at = 0; at < n; at += BIN_CHUNK) {
      const int64_t c = std::min<int64_t>(n - at, BIN_CHUNK);
      const float *px = x + at, *py = y + at, *pz = z + at, *pm = m + at;
      gc_launch_after(ctx, GK_DEPOSIT_RUNS, k1, dim3(std::min(gc_blocks(c, 2048), sms * 3u)), dim3(512), 0, px, py, pz,
                (long long)c, d, inv_dx, per, sc, items, ctx->dstatus);
      gc_launch_after(ctx, GK_DEPOSIT_RUNS, k2, dim3(std::min(gc_blocks(c, 2048), sms * 2u)), dim3(512), 0, px, py, pz, pm,
                (long long)c, d, inv_dx, qexp, sc, copy, rare, ctx->dstatus);
      gc_launch_after(ctx, GK_DEPOSIT_RUNS, k_bin_deposit, dim3(sms * 5u), dim3(256), 0, (const float4 *)copy, (int)c,
                ctx->G, per, (const BinScratch *)sc, (const int2 *)items, ctx->q, ctx->dstatus);
      gc_launch_after(ctx, GK_DEPOSIT_RUNS, k4, dim3(sms), dim3(256), 0, px, py, pz, pm, d, inv_dx, qexp,
                (const BinScratch *)sc, (const int *)rare, ctx->q);
    }
  }
  GC_LAUNCH_CHECK(ctx, "deposit");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// q -> rho / b, zero q, exact integer column moments, ||b||^2
// ------------------------------------------------------------------------------
// One warp per (i,j) column, blocks persistent over batches of 8 cpw columns. Column
// sums S0 = sum q, S1 = sum q k and S2 = sum q k^2 are exact in integers (S2 split at
// bit 32), and so are the grid's ten moments: each is kept as three limbs (24 bits, 32
// for S2) that take the columns' products with 1, i, j, i^2, ij, j^2 in 64 bits and are added
// over blocks by integer atomics; the last block puts the limbs together and rounds
// once. Block partials of ||b||^2 (FP32 column sums, added in FP64 in a fixed order).
//
// FP64 is kept out because an addition takes its quarter of the SM 64 clocks a warp,
// whichever lanes take part. With every column's terms in FP64 on lane 0 of its warp and
// 11 x 456 partials for the last block to add, a 64^3 grid took 20 us; with the terms of
// 32 columns in the lanes of a warp 13, of which 5k clk were the warp's and 9k the
// last block's additions; in integers 8 (100^3: 19 -> 12; 128^3: 24 -> 14; at 256^3,
// 47 -> 39, the grid's bytes are what is left). Three warps beside the eight that walk
// columns take a lane per column of a batch, while the eight go on to the next.
#define CQ_THREADS 352
struct CqCol {
  long long s0, s1, s2h;
  unsigned long long s2l;
  float bb;
};

// l0 + l1 2^r1 + l2 2^r2 of a sum of limbs, rounded once.
__device__ __forceinline__ double limbs_to_double(long long l0, long long l1, long long l2, int r1, int r2) {
  __int128 v = (__int128)l0 + ((__int128)l1 << r1) + ((__int128)l2 << r2);
  const bool neg = v < 0;
  if (neg) v = -v;
  unsigned long long hi = (unsigned long long)(v >> 64), lo = (unsigned long long)v;
  double d;
  if (hi == 0) {
    d = __ull2double_rn(lo);
  } else {  // 64 leading bits, the rest as a sticky bit below them
    const int z = __clzll((long long)hi);
    unsigned long long top = z ? (hi << z) | (lo >> (64 - z)) : hi;
    if (z ? (lo << z) != 0 : lo != 0) top |= 1ull;
    d = ldexp(__ull2double_rn(top), 64 - z);
  }
  return neg ? -d : d;
}

__global__ void __launch_bounds__(CQ_THREADS, 3)
    k_convert_q(long long *__restrict__ qg, int G, int cpw, double dx, const double *__restrict__ qexp,
                float *__restrict__ rho, float *__restrict__ b, double bfac, double *__restrict__ parts,
                unsigned *__restrict__ ticket, long long *__restrict__ limbs, double *__restrict__ mom,
                double *__restrict__ bnorm2) {
  gc_after();
  __shared__ CqCol cols[2][32];
  __shared__ long long red[3][12][33];
  __shared__ double bsum[4];
  __shared__ bool last_s;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int E = (int)(*qexp);
  const float qinv = ldexpf(1.0f, E);
  const float bscale = (float)(ldexp(1.0, E) * bfac);
  const int ncols = G * G, batch = 8 * cpw;
  // limbs of the warp's moments (warps 8, 9, 10), a column of `red` per lane: in registers
  // they would be live in the other warps too
  if (wid >= 8) {
    for (int t = 0; t < 12; ++t) red[wid - 8][t][lane] = 0;
  }
  double bacc = 0.0;
  int buf = 0;
  for (int base = blockIdx.x * batch; base < ncols; base += gridDim.x * batch, buf ^= 1) {
    if (wid < 8) {
      for (int c = 0; c < cpw; ++c) {
        const int col = base + 8 * c + wid;
        if (col >= ncols) break;
        long long *p = qg + (size_t)col * G;
        float *rp = rho ? rho + (size_t)col * G : nullptr;
        float *bp = b ? b + (size_t)col * G : nullptr;
        long long S0 = 0, S1 = 0, S2h = 0;
        unsigned long long S2l = 0;
        float bb = 0.0f;
        bool some = false;
        for (int k0 = 0; k0 < G; k0 += 32 * 8) {
          long long qv[8];
          bool nz = false;
#pragma unroll
          for (int t = 0; t < 8; ++t) {  // all loads of the lane in flight together
            const int k = k0 + 32 * t + lane;
            qv[t] = k < G ? p[k] : 0;
            nz |= qv[t] != 0;
          }
          if (!__any_sync(0xffffffffu, nz)) {  // an empty stretch (most of a disk's box): zeros out, q stays 0
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              const int k = k0 + 32 * t + lane;
              if (k >= G) continue;
              if (rp) rp[k] = 0.0f;
              if (bp) bp[k] = 0.0f;
            }
            continue;
          }
          some = true;
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const int k = k0 + 32 * t + lane;
            if (k >= G) continue;
            if (qv[t] != 0) p[k] = 0;  // clear for the next deposit (zeros need no store)
            const float qf = i64_to_f32_rn(qv[t]);  // one rounding, as (float)q
            if (rp) rp[k] = __fmul_rn(qf, qinv);
            const float bv = __fmul_rn(qf, bscale);
            if (bp) bp[k] = bv;
            bb += bv * bv;
            const long long kk = k;
            S0 += qv[t];
            S1 += qv[t] * kk;
            S2h += (qv[t] >> 32) * (kk * kk);
            S2l += (unsigned long long)(qv[t] & 0xffffffffLL) * (unsigned long long)(kk * kk);
          }
        }
        if (some) {  // exact integer warp sums (no FP64 per lane)
          for (int o = 16; o > 0; o >>= 1) {
            S0 += __shfl_down_sync(0xffffffffu, S0, o);
            S1 += __shfl_down_sync(0xffffffffu, S1, o);
            S2h += __shfl_down_sync(0xffffffffu, S2h, o);
            S2l += __shfl_down_sync(0xffffffffu, S2l, o);
            bb += __shfl_down_sync(0xffffffffu, bb, o);
          }
        }
        if (lane == 0) cols[buf][8 * c + wid] = {S0, S1, S2h, S2l, bb};
      }
    }
    __syncthreads();  // the other buffer is free again two batches on, behind the next barrier
    if (wid >= 8 && ticket) {
      const int col = base + lane;
      if (lane < batch && col < ncols) {
        const CqCol q = cols[buf][lane];
        const long long i = col / G, j = col - i * G;
        // warp 8: M, x, y; warp 9: xx, yy, xy; warp 10: z, xz, yz and zz
        const long long S = wid == 10 ? q.s1 : q.s0;
        const long long w0 = wid == 9 ? i * i : 1, w1 = wid == 9 ? j * j : i, w2 = wid == 9 ? i * j : j;
        const long long a0 = S & 0xffffff, a1 = (S >> 24) & 0xffffff, a2 = S >> 48;
        long long(*L)[33] = red[wid - 8];
        L[0][lane] += a0 * w0; L[1][lane] += a1 * w0; L[2][lane] += a2 * w0;
        L[3][lane] += a0 * w1; L[4][lane] += a1 * w1; L[5][lane] += a2 * w1;
        L[6][lane] += a0 * w2; L[7][lane] += a1 * w2; L[8][lane] += a2 * w2;
        if (wid == 10) {
          L[9][lane] += (long long)(q.s2l & 0xffffffffull);
          L[10][lane] += (long long)(q.s2l >> 32) + q.s2h;
        } else if (wid == 8) {
          bacc += (double)q.bb;
        }
      }
    }
  }
  if (!ticket) return;
  if (wid >= 8) {
    __syncwarp();
    if (lane < (wid == 10 ? 11 : 9)) {
      long long x = 0;
#pragma unroll 8
      for (int l = 0; l < 32; ++l) x += red[wid - 8][lane][l];
      const int m = lane / 3, v = wid == 8 ? m : (wid == 9 ? (m == 2 ? 7 : 4 + m) : (m == 0 ? 3 : (m == 3 ? 6 : 7 + m)));
      if (x != 0) atomicAdd((unsigned long long *)(limbs + 3 * v + (lane - 3 * m)), (unsigned long long)x);
    }
    if (wid == 8) {
      for (int o = 16; o > 0; o >>= 1) bacc += __shfl_down_sync(0xffffffffu, bacc, o);
      if (lane == 0) parts[blockIdx.x] = bacc;
    }
    __threadfence();  // before the block's ticket
  }
  __syncthreads();
  if (threadIdx.x == 256) last_s = atomicAdd(ticket, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  if (wid < 4) {
    double x = 0.0;
#pragma unroll 4
    for (int r = threadIdx.x; r < (int)gridDim.x; r += 128) x += __ldcg(parts + r);
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) bsum[wid] = x;
  }
  if (wid == 8) {
    if (lane < 10) {
      const long long l0 = __ldcg(limbs + 3 * lane), l1 = __ldcg(limbs + 3 * lane + 1), l2 = __ldcg(limbs + 3 * lane + 2);
      const double msc = ldexp(1.0, E) * dx * dx * dx;  // mass of one quantum
      const double s = lane == 0 ? 1.0 : (lane < 4 ? dx : dx * dx);
      mom[lane] = limbs_to_double(l0, l1, l2, lane == 6 ? 32 : 24, 48) * msc * s;
    }
    __syncwarp();
    if (lane < 30) limbs[lane] = 0;  // for the next call
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mom[10] = (bsum[0] + bsum[1]) + (bsum[2] + bsum[3]);
    *bnorm2 = mom[10];
    *ticket = 0u;
  }
}

// Columns a warp takes per batch: four where that leaves a batch for every SM,
// else two or one (a small grid is bound by latency, and wants its columns spread).
int gc_convert_cpw(int G) {
  int cpw = 4;
  while (cpw > 1 && (long long)G * G < 8LL * gc_sms() * cpw) cpw >>= 1;
  return cpw;
}

int gc_max_fixed_point_bits(const gc_ctx *ctx) {
  int lg = 0;
  while ((1 << lg) < ctx->G) ++lg;
  const int b = 62 - lg;
  return b > 60 ? 60 : b;
}

int gc_convert_q(gc_ctx *ctx, const double *qexp, float *rho_out, float *b_out) {
  const long long cols = (long long)ctx->G * ctx->G;
  const int cpw = gc_convert_cpw(ctx->G);
  unsigned nb = gc_blocks(cols, 8 * cpw);
  if (nb > gc_sms() * 3u) nb = gc_sms() * 3u;  // persistent: 3 CTAs per SM
  int s = gc_ensure_red(ctx, (size_t)nb * 11);
  if (s) return s;
  const double bfac = 4.0 * M_PI * ctx->grav * ctx->dx * ctx->dx;
  gc_launch_after(ctx, GK_CONVERT_Q, k_convert_q, dim3(nb), dim3(CQ_THREADS), 0, ctx->q, ctx->G, cpw, ctx->dx, qexp, rho_out, b_out,
            bfac, ctx->red, reinterpret_cast<unsigned *>(ctx->dsmall + GC_S_TICKET),
            reinterpret_cast<long long *>(ctx->dsmall + GC_S_LIMBS), ctx->dmom, ctx->dsmall + GC_S_BNORM2);
  GC_LAUNCH_CHECK(ctx, "convert q");
  return GC_OK;
}

extern "C" int gc_deposit_cic(gc_ctx *ctx, const float *x, const float *y, const float *z, const float *m, int64_t n,
                              int fixed_point_bits, float *rho) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, rho, "gc_deposit_cic: NULL rho");
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range: %lld", (long long)n);
  GC_REQUIRE(ctx, n == 0 || (x && y && z && m), "gc_deposit_cic: NULL particle array");
  GC_REQUIRE(ctx, fixed_point_bits >= 24 && fixed_point_bits <= gc_max_fixed_point_bits(ctx),
             "fixed_point_bits must be in [24, %d] for a %d^3 grid", gc_max_fixed_point_bits(ctx), ctx->G);
  int s;
  if (n > 0) {
    if ((s = gc_fixed_point_setup(ctx, m, n, fixed_point_bits, GC_S_MASS, GC_S_QEXP))) return s;
    if ((s = gc_deposit_q(ctx, x, y, z, m, n, fixed_point_bits, ctx->dsmall + GC_S_QEXP, true))) return s;
  }
  return gc_convert_q(ctx, ctx->dsmall + GC_S_QEXP, rho, nullptr);
}

// ------------------------------------------------------------------------------
// gradient (deposit.py:132-174)
// ------------------------------------------------------------------------------
__device__ __forceinline__ float grad_comp(const float *__restrict__ phi, size_t c, size_t stride, int idx, int G,
                                           float inv_dx, float inv_2dx) {
  if (idx == 0) return -__fmul_rn(__fsub_rn(phi[c + stride], phi[c]), inv_dx);
  if (idx == G - 1) return -__fmul_rn(__fsub_rn(phi[c], phi[c - stride]), inv_dx);
  return -__fmul_rn(__fsub_rn(phi[c + stride], phi[c - stride]), inv_2dx);
}

struct GradCtx {
  int G;
  float inv_dx, inv_2dx;
};

__host__ static GradCtx make_grad(const gc_ctx *ctx) {
  GradCtx g;
  g.G = ctx->G;
  const float dx = (float)ctx->dx;
  g.inv_dx = 1.0f / dx;
  g.inv_2dx = 1.0f / (2.0f * dx);
  return g;
}

__global__ void __launch_bounds__(256)
    k_grad(const float *__restrict__ phi, float *__restrict__ ax, float *__restrict__ ay, float *__restrict__ az,
           GradCtx g) {
  gc_after();
  const int k = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= g.G || j >= g.G) return;
  const size_t G = g.G;
  const size_t c = ((size_t)i * G + j) * G + k;
  ax[c] = grad_comp(phi, c, G * G, i, g.G, g.inv_dx, g.inv_2dx);
  ay[c] = grad_comp(phi, c, G, j, g.G, g.inv_dx, g.inv_2dx);
  az[c] = grad_comp(phi, c, 1, k, g.G, g.inv_dx, g.inv_2dx);
}

extern "C" int gc_potential_to_accel(gc_ctx *ctx, const float *phi, float *ax, float *ay, float *az) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, phi && ax && ay && az, "gc_potential_to_accel: NULL pointer");
  const GradCtx g = make_grad(ctx);
  gc_launch_after(ctx, GK_GRAD, k_grad, dim3(dim3(gc_blocks(g.G, 32), gc_blocks(g.G, 8), g.G)), dim3(dim3(32, 8)), 0, phi, ax, ay, az, g);
  GC_LAUNCH_CHECK(ctx, "grad");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// gather (deposit.py:85-129)
// ------------------------------------------------------------------------------
#define PACK_MIN 4194304  // particles, and at least an eighth of the nodes
#define PACK_LINES 16     // stretches of 32 particles that tell whether they come in order

// Particles whose corners are all nodes of the grid load the 24 values at once; bounds
// checks and an address for each corner made this bound by instructions (8M particles on
// 256^3 in the order of their cells, a Gaussian: 113 us, 87 so; 32 registers, eight CTAs an
// SM: with six 92).
//
// With g4 (many particles) every block looks at the same PACK_LINES stretches, spread over
// the array. Where few neighbours lie near each other the blocks set the three fields side
// by side for k_gather_packed instead, and *scattered tells it so. Few: an eighth of the
// pairs; half of them with more particles than nodes, whose packing then costs less than it
// saves (particles one cell off their order: 4.2M on 256^3 117 us from the fields, 165
// packed; 20M on 256^3 504 and 410, 8M on 128^3 206 and 146). A look costs 1 us, the
// kernel that returns 3. g4 and scattered are the call's own.
__global__ void __launch_bounds__(256, 8)
    k_gather(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z, long long n,
             const float *__restrict__ axg, const float *__restrict__ ayg, const float *__restrict__ azg,
             float *__restrict__ ax, float *__restrict__ ay, float *__restrict__ az, float dx, int G,
             float4 *__restrict__ g4, int *__restrict__ scattered) {
  gc_after();
  if (g4) {
    __shared__ int near_s[8];
    const int warp = threadIdx.x >> 5;
    int c = 0;
#pragma unroll
    for (int s = 0; s < PACK_LINES / 8; ++s) {
      const long long p = (n - 32) * (warp + 8 * s) / (PACK_LINES - 1) + (threadIdx.x & 31);
      c += near_pairs(__ldg(x + p), __ldg(y + p), __ldg(z + p), dx);
    }
    if ((threadIdx.x & 31) == 0) near_s[warp] = c;
    __syncthreads();
    c = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) c += near_s[w];
    const size_t nodes = (size_t)G * G * G;
    const bool sc = c < PACK_LINES * 31 / ((size_t)n > nodes + nodes / 8 ? 2 : 8);
    if (blockIdx.x == 0 && threadIdx.x == 0) *scattered = sc;
    if (sc) {
      for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < nodes; i += (size_t)gridDim.x * 256)
        g4[i] = make_float4(axg[i], ayg[i], azg[i], 0.0f);
      return;
    }
  }
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    CellPos c;
    if (gc_cell_of(x[p], y[p], z[p], dx, G, c)) {
      const float wx[2] = {__fsub_rn(1.0f, c.fx), c.fx};
      const float wy[2] = {__fsub_rn(1.0f, c.fy), c.fy};
      const float wz[2] = {__fsub_rn(1.0f, c.fz), c.fz};
      if (min(min(c.ix, c.iy), c.iz) >= 0 && max(max(c.ix, c.iy), c.iz) + 1 < G) {
        const int at = (c.ix * G + c.iy) * G + c.iz;  // G^3 <= 2^30
        float u[8], v[8], w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = __ldg(axg + at + ((k >> 2) * G + ((k >> 1) & 1)) * G + (k & 1));
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldg(ayg + at + ((k >> 2) * G + ((k >> 1) & 1)) * G + (k & 1));
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __ldg(azg + at + ((k >> 2) * G + ((k >> 1) & 1)) * G + (k & 1));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float f = __fmul_rn(__fmul_rn(wx[k >> 2], wy[(k >> 1) & 1]), wz[k & 1]);
          sx = __fadd_rn(sx, __fmul_rn(f, u[k]));
          sy = __fadd_rn(sy, __fmul_rn(f, v[k]));
          sz = __fadd_rn(sz, __fmul_rn(f, w[k]));
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int jx = c.ix + (k >> 2), jy = c.iy + ((k >> 1) & 1), jz = c.iz + (k & 1);
          if ((unsigned)jx >= (unsigned)G || (unsigned)jy >= (unsigned)G || (unsigned)jz >= (unsigned)G) continue;
          const float f = __fmul_rn(__fmul_rn(wx[k >> 2], wy[(k >> 1) & 1]), wz[k & 1]);
          const size_t idx = ((size_t)jx * G + jy) * G + jz;
          sx = __fadd_rn(sx, __fmul_rn(f, axg[idx]));
          sy = __fadd_rn(sy, __fmul_rn(f, ayg[idx]));
          sz = __fadd_rn(sz, __fmul_rn(f, azg[idx]));
        }
      }
    }
    ax[p] = sx;
    ay[p] = sy;
    az[p] = sz;
  }
}

// k_gather for many scattered particles, from the packed fields: the same sums in the
// same order, 8 loads of 16 bytes a particle where three fields take 24 of 4, each of them
// another sector of the L2, which is what bounds it. In no order, a Gaussian, with the packing: 8M on 256^3 633 us
// from the fields, 273 so; 20M 1569 and 554; 4.2M on 64^3 222 and 96. (One kernel for
// both kinds was slower for ordered particles: its registers.)
__global__ void __launch_bounds__(256)
    k_gather_packed(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z, long long n,
                    const int *__restrict__ scattered, const float4 *__restrict__ g4, float *__restrict__ ax,
                    float *__restrict__ ay, float *__restrict__ az, float dx, int G) {
  gc_after();
  if (!*scattered) return;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    CellPos c;
    if (gc_cell_of(x[p], y[p], z[p], dx, G, c)) {
      const float wx[2] = {__fsub_rn(1.0f, c.fx), c.fx};
      const float wy[2] = {__fsub_rn(1.0f, c.fy), c.fy};
      const float wz[2] = {__fsub_rn(1.0f, c.fz), c.fz};
      float4 v[8];
      bool in[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int jx = c.ix + (k >> 2), jy = c.iy + ((k >> 1) & 1), jz = c.iz + (k & 1);
        in[k] = (unsigned)jx < (unsigned)G && (unsigned)jy < (unsigned)G && (unsigned)jz < (unsigned)G;
        v[k] = in[k] ? __ldg(g4 + ((size_t)jx * G + jy) * G + jz) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (!in[k]) continue;
        const float w = __fmul_rn(__fmul_rn(wx[k >> 2], wy[(k >> 1) & 1]), wz[k & 1]);
        sx = __fadd_rn(sx, __fmul_rn(w, v[k].x));
        sy = __fadd_rn(sy, __fmul_rn(w, v[k].y));
        sz = __fadd_rn(sz, __fmul_rn(w, v[k].z));
      }
    }
    ax[p] = sx;
    ay[p] = sy;
    az[p] = sz;
  }
}

extern "C" int gc_gather_accel(gc_ctx *ctx, const float *x, const float *y, const float *z, int64_t n,
                               const float *ax_g, const float *ay_g, const float *az_g, float *acc_x, float *acc_y,
                               float *acc_z) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range");
  if (n == 0) return GC_OK;
  GC_REQUIRE(ctx, x && y && z && ax_g && ay_g && az_g && acc_x && acc_y && acc_z, "gc_gather_accel: NULL pointer");
  unsigned nb = gc_blocks(n, 256);
  if (nb > gc_sms() * 32u) nb = gc_sms() * 32u;
  const size_t nodes = (size_t)ctx->G * ctx->G * ctx->G;
  void *own = nullptr;
  if (n >= PACK_MIN && (size_t)n >= nodes / 8) gc_scratch_get(ctx, nodes * sizeof(float4) + 16, &own);
  float4 *g4 = (float4 *)own;
  int *scattered = own ? reinterpret_cast<int *>(g4 + nodes) : nullptr;
  gc_launch_after(ctx, GK_GATHER, k_gather, dim3(nb), dim3(256), 0, x, y, z, (long long)n, ax_g, ay_g, az_g, acc_x, acc_y,
                  acc_z, (float)ctx->dx, ctx->G, g4, scattered);
  if (own) {
    gc_launch_after(ctx, GK_GATHER, k_gather_packed, dim3(std::min(nb, gc_sms() * 16u)), dim3(256), 0, x, y, z, (long long)n,
                    (const int *)scattered, (const float4 *)g4, acc_x, acc_y, acc_z, (float)ctx->dx, ctx->G);
    gc_scratch_put(ctx, own);
  }
  GC_LAUNCH_CHECK(ctx, "gather");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// kick / drift (integrator.py:27-59)
// ------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_axpy3(float *__restrict__ u, float *__restrict__ v, float *__restrict__ w,
                                               const float *__restrict__ a, const float *__restrict__ b,
                                               const float *__restrict__ c, long long n, float dt) {
  gc_after();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    u[p] = __fadd_rn(u[p], __fmul_rn(a[p], dt));
    v[p] = __fadd_rn(v[p], __fmul_rn(b[p], dt));
    w[p] = __fadd_rn(w[p], __fmul_rn(c[p], dt));
  }
}

// The same on four particles a thread (arrays on 16-byte boundaries): all loads of the
// three components in flight together, where one particle a thread leaves the copy rate
// at 5.0 TB/s (10M particles 72 us, 51 so).
__global__ void __launch_bounds__(256)
    k_axpy3x4(float4 *__restrict__ u, float4 *__restrict__ v, float4 *__restrict__ w, const float4 *__restrict__ a,
              const float4 *__restrict__ b, const float4 *__restrict__ c, long long n, float dt) {
  gc_after();
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (4 * p + 3 < n) {
    float4 U = u[p], V = v[p], W = w[p];
    const float4 A = a[p], B = b[p], C = c[p];
    U.x = __fadd_rn(U.x, __fmul_rn(A.x, dt)); U.y = __fadd_rn(U.y, __fmul_rn(A.y, dt));
    U.z = __fadd_rn(U.z, __fmul_rn(A.z, dt)); U.w = __fadd_rn(U.w, __fmul_rn(A.w, dt));
    V.x = __fadd_rn(V.x, __fmul_rn(B.x, dt)); V.y = __fadd_rn(V.y, __fmul_rn(B.y, dt));
    V.z = __fadd_rn(V.z, __fmul_rn(B.z, dt)); V.w = __fadd_rn(V.w, __fmul_rn(B.w, dt));
    W.x = __fadd_rn(W.x, __fmul_rn(C.x, dt)); W.y = __fadd_rn(W.y, __fmul_rn(C.y, dt));
    W.z = __fadd_rn(W.z, __fmul_rn(C.z, dt)); W.w = __fadd_rn(W.w, __fmul_rn(C.w, dt));
    u[p] = U; v[p] = V; w[p] = W;
  } else if (4 * p < n) {
    for (long long i = 4 * p; i < n; ++i) {
      float *uf = reinterpret_cast<float *>(u), *vf = reinterpret_cast<float *>(v), *wf = reinterpret_cast<float *>(w);
      const float *af = reinterpret_cast<const float *>(a), *bf = reinterpret_cast<const float *>(b),
                  *cf = reinterpret_cast<const float *>(c);
      uf[i] = __fadd_rn(uf[i], __fmul_rn(af[i], dt));
      vf[i] = __fadd_rn(vf[i], __fmul_rn(bf[i], dt));
      wf[i] = __fadd_rn(wf[i], __fmul_rn(cf[i], dt));
    }
  }
}

static int axpy3(gc_ctx *ctx, float *u, float *v, float *w, const float *a, const float *b, const float *c,
                 int64_t n, float dt, const char *what) {
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range");
  if (n == 0) return GC_OK;
  GC_REQUIRE(ctx, u && v && w && a && b && c, "%s: NULL pointer", what);
  const uintptr_t all = (uintptr_t)u | (uintptr_t)v | (uintptr_t)w | (uintptr_t)a | (uintptr_t)b | (uintptr_t)c;
  if ((all & 15) == 0) {
    gc_launch_after(ctx, GK_AXPY, k_axpy3x4, dim3(gc_blocks((n + 3) / 4, 256)), dim3(256), 0, reinterpret_cast<float4 *>(u),
              reinterpret_cast<float4 *>(v), reinterpret_cast<float4 *>(w), reinterpret_cast<const float4 *>(a),
              reinterpret_cast<const float4 *>(b), reinterpret_cast<const float4 *>(c), (long long)n, dt);
  } else {
    unsigned nb = gc_blocks(n, 256);
    if (nb > gc_sms() * 32u) nb = gc_sms() * 32u;
    gc_launch_after(ctx, GK_AXPY, k_axpy3, dim3(nb), dim3(256), 0, u, v, w, a, b, c, (long long)n, dt);
  }
  GC_LAUNCH_CHECK(ctx, what);
  return GC_OK;
}

extern "C" int gc_kick(gc_ctx *ctx, float *vx, float *vy, float *vz, const float *ax, const float *ay, const float *az,
                       int64_t n, float dt) {
  if (!ctx) return GC_ERR_ARG;
  return axpy3(ctx, vx, vy, vz, ax, ay, az, n, dt, "kick");
}

extern "C" int gc_drift(gc_ctx *ctx, float *px, float *py, float *pz, const float *vx, const float *vy,
                        const float *vz, int64_t n, float dt) {
  if (!ctx) return GC_ERR_ARG;
  return axpy3(ctx, px, py, pz, vx, vy, vz, n, dt, "drift");
}

// ------------------------------------------------------------------------------
// fused: gather of -grad(phi) computed on the fly + KDK kicks + drift
// ------------------------------------------------------------------------------
struct FusedCtx {
  float dx, inv_dx, inv_2dx;
  int G;
  float h, dt;
  int mode;
  int diag;
};

// Acceleration at a particle: the CIC gather of the node field g = -grad(phi),
// each node's g formed exactly as _potential_to_accel does (deposit.py:148-174).
__device__ __forceinline__ void gather_grad(const float *__restrict__ phi, float x, float y, float z,
                                            const FusedCtx &f, float &ax, float &ay, float &az) {
  ax = ay = az = 0.0f;
  CellPos c;
  if (!gc_cell_of(x, y, z, f.dx, f.G, c)) return;
  const int G = f.G;
  const size_t sG = (size_t)G;
  const float wx[2] = {__fsub_rn(1.0f, c.fx), c.fx};
  const float wy[2] = {__fsub_rn(1.0f, c.fy), c.fy};
  const float wz[2] = {__fsub_rn(1.0f, c.fz), c.fz};
#pragma unroll
  for (int cx = 0; cx < 2; ++cx)
#pragma unroll
    for (int cy = 0; cy < 2; ++cy)
#pragma unroll
      for (int cz = 0; cz < 2; ++cz) {
        const int jx = c.ix + cx, jy = c.iy + cy, jz = c.iz + cz;
        if ((unsigned)jx < (unsigned)G && (unsigned)jy < (unsigned)G && (unsigned)jz < (unsigned)G) {
          const size_t idx = ((size_t)jx * sG + jy) * sG + jz;
          const float gx = grad_comp(phi, idx, sG * sG, jx, G, f.inv_dx, f.inv_2dx);
          const float gy = grad_comp(phi, idx, sG, jy, G, f.inv_dx, f.inv_2dx);
          const float gz = grad_comp(phi, idx, 1, jz, G, f.inv_dx, f.inv_2dx);
          const float w = __fmul_rn(__fmul_rn(wx[cx], wy[cy]), wz[cz]);
          ax = __fadd_rn(ax, __fmul_rn(w, gx));
          ay = __fadd_rn(ay, __fmul_rn(w, gy));
          az = __fadd_rn(az, __fmul_rn(w, gz));
        }
      }
}

// Per-thread diagnostic sums (diagnostics_device.py:56-74: M, KE, P, L, M x) in
// double-float: every product of f32 state is formed exactly (TwoProduct with an
// FMA) or to ~2^-46, and accumulated as an unevaluated sum hi + lo (Knuth's
// TwoSum), all in FP32 instructions; the per-thread totals go to FP64 for the
// block and grid reductions. FP64 arithmetic per particle would run at a small
// fraction of the FP32 rate on this part (it cost ~4 ms per 100M particles).
struct DiagAcc {
  float h[11], l[11];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int t = 0; t < 11; ++t) h[t] = l[t] = 0.0f;
  }
  // exact a*b = p + e
  static __device__ __forceinline__ void tp(float a, float b, float &p, float &e) {
    p = __fmul_rn(a, b);
    e = __fmaf_rn(a, b, -p);
  }
  // exact a+b = s + e
  static __device__ __forceinline__ void ts(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  }
  __device__ __forceinline__ void add(int t, float ph, float pl) {
    float s, e;
    ts(h[t], ph, s, e);
    h[t] = s;
    l[t] = __fadd_rn(l[t], __fadd_rn(e, pl));
  }
  // m (a*b - c*d) to ~2^-46 relative
  static __device__ __forceinline__ void cross(float m, float a, float b, float c, float d, float &q, float &ql) {
    float p1, e1, p2, e2, s, r, qe;
    tp(a, b, p1, e1);
    tp(c, d, p2, e2);
    ts(p1, -p2, s, r);
    const float sl = __fadd_rn(r, __fsub_rn(e1, e2));
    tp(s, m, q, qe);
    ql = __fmaf_rn(sl, m, qe);
  }
  __device__ __forceinline__ void particle(float m, float X, float Y, float Z, float VX, float VY, float VZ) {
    float p, e, q, ql;
    add(0, m, 0.0f);
    {  // 0.5 m |v|^2
      float a1, e1, a2, e2, a3, e3, s1, r1, s2, r2, qe;
      tp(VX, VX, a1, e1);
      tp(VY, VY, a2, e2);
      tp(VZ, VZ, a3, e3);
      ts(a1, a2, s1, r1);
      ts(s1, a3, s2, r2);
      const float sl = __fadd_rn(__fadd_rn(__fadd_rn(e1, e2), e3), __fadd_rn(r1, r2));
      tp(s2, m, q, qe);
      ql = __fmaf_rn(sl, m, qe);
      add(1, __fmul_rn(0.5f, q), __fmul_rn(0.5f, ql));
    }
    tp(m, VX, p, e); add(2, p, e);
    tp(m, VY, p, e); add(3, p, e);
    tp(m, VZ, p, e); add(4, p, e);
    cross(m, Y, VZ, Z, VY, q, ql); add(5, q, ql);
    cross(m, Z, VX, X, VZ, q, ql); add(6, q, ql);
    cross(m, X, VY, Y, VX, q, ql); add(7, q, ql);
    tp(m, X, p, e); add(8, p, e);
    tp(m, Y, p, e); add(9, p, e);
    tp(m, Z, p, e); add(10, p, e);
  }
  __device__ __forceinline__ void to_double(double (&dv)[11]) const {
#pragma unroll
    for (int t = 0; t < 11; ++t) dv[t] = (double)h[t] + (double)l[t];
  }
};

template <bool DIAG>
__global__ void __launch_bounds__(256)
    k_gather_kick_drift(float *__restrict__ x, float *__restrict__ y, float *__restrict__ z, float *__restrict__ vx,
                        float *__restrict__ vy, float *__restrict__ vz, const float *__restrict__ m, long long n,
                        const float *__restrict__ phi, FusedCtx f, float *__restrict__ axo, float *__restrict__ ayo,
                        float *__restrict__ azo, double *__restrict__ parts) {
  DiagAcc acc;
  acc.zero();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    float px = x[p], py = y[p], pz = z[p];
    float ux = vx[p], uy = vy[p], uz = vz[p];
    float ax, ay, az;
    gather_grad(phi, px, py, pz, f, ax, ay, az);
    if (axo) {
      axo[p] = ax;
      ayo[p] = ay;
      azo[p] = az;
    }
    if (f.mode != GC_STEP_PRIME) {  // closing half-kick of the previous step (integrator.py:131)
      ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
      uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
      uz = __fadd_rn(uz, __fmul_rn(az, f.h));
    }
    if (DIAG) {  // synchronised state (diagnostics_device.py:56-74)
      acc.particle(m[p], px, py, pz, ux, uy, uz);
    }
    if (f.mode != GC_STEP_CLOSE) {  // opening half-kick + drift (integrator.py:128-129)
      ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
      uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
      uz = __fadd_rn(uz, __fmul_rn(az, f.h));
      x[p] = __fadd_rn(px, __fmul_rn(ux, f.dt));
      y[p] = __fadd_rn(py, __fmul_rn(uy, f.dt));
      z[p] = __fadd_rn(pz, __fmul_rn(uz, f.dt));
    }
    vx[p] = ux;
    vy[p] = uy;
    vz[p] = uz;
  }
  if (DIAG) {
    double dv[11];
    acc.to_double(dv);
    block_partials<11>(dv, parts + (size_t)blockIdx.x * 11);
  }
}

// Variant with the node field g = -grad(phi) precomputed as float4 (x, y, z, 0):
// one pass over phi writes it (k_grad4), then each particle reads its 8 corner
// nodes with one 16-byte load each. Same arithmetic as gather_grad.
__global__ void __launch_bounds__(256) k_grad4(const float *__restrict__ phi, float4 *__restrict__ g4, GradCtx g) {
  gc_after();
  const int k = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y;
  const int i = blockIdx.z;
  if (k >= g.G || j >= g.G) return;
  const size_t G = g.G;
  const size_t c = ((size_t)i * G + j) * G + k;
  g4[c] = make_float4(grad_comp(phi, c, G * G, i, g.G, g.inv_dx, g.inv_2dx),
                      grad_comp(phi, c, G, j, g.G, g.inv_dx, g.inv_2dx),
                      grad_comp(phi, c, 1, k, g.G, g.inv_dx, g.inv_2dx), 0.0f);
}

template <bool POW2>
__device__ __forceinline__ void gather_g4(const float4 *__restrict__ g4, float x, float y, float z, const FusedCtx &f,
                                          float &ax, float &ay, float &az) {
  ax = ay = az = 0.0f;
  CellPos c;
  if (POW2) {  // x / dx == x * (1/dx) exactly when dx is a power of two
    const float gx = __fmul_rn(x, f.inv_dx), gy = __fmul_rn(y, f.inv_dx), gz = __fmul_rn(z, f.inv_dx);
    const float hi = (float)f.G;
    if (!(gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi)) return;
    const float flx = floorf(gx), fly = floorf(gy), flz = floorf(gz);
    c.ix = (int)flx; c.iy = (int)fly; c.iz = (int)flz;
    c.fx = __fsub_rn(gx, flx); c.fy = __fsub_rn(gy, fly); c.fz = __fsub_rn(gz, flz);
  } else if (!gc_cell_of(x, y, z, f.dx, f.G, c)) {
    return;
  }
  const int G = f.G;
  const float wx[2] = {__fsub_rn(1.0f, c.fx), c.fx};
  const float wy[2] = {__fsub_rn(1.0f, c.fy), c.fy};
  const float wz[2] = {__fsub_rn(1.0f, c.fz), c.fz};
  const bool interior = c.ix >= 0 && c.iy >= 0 && c.iz >= 0 && c.ix + 1 < G && c.iy + 1 < G && c.iz + 1 < G;
  const int base = (c.ix * G + c.iy) * G + c.iz;  // G^3 < 2^31 (G <= 1024)
#pragma unroll
  for (int cx = 0; cx < 2; ++cx)
#pragma unroll
    for (int cy = 0; cy < 2; ++cy)
#pragma unroll
      for (int cz = 0; cz < 2; ++cz) {
        const int jx = c.ix + cx, jy = c.iy + cy, jz = c.iz + cz;
        if (interior || ((unsigned)jx < (unsigned)G && (unsigned)jy < (unsigned)G && (unsigned)jz < (unsigned)G)) {
          const float4 gv = __ldg(g4 + base + (cx * G + cy) * G + cz);
          const float w = __fmul_rn(__fmul_rn(wx[cx], wy[cy]), wz[cz]);
          ax = __fadd_rn(ax, __fmul_rn(w, gv.x));
          ay = __fadd_rn(ay, __fmul_rn(w, gv.y));
          az = __fadd_rn(az, __fmul_rn(w, gv.z));
        }
      }
}

// One particle of the fused pass (closing half-kick, diagnostics, opening
// half-kick, drift) given its acceleration; writes back x, v.
template <bool DIAG>
__device__ __forceinline__ void kd_update(long long p, float px, float py, float pz, float ux, float uy, float uz,
                                          float ax, float ay, float az, float *__restrict__ x, float *__restrict__ y,
                                          float *__restrict__ z, float *__restrict__ vx, float *__restrict__ vy,
                                          float *__restrict__ vz, const float *__restrict__ m, const FusedCtx &f,
                                          DiagAcc &acc) {
  if (f.mode != GC_STEP_PRIME) {
    ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
    uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
    uz = __fadd_rn(uz, __fmul_rn(az, f.h));
  }
  if (DIAG) {
    acc.particle(m[p], px, py, pz, ux, uy, uz);
  }
  if (f.mode != GC_STEP_CLOSE) {
    ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
    uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
    uz = __fadd_rn(uz, __fmul_rn(az, f.h));
    x[p] = __fadd_rn(px, __fmul_rn(ux, f.dt));
    y[p] = __fadd_rn(py, __fmul_rn(uy, f.dt));
    z[p] = __fadd_rn(pz, __fmul_rn(uz, f.dt));
  }
  vx[p] = ux;
  vy[p] = uy;
  vz[p] = uz;
}

template <bool DIAG, bool POW2>
__global__ void __launch_bounds__(256)
    k_gather4_kick_drift(float *__restrict__ x, float *__restrict__ y, float *__restrict__ z, float *__restrict__ vx,
                         float *__restrict__ vy, float *__restrict__ vz, const float *__restrict__ m, long long n,
                         const float4 *__restrict__ g4, FusedCtx f, double *__restrict__ parts) {
  DiagAcc acc;
  acc.zero();
  // software pipelined: the next particle's state is loaded before this one's
  // corner gather, so its DRAM latency overlaps the gather's L2 latency
  const long long stride = (long long)gridDim.x * blockDim.x;
  long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  float nx = 0.0f, ny = 0.0f, nz = 0.0f, nvx = 0.0f, nvy = 0.0f, nvz = 0.0f;
  if (p < n) { nx = x[p]; ny = y[p]; nz = z[p]; nvx = vx[p]; nvy = vy[p]; nvz = vz[p]; }
  for (; p < n; p += stride) {
    const float px = nx, py = ny, pz = nz, ux = nvx, uy = nvy, uz = nvz;
    const long long q = p + stride;
    if (q < n) { nx = x[q]; ny = y[q]; nz = z[q]; nvx = vx[q]; nvy = vy[q]; nvz = vz[q]; }
    float ax, ay, az;
    gather_g4<POW2>(g4, px, py, pz, f, ax, ay, az);
    kd_update<DIAG>(p, px, py, pz, ux, uy, uz, ax, ay, az, x, y, z, vx, vy, vz, m, f, acc);
  }
  if (DIAG) {
    double dv[11];
    acc.to_double(dv);
    block_partials<11>(dv, parts + (size_t)blockIdx.x * 11);
  }
}

// The same particle pass with the particle state streamed by the TMA engine: a
// CTA owns tiles of GT_TILE particles (round robin); one thread arms an
// mbarrier and issues 1-D bulk copies (x, y, z, vx, vy, vz, and m when
// depositing) of the next tile into the other half of a double buffer while all
// threads work on the current one, reading the state from shared memory,
// gathering the corners from the float4 grid, and writing the new state back in
// place; the tile then leaves with six bulk stores. The DRAM streams never wait
// for the gather's dependent loads.
//
// With DEP the pass also deposits the drifted positions (the next step's
// density) into the int64 grid while the stores drain: warp w takes the tile's
// particles [128 w, 128 w + 128) 32 at a time, exactly as k_deposit_sorted does
// (two full-warp reductions for the main cells, direct adds for the others, a
// per-warp shared-memory box), so the density is the one k_deposit_sorted
// would produce from the stored positions, bit for bit.
//
// Full tiles only; the remainder goes through plain loads (and per-particle
// deposits). Waits are bounded (clock budget): a timeout raises
// GC_FLAG_TIMEOUT and the CTA stops issuing.
#define GT_TILE 1024
#define GT_BUDGET 2000000000LL
#define GT_WBOX 512  // nodes of one warp's deposit box
// dynamic shared memory: two buffers of 7 arrays, the warps' boxes
#define GT_SMEM(dep) (2 * ((dep) ? 7 : 6) * GT_TILE * 4 + ((dep) ? 8 * GT_WBOX * 4 : 0))

template <bool POW2>
__device__ __forceinline__ void gt_particle(float *s0, float *s1, float *s2, float *s3, float *s4, float *s5, int i,
                                            const float4 *__restrict__ g4, const FusedCtx &f) {
  const float px = s0[i], py = s1[i], pz = s2[i];
  float ux = s3[i], uy = s4[i], uz = s5[i];
  float ax, ay, az;
  gather_g4<POW2>(g4, px, py, pz, f, ax, ay, az);
  if (f.mode != GC_STEP_PRIME) {
    ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
    uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
    uz = __fadd_rn(uz, __fmul_rn(az, f.h));
  }
  if (f.mode != GC_STEP_CLOSE) {
    ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
    uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
    uz = __fadd_rn(uz, __fmul_rn(az, f.h));
    s0[i] = __fadd_rn(px, __fmul_rn(ux, f.dt));
    s1[i] = __fadd_rn(py, __fmul_rn(uy, f.dt));
    s2[i] = __fadd_rn(pz, __fmul_rn(uz, f.dt));
  }
  s3[i] = ux;
  s4[i] = uy;
  s5[i] = uz;
}

// Deposit of 128 staged particles (warp-contiguous, the k_deposit_sorted rules)
// into the warp's box or the grid.
template <bool POW2>
__device__ __forceinline__ void gt_deposit_warp(const float *s0, const float *s1, const float *s2, const float *s6,
                                                int base, int *wbox, const DepCtx &d, float inv_dx, float qscale,
                                                long long *__restrict__ qg, unsigned *__restrict__ status, int lane) {
  float px[4], py[4], pz[4], pm[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = base + 32 * j + lane;
    px[j] = s0[i]; py[j] = s1[i]; pz[j] = s2[i]; pm[j] = s6[i];
  }
  DepBox bx;
  bx.b = wbox;
  bool use_box;
  int nx;
  {
    float xl = 3.0e38f, yl = 3.0e38f, zl = 3.0e38f, xh = -3.0e38f, yh = -3.0e38f, zh = -3.0e38f;
    unsigned mb = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      xl = fminf(xl, px[j]); xh = fmaxf(xh, px[j]);
      yl = fminf(yl, py[j]); yh = fmaxf(yh, py[j]);
      zl = fminf(zl, pz[j]); zh = fmaxf(zh, pz[j]);
      mb = max(mb, __float_as_uint(pm[j]) & 0x7fffffffu);
    }
    const float gl = -1.0f, gh = (float)d.G - 1.0f;
    const float cl[3] = {xl, yl, zl}, ch[3] = {xh, yh, zh};
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float l = POW2 ? __fmul_rn(cl[a], inv_dx) : __fdiv_rn(cl[a], d.dx);
      float h = POW2 ? __fmul_rn(ch[a], inv_dx) : __fdiv_rn(ch[a], d.dx);
      l = fminf(fmaxf(floorf(l), gl), gh);
      h = fminf(fmaxf(floorf(h), gl), gh);
      const bool any_pt = cl[a] <= ch[a];
      lo[a] = __reduce_min_sync(0xffffffffu, any_pt ? (int)l : 0x7fffffff);
      hi[a] = __reduce_max_sync(0xffffffffu, any_pt ? (int)h : -0x7fffffff);
    }
    mb = __reduce_max_sync(0xffffffffu, mb);
    bx.x0 = lo[0]; bx.y0 = lo[1]; bx.z0 = lo[2];
    nx = hi[0] - lo[0] + 2;
    bx.ny = hi[1] - lo[1] + 2;
    bx.nz = hi[2] - lo[2] + 2;
    bx.nyz = bx.ny * bx.nz;
    const float mq = __fmul_rn(__fmul_rn(__uint_as_float(mb), d.inv_vol), qscale);
    use_box = hi[0] >= lo[0] && (long long)nx * bx.nyz <= GT_WBOX &&
              __fmul_rn(fminf(mq, 4194304.0f) + 1.0f, 128.0f) < 1073741824.0f;
  }
  unsigned large = 0;
  const long long nrem = 1LL << 40;  // all 128 particles exist
  if (use_box)
    dep_warp_pass<POW2, true, 4>(px, py, pz, pm, nrem, d, inv_dx, qscale, bx, qg, status, lane, large);
  else
    dep_warp_pass<POW2, false, 4>(px, py, pz, pm, nrem, d, inv_dx, qscale, bx, qg, status, lane, large);
  while (large) {  // rare: point masses
    const int j = __ffs(large) - 1;
    large &= large - 1;
    const int i = base + 32 * j + lane;
    const float gx = POW2 ? __fmul_rn(s0[i], inv_dx) : __fdiv_rn(s0[i], d.dx);
    const float gy = POW2 ? __fmul_rn(s1[i], inv_dx) : __fdiv_rn(s1[i], d.dx);
    const float gz = POW2 ? __fmul_rn(s2[i], inv_dx) : __fdiv_rn(s2[i], d.dx);
    const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
    large_to_grid(qg, d.G, ix, iy, iz, __fmul_rn(s6[i], d.inv_vol), __fsub_rn(gx, __int2float_rn(ix)),
                  __fsub_rn(gy, __int2float_rn(iy)), __fsub_rn(gz, __int2float_rn(iz)), qscale);
  }
  if (use_box) {
    __syncwarp();
    const int vol = nx * bx.nyz;
    for (int i = lane; i < vol; i += 32) {
      const int v = wbox[i];
      if (v == 0) continue;
      wbox[i] = 0;
      const int rx = i / bx.nyz, rem = i - rx * bx.nyz, ry = rem / bx.nz, rz = rem - ry * bx.nz;
      const int jx = bx.x0 + rx, jy = bx.y0 + ry, jz = bx.z0 + rz;
      if ((unsigned)jx < (unsigned)d.G && (unsigned)jy < (unsigned)d.G && (unsigned)jz < (unsigned)d.G)
        atomicAdd((unsigned long long *)(qg + ((size_t)jx * d.G + jy) * d.G + jz), (unsigned long long)(long long)v);
    }
    __syncwarp();
  }
}

// One particle of the remainder: its corners straight to the grid.
template <bool POW2>
__device__ __forceinline__ void gt_deposit_one(float px, float py, float pz, float pm, const DepCtx &d, float inv_dx,
                                               float qscale, long long *__restrict__ qg,
                                               unsigned *__restrict__ status) {
  float gx, gy, gz;
  if (POW2) {
    gx = __fmul_rn(px, inv_dx); gy = __fmul_rn(py, inv_dx); gz = __fmul_rn(pz, inv_dx);
  } else {
    gx = __fdiv_rn(px, d.dx); gy = __fdiv_rn(py, d.dx); gz = __fdiv_rn(pz, d.dx);
  }
  const float hi = (float)d.G;
  if (!(gx >= -1.0f && gx < hi && gy >= -1.0f && gy < hi && gz >= -1.0f && gz < hi)) {
    if (!gc_finite3(px, py, pz)) atomicOr(status, GC_FLAG_NONFINITE_POS);
    return;
  }
  const int ix = __float2int_rd(gx), iy = __float2int_rd(gy), iz = __float2int_rd(gz);
  const float fx = __fsub_rn(gx, __int2float_rn(ix)), fy = __fsub_rn(gy, __int2float_rn(iy)),
              fz = __fsub_rn(gz, __int2float_rn(iz));
  large_to_grid(qg, d.G, ix, iy, iz, __fmul_rn(pm, d.inv_vol), fx, fy, fz, qscale);
}

template <bool POW2, bool DEP>
__global__ void __launch_bounds__(256)
    k_gather4_tma(float *__restrict__ x, float *__restrict__ y, float *__restrict__ z, float *__restrict__ vx,
                  float *__restrict__ vy, float *__restrict__ vz, const float *__restrict__ m, long long n,
                  const float4 *__restrict__ g4, FusedCtx f, DepCtx d, float inv_dx, const double *__restrict__ qexp,
                  long long *__restrict__ qg, unsigned *__restrict__ status) {
  gc_after();
  using namespace umma;
  constexpr int NA = DEP ? 7 : 6;
  extern __shared__ __align__(128) float gt_smem[];
  float *buf = gt_smem;                               // [2][NA][GT_TILE]
  int *wboxes = reinterpret_cast<int *>(gt_smem + 2 * NA * GT_TILE);  // [8][GT_WBOX] when DEP
  __shared__ __align__(8) uint64_t bar[2];
  const float *src[7] = {x, y, z, vx, vy, vz, m};
  float *const dst[6] = {x, y, z, vx, vy, vz};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long ntiles = n / GT_TILE;
  const float qscale = DEP ? ldexpf(1.0f, -(int)(*qexp)) : 1.0f;
  if (DEP)
    for (int i = tid; i < 8 * GT_WBOX; i += 256) wboxes[i] = 0;  // every flush zeroes what it read
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const uint32_t tile_bytes = GT_TILE * 4;
  long long t = blockIdx.x;
  if (tid == 0 && t < ntiles) {
    mbar_arrive_expect_tx(&bar[0], NA * tile_bytes);
#pragma unroll
    for (int a = 0; a < NA; ++a) bulk_g2s(buf + a * GT_TILE, src[a] + t * GT_TILE, tile_bytes, &bar[0]);
  }
  for (int it = 0; t < ntiles; ++it, t += gridDim.x) {
    const int b = it & 1;
    float *cur = buf + b * NA * GT_TILE, *nxt = buf + (b ^ 1) * NA * GT_TILE;
    const long long tn = t + gridDim.x;
    if (tid == 0 && tn < ntiles) {  // prefetch the next tile into the other buffer
      bulk_wait_read_all();          // its previous tile's stores have read it
      mbar_arrive_expect_tx(&bar[b ^ 1], NA * tile_bytes);
#pragma unroll
      for (int a = 0; a < NA; ++a) bulk_g2s(nxt + a * GT_TILE, src[a] + tn * GT_TILE, tile_bytes, &bar[b ^ 1]);
    }
    const bool got = mbar_wait(&bar[b], (uint32_t)(it >> 1) & 1u, GT_BUDGET);
    if (!__syncthreads_and(got)) {  // the block leaves together
      if (tid == 0) {  // record it, and give the copies still in flight a bounded time to land
        atomicOr(status, GC_FLAG_TIMEOUT);
        mbar_wait(&bar[b], (uint32_t)(it >> 1) & 1u, GT_BUDGET);
        if (tn < ntiles) mbar_wait(&bar[b ^ 1], (uint32_t)((it + 1) >> 1) & 1u, GT_BUDGET);
        bulk_wait_all();
      }
      return;
    }
    float *s0 = cur, *s1 = cur + GT_TILE, *s2 = cur + 2 * GT_TILE, *s3 = cur + 3 * GT_TILE, *s4 = cur + 4 * GT_TILE,
          *s5 = cur + 5 * GT_TILE;
#pragma unroll 4
    for (int i = tid; i < GT_TILE; i += 256) gt_particle<POW2>(s0, s1, s2, s3, s4, s5, i, g4, f);
    fence_async_smem();  // this thread's shared-memory writes -> visible to the bulk stores
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int a = 0; a < 6; ++a) bulk_s2g(dst[a] + t * GT_TILE, cur + a * GT_TILE, tile_bytes);
      bulk_commit();
    }
    if (DEP) {  // the drifted positions' density while the stores drain
      gt_deposit_warp<POW2>(s0, s1, s2, cur + 6 * GT_TILE, 128 * warp, wboxes + warp * GT_WBOX, d, inv_dx, qscale,
                            qg, status, lane);
      fence_async_smem();
      __syncthreads();  // the buffer is free for the prefetch of the tile after next
    }
  }
  if (tid == 0) bulk_wait_all();
  // the remainder after the full tiles: plain loads, every CTA a slice
  const long long r0 = ntiles * GT_TILE;
  for (long long p = r0 + blockIdx.x * (long long)blockDim.x + tid; p < n; p += (long long)gridDim.x * blockDim.x) {
    float px = x[p], py = y[p], pz = z[p], ux = vx[p], uy = vy[p], uz = vz[p];
    float ax, ay, az;
    gather_g4<POW2>(g4, px, py, pz, f, ax, ay, az);
    if (f.mode != GC_STEP_PRIME) {
      ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
      uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
      uz = __fadd_rn(uz, __fmul_rn(az, f.h));
    }
    if (f.mode != GC_STEP_CLOSE) {
      ux = __fadd_rn(ux, __fmul_rn(ax, f.h));
      uy = __fadd_rn(uy, __fmul_rn(ay, f.h));
      uz = __fadd_rn(uz, __fmul_rn(az, f.h));
      px = __fadd_rn(px, __fmul_rn(ux, f.dt));
      py = __fadd_rn(py, __fmul_rn(uy, f.dt));
      pz = __fadd_rn(pz, __fmul_rn(uz, f.dt));
      x[p] = px;
      y[p] = py;
      z[p] = pz;
    }
    vx[p] = ux;
    vy[p] = uy;
    vz[p] = uz;
    if (DEP) gt_deposit_one<POW2>(px, py, pz, m[p], d, inv_dx, qscale, qg, status);
  }
}

int gc_gather_kick_drift(gc_ctx *ctx, const gc_particles *p, float dt, int mode, int diag, int grad_grid,
                         int deposit_next, float *axo, float *ayo, float *azo, int *nparts_out, int *deposited) {
  if (deposited) *deposited = 0;
  FusedCtx f;
  f.dx = (float)ctx->dx;
  f.inv_dx = 1.0f / f.dx;
  f.inv_2dx = 1.0f / (2.0f * f.dx);
  f.G = ctx->G;
  f.dt = dt;
  f.h = 0.5f * dt;
  f.mode = mode;
  f.diag = diag;
  unsigned nb = gc_blocks(p->n, 256);
  if (nb > gc_sms() * 16u) nb = gc_sms() * 16u;
  int s = gc_ensure_red(ctx, (size_t)nb * 11);
  if (s) return s;
  if (grad_grid && !axo) {
    const size_t g3 = (size_t)ctx->G * ctx->G * ctx->G;
    if (!ctx->g4) GC_CUDA(ctx, cudaMalloc(&ctx->g4, g3 * sizeof(float4)));
    const GradCtx g = make_grad(ctx);
    gc_launch_after(ctx, GK_GRAD, k_grad4, dim3(gc_blocks(g.G, 32), gc_blocks(g.G, 8), g.G), dim3(32, 8), 0, ctx->hi,
              (float4 *)ctx->g4, g);
    int fe = 0;
    const bool pow2 = std::frexp(f.dx, &fe) == 0.5f;  // then inv_dx is exact
    const uintptr_t al = (uintptr_t)p->x | (uintptr_t)p->y | (uintptr_t)p->z | (uintptr_t)p->vx | (uintptr_t)p->vy |
                         (uintptr_t)p->vz;
    const bool dep = deposit_next && mode != GC_STEP_CLOSE && ((uintptr_t)p->m & 15u) == 0;
    if (!diag && (al & 15u) == 0 && p->n >= GT_TILE) {
      if (!ctx->gt_smem_set) {  // opt in to more than 48 KB of dynamic shared memory (once per context)
        GC_CUDA(ctx, cudaFuncSetAttribute(k_gather4_tma<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM(false)));
        GC_CUDA(ctx, cudaFuncSetAttribute(k_gather4_tma<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM(false)));
        GC_CUDA(ctx, cudaFuncSetAttribute(k_gather4_tma<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM(true)));
        GC_CUDA(ctx, cudaFuncSetAttribute(k_gather4_tma<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GT_SMEM(true)));
        ctx->gt_smem_set = 1;
      }
      // bulk-streamed state, persistent: 4 CTAs per SM (3 when depositing: 72 KB each)
      const long long ntiles = p->n / GT_TILE;
      const long long per_sm = dep ? 3 : 4;
      const unsigned nbt = (unsigned)(ntiles < (long long)gc_sms() * per_sm ? ntiles : (long long)gc_sms() * per_sm);
      DepCtx d;
      d.dx = (float)ctx->dx;
      d.inv_vol = 1.0f / ((d.dx * d.dx) * d.dx);
      d.G = ctx->G;
      const float inv_dx_dep = pow2 ? std::ldexp(1.0f, 1 - fe) : 0.0f;
      auto k = dep ? (pow2 ? k_gather4_tma<true, true> : k_gather4_tma<false, true>)
                   : (pow2 ? k_gather4_tma<true, false> : k_gather4_tma<false, false>);
      gc_launch_after(ctx, GK_GATHER_KD, k, dim3(nbt), dim3(256), GT_SMEM(dep), p->x, p->y, p->z, p->vx, p->vy, p->vz, p->m,
                (long long)p->n, (const float4 *)ctx->g4, f, d, inv_dx_dep, (const double *)(ctx->dsmall + GC_S_QEXP_PM),
                ctx->q, ctx->dstatus);
      if (dep && deposited) *deposited = 1;
    } else {
      auto k = diag ? (pow2 ? k_gather4_kick_drift<true, true> : k_gather4_kick_drift<true, false>)
                    : (pow2 ? k_gather4_kick_drift<false, true> : k_gather4_kick_drift<false, false>);
      gc_launch(ctx, GK_GATHER_KD, k, dim3(nb), dim3(256), 0, p->x, p->y, p->z, p->vx, p->vy, p->vz, p->m,
                (long long)p->n, (const float4 *)ctx->g4, f, ctx->red);
    }
  } else if (diag) {
    gc_launch(ctx, GK_GATHER_KD, k_gather_kick_drift<true>, dim3(nb), dim3(256), 0, p->x, p->y, p->z, p->vx, p->vy,
              p->vz, p->m, (long long)p->n, ctx->hi, f, axo, ayo, azo, ctx->red);
  } else {
    gc_launch(ctx, GK_GATHER_KD, k_gather_kick_drift<false>, dim3(nb), dim3(256), 0, p->x, p->y, p->z, p->vx, p->vy,
              p->vz, p->m, (long long)p->n, ctx->hi, f, axo, ayo, azo, ctx->red);
  }
  GC_LAUNCH_CHECK(ctx, "gather_kick_drift");
  if (nparts_out) *nparts_out = (int)nb;
  return GC_OK;
}

// ------------------------------------------------------------------------------
// diagnostics (diagnostics_device.py)
// ------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_diag_particles(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                     const float *__restrict__ vx, const float *__restrict__ vy, const float *__restrict__ vz,
                     const float *__restrict__ m, long long n, double *__restrict__ parts) {
  DiagAcc acc;
  acc.zero();
  // two particles' loads in flight ahead of the sums (about 180 FP32 instructions a
  // particle: they bound this kernel, not the 28 bytes; 10M particles 127 -> 86 us)
  const long long T = (long long)gridDim.x * blockDim.x;
  long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  float a[7], b[7];
  auto load = [&](float (&v)[7], long long q) {
    const float *const src[7] = {m, x, y, z, vx, vy, vz};
#pragma unroll
    for (int i = 0; i < 7; ++i) v[i] = q < n ? src[i][q] : 0.0f;
  };
  load(a, p);
  load(b, p + T);
  for (; p < n; p += 2 * T) {
    float c[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) c[i] = a[i];
    load(a, p + 2 * T);
    acc.particle(c[0], c[1], c[2], c[3], c[4], c[5], c[6]);
    if (p + T >= n) break;
#pragma unroll
    for (int i = 0; i < 7; ++i) c[i] = b[i];
    load(b, p + 3 * T);
    acc.particle(c[0], c[1], c[2], c[3], c[4], c[5], c[6]);
  }
  double dv[11];
  acc.to_double(dv);
  block_partials<11>(dv, parts + (size_t)blockIdx.x * 11);
}

extern "C" int gc_diag_particles(gc_ctx *ctx, const float *x, const float *y, const float *z, const float *vx,
                                 const float *vy, const float *vz, const float *m, int64_t n, double out[11]) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, out, "gc_diag_particles: NULL out");
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range");
  GC_REQUIRE(ctx, n == 0 || (x && y && z && vx && vy && vz && m), "gc_diag_particles: NULL pointer");
  int nb = (int)gc_blocks(n, 512);
  if (nb > (int)gc_sms() * 4) nb = (int)gc_sms() * 4;  // the same number of blocks on every SM
  int s = gc_ensure_red(ctx, (size_t)nb * 11);
  if (s) return s;
  gc_launch(ctx, GK_DIAG, k_diag_particles, dim3(nb), dim3(256), 0, x, y, z, vx, vy, vz, m, (long long)n, ctx->red);
  GC_LAUNCH_CHECK(ctx, "diag particles");
  if ((s = gc_finalize(ctx, ctx->red, nb, 11, ctx->ddiag))) return s;
  GC_CUDA(ctx, cudaMemcpyAsync(out, ctx->ddiag, 11 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GC_OK;
}

// Sum of a*b. FP64 warp instructions take 16 clocks of the SM on this part, so DOT_U
// products of a thread are first summed in FP32 as an unevaluated three-part sum
// (products by FMA, every addition by TwoSum: exact but for terms below 2^-70 of the
// largest), and only its parts go to the thread's FP64 sum. Bound by HBM: 134 MB at
// 256^3, 105 us with a conversion and an FP64 multiply-add per element, 34 us now.
//
// The error terms of products below 2^-126 are cut off at 2^-149, too coarse where the
// largest is below 1e-20; such products, and ones beyond 1e30, are summed again
// with both factors scaled to about 1 by powers of two, and in FP64 only what is still out
// of range (no largest of 1e-20 of the factors', infinities, NaN). The call at 256^3: 62 us, 88
// where every product is scaled; 161 where FP64 took those from memory, 136 in FP64 throughout.
#define DOT_U 16
// The three parts of the sum of x * y, or of sx x * sy y; false where they are not exact enough.
template <bool SCALED>
__device__ __forceinline__ bool dot_parts(const float (&x)[DOT_U], const float (&y)[DOT_U], float sx, float sy, float &h,
                                          float &m, float &l) {
  float big = 0.0f;
  h = m = l = 0.0f;
#pragma unroll
  for (int u = 0; u < DOT_U; ++u) {
    const float xs = SCALED ? __fmul_rn(x[u], sx) : x[u], ys = SCALED ? __fmul_rn(y[u], sy) : y[u];
    const float p = __fmul_rn(xs, ys), pe = __fmaf_rn(xs, ys, -p);
    float e, f, g;
    df_two_sum(h, p, h, e);
    df_two_sum(m, e, m, f);
    df_two_sum(m, pe, m, g);
    l = __fadd_rn(l, __fadd_rn(f, g));
    big = fmaxf(big, fabsf(p));
  }
  return big >= 1e-20f && big < 1e30f && fabsf(h) < 1e30f;  // (an infinity or a NaN leaves a NaN in h)
}

__device__ __forceinline__ void dot_load(const float *__restrict__ a, const float *__restrict__ b, size_t t0, size_t T,
                                         size_t n, float (&x)[DOT_U], float (&y)[DOT_U]) {
#pragma unroll
  for (int u = 0; u < DOT_U; ++u) {
    const size_t t = t0 + u * T;
    x[u] = t < n ? a[t] : 0.0f;
    y[u] = t < n ? b[t] : 0.0f;
  }
}

// The same products over again (out of line: the ordinary ones keep their registers).
__device__ __noinline__ double dot_again(const float *__restrict__ a, const float *__restrict__ b, size_t t0, size_t T,
                                         size_t n) {
  float x[DOT_U], y[DOT_U];
  dot_load(a, b, t0, T, n, x, y);
  float mx = 0.0f, my = 0.0f;
  bool fin = true;
#pragma unroll
  for (int u = 0; u < DOT_U; ++u) {
    mx = fmaxf(mx, fabsf(x[u]));
    my = fmaxf(my, fabsf(y[u]));
    fin &= fabsf(x[u]) <= 3.402823466e38f && fabsf(y[u]) <= 3.402823466e38f;
  }
  if (fin && (mx == 0.0f || my == 0.0f)) return 0.0;
  const int ex = min(max((int)(__float_as_uint(mx) >> 23), 1), 253), ey = min(max((int)(__float_as_uint(my) >> 23), 1), 253);
  float h, m, l;
  if (dot_parts<true>(x, y, __uint_as_float((unsigned)(254 - ex) << 23), __uint_as_float((unsigned)(254 - ey) << 23), h, m, l))
    return ((double)h + ((double)m + (double)l)) * __longlong_as_double((long long)(ex + ey - 254 + 1023) << 52);
  double s = 0.0;
#pragma unroll 1
  for (int u = 0; u < DOT_U; ++u) {
    const size_t t = t0 + u * T;
    if (t < n) s += (double)a[t] * (double)b[t];
  }
  return s;
}

__global__ void __launch_bounds__(256) k_dot(const float *__restrict__ a, const float *__restrict__ b, size_t n,
                                             double *__restrict__ parts) {
  double acc[1] = {0.0};
  const size_t T = (size_t)gridDim.x * blockDim.x;
  for (size_t t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t0 < n; t0 += DOT_U * T) {
    float x[DOT_U], y[DOT_U], h, m, l;
    dot_load(a, b, t0, T, n, x, y);
    unsigned some = 0;  // any of a: empty stretches are most of a disk's box
#pragma unroll
    for (int u = 0; u < DOT_U; ++u) some |= __float_as_uint(x[u]);
    const bool ok = dot_parts<false>(x, y, 1.0f, 1.0f, h, m, l);
    if (ok || ((some & 0x7fffffffu) == 0 && h == 0.0f)) {
      acc[0] += (double)h;
      acc[0] += (double)m + (double)l;
    } else {
      acc[0] += dot_again(a, b, t0, T, n);
    }
  }
  block_partials<1>(acc, parts + blockIdx.x);
}

int gc_dot_async(gc_ctx *ctx, const float *a, const float *b, size_t n, double *dst) {
  int nb = (int)gc_sms() * 8;
  if ((size_t)nb * 256 * DOT_U > n + 256 * DOT_U) nb = (int)gc_blocks((long long)n, 256 * DOT_U);
  int s = gc_ensure_red(ctx, nb);
  if (s) return s;
  gc_launch(ctx, GK_REDUCE, k_dot, dim3(nb), dim3(256), 0, a, b, n, ctx->red);
  GC_LAUNCH_CHECK(ctx, "dot");
  return gc_finalize(ctx, ctx->red, nb, 1, dst);
}

extern "C" int gc_diag_grid_pe(gc_ctx *ctx, const float *rho, const float *phi, double *out) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, rho && phi && out, "gc_diag_grid_pe: NULL pointer");
  const size_t g3 = (size_t)ctx->G * ctx->G * ctx->G;
  int s = gc_dot_async(ctx, rho, phi, g3, ctx->ddiag + 12);
  if (s) return s;
  GC_CUDA(ctx, cudaMemcpyAsync(out, ctx->ddiag + 12, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GC_OK;
}

// The bin of a particle is floor(r inv_binw) with r in FP64. An FP64 distance costs
// about 40 FP64 warp instructions of 16 clocks each, so the distance is taken in FP32
// first: its relative error is below 12 * 2^-24 (two roundings in each difference, three
// in the squares and their sum, one each in the root, 1/binw and the product), and the
// centre's rounding to FP32 moves it by at most the sum of the three differences. Only
// where a bin edge lies within that margin (or FP32 leaves its range) is the bin
// decided in FP64, so every particle falls in the same bin as before. The masses
// are summed exactly: an addition to FP64 shared memory is a chain of
// compare-and-swaps with an FP64 instruction in each, so a block takes the smallest
// positive mass exponent of its particles, sums masses up to 2^8 times that in units
// of its last place with 32-bit integer additions (carries into a second word), and only
// others in FP64. Masses are added up in FP64 when a block hands in its bins; one
// large block per SM, because all of them contend for the few bins of a disk. Measured
// for 10M particles and 2048 bins: 461 us in FP64 throughout, 117 with FP32 distances
// and FP64 sums (one histogram a block or four), 68 us now.
#define HIST_THREADS 1024
__global__ void __launch_bounds__(HIST_THREADS)
    k_radial_hist(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                  const float *__restrict__ m, long long n, double cx, double cy, double cz, double inv_binw, int nbins,
                  double *__restrict__ hist) {
  extern __shared__ double sh[];  // [nbins] FP64 sums, then the low and high words
  unsigned *lo_w = reinterpret_cast<unsigned *>(sh + nbins), *hi_w = lo_w + nbins;
  __shared__ unsigned emin_s;
  if (threadIdx.x == 0) emin_s = 255u;
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    sh[b] = 0.0;
    lo_w[b] = hi_w[b] = 0u;
  }
  __syncthreads();
  {
    unsigned e = 255u;  // exponent field of the smallest normal positive mass (255: none)
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x) {
      const unsigned u = __float_as_uint(m[p]) >> 23;  // sign and exponent
      if (u >= 1u && u < 255u) e = min(e, u);
    }
    e = __reduce_min_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMin(&emin_s, e);
  }
  __syncthreads();
  const unsigned emin = emin_s;
  const float cxf = (float)cx, cyf = (float)cy, czf = (float)cz, invf = (float)inv_binw;
  const float off = __fmul_ru(
      __fadd_ru(__fadd_ru(__double2float_ru(fabs(cx - (double)cxf)), __double2float_ru(fabs(cy - (double)cyf))),
                __double2float_ru(fabs(cz - (double)czf))),
      __fmul_ru(1.0001f, fabsf(invf)));
  const float nb = (float)nbins;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const float px = x[p], py = y[p], pz = z[p], pm = m[p];
    const float dx = px - cxf, dy = py - cyf, dz = pz - czf;
    const float r2 = dx * dx + dy * dy + dz * dz, f = __fsqrt_rn(r2) * invf;
    const float margin = f * 9.5367431640625e-7f + off;  // 2^-20 f
    const float lo = f - margin, hi = f + margin;
    int b;
    if (r2 > 1e-30f && r2 < 1e30f && invf > 1e-30f && invf < 1e30f && lo >= nb) {
      b = nbins - 1;
    } else if (r2 > 1e-30f && r2 < 1e30f && invf > 1e-30f && invf < 1e30f && hi < nb && floorf(lo) == floorf(hi)) {
      b = (int)lo;
    } else {
      const double rx = (double)px - cx, ry = (double)py - cy, rz = (double)pz - cz;
      const double r = sqrt(rx * rx + ry * ry + rz * rz);
      const double fb = r * inv_binw;
      b = fb >= (double)nbins ? nbins - 1 : (int)fb;
    }
    if (b < 0) b = 0;
    const unsigned u = __float_as_uint(pm), ex = u >> 23, sh_e = ex - emin;  // (wraps for the rest)
    if (sh_e < 8u && ex < 255u) {
      const unsigned q = ((u & 0x7fffffu) | 0x800000u) << sh_e;
      const unsigned old = atomicAdd(&lo_w[b], q);
      if (old + q < old) atomicAdd(&hi_w[b], 1u);
    } else if (pm != 0.0f) {
      atomicAdd(&sh[b], (double)pm);
    }
  }
  __syncthreads();
  const double unit = ldexp(1.0, (int)emin - 150);
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
    const double v = sh[b] + ((double)hi_w[b] * 4294967296.0 + (double)lo_w[b]) * unit;
    if (v != 0.0) atomicAdd(&hist[b], v);
  }
}

extern "C" int gc_radial_histogram(gc_ctx *ctx, const float *x, const float *y, const float *z, const float *m,
                                   int64_t n, double cx, double cy, double cz, double inv_binw, int nbins,
                                   double *hist) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, hist, "gc_radial_histogram: NULL hist");
  GC_REQUIRE(ctx, nbins >= 1 && nbins <= 6144, "nbins must be in [1, 6144]");
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range");
  GC_CUDA(ctx, cudaMemsetAsync(hist, 0, nbins * sizeof(double), ctx->stream));
  if (n == 0) return GC_OK;
  GC_REQUIRE(ctx, x && y && z && m, "gc_radial_histogram: NULL pointer");
  const size_t smem = nbins * (sizeof(double) + 2 * sizeof(unsigned));
  if (smem > 48 * 1024)
    GC_CUDA(ctx, cudaFuncSetAttribute(k_radial_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  unsigned nb = gc_blocks(n, HIST_THREADS);
  if (nb > gc_sms()) nb = gc_sms();
  gc_launch(ctx, GK_HIST, k_radial_hist, dim3(nb), dim3(HIST_THREADS), smem, x, y, z, m, (long long)n, cx, cy, cz,
            inv_binw, nbins, hist);
  GC_LAUNCH_CHECK(ctx, "radial hist");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// headless 2-D projection (viz/project.py:26-46)
// ------------------------------------------------------------------------------
// Nearest-bin mass histogram over two in-plane axes: ia = floor((a - lo_a)/binw_a)
// in f32 as the reference; mass outside [0, bins) is dropped.
__global__ void __launch_bounds__(256)
    k_project_ngp(const float *__restrict__ pa, const float *__restrict__ pb, const float *__restrict__ m, long long n,
                  float lo_a, float lo_b, float bw_a, float bw_b, int bins, float *__restrict__ img) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const float ga = floorf(__fdiv_rn(__fsub_rn(pa[p], lo_a), bw_a));
    const float gb = floorf(__fdiv_rn(__fsub_rn(pb[p], lo_b), bw_b));
    if (!(ga >= 0.0f && ga < (float)bins && gb >= 0.0f && gb < (float)bins)) continue;
    atomicAdd(img + (size_t)(int)ga * bins + (int)gb, m[p]);
  }
}

extern "C" int gc_project_ngp(gc_ctx *ctx, const float *pa, const float *pb, const float *m, int64_t n, double lo_a,
                              double lo_b, double binw_a, double binw_b, int bins, float *img) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, img, "gc_project_ngp: NULL image");
  GC_REQUIRE(ctx, bins >= 1 && bins <= 16384, "bins must be in [1, 16384]");
  GC_REQUIRE(ctx, binw_a > 0.0 && binw_b > 0.0, "bin widths must be positive");
  GC_REQUIRE(ctx, n >= 0 && n < (1LL << 31), "particle count out of range");
  GC_CUDA(ctx, cudaMemsetAsync(img, 0, (size_t)bins * bins * sizeof(float), ctx->stream));
  if (n == 0) return GC_OK;
  GC_REQUIRE(ctx, pa && pb && m, "gc_project_ngp: NULL particle array");
  unsigned nb = gc_blocks(n, 256);
  if (nb > gc_sms() * 16u) nb = gc_sms() * 16u;
  gc_launch(ctx, GK_PROJECT, k_project_ngp, dim3(nb), dim3(256), 0, pa, pb, m, (long long)n, (float)lo_a, (float)lo_b,
            (float)binw_a, (float)binw_b, bins, img);
  GC_LAUNCH_CHECK(ctx, "project");
  return GC_OK;
}

// ------------------------------------------------------------------------------
// self-test of the bounded mbarrier wait (the wait of the TMA particle pass and
// of the tensor-core kernels): one thread arms an mbarrier for one arrival and,
// unless `arrive` is set, nobody arrives; the wait must give up after `budget`
// SM clocks and raise GC_FLAG_TIMEOUT instead of spinning on.
// ------------------------------------------------------------------------------
__global__ void k_selftest_wait(unsigned *__restrict__ status, long long budget, int arrive) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  umma::mbar_init(&bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (arrive) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&bar)) : "memory");
  if (!umma::mbar_wait(&bar, 0u, budget)) atomicOr(status, GC_FLAG_TIMEOUT);
}

extern "C" int gc_selftest_wait_timeout(void *stream, uint32_t *status, int64_t budget_cycles, int arrive) {
  if (!status || budget_cycles < 1 || budget_cycles > GT_BUDGET) {
    gc_set_error(nullptr, "gc_selftest_wait_timeout: status required, budget in [1, %lld] clocks",
                 (long long)GT_BUDGET);
    return GC_ERR_ARG;
  }
  k_selftest_wait<<<1, 32, 0, (cudaStream_t)stream>>>((unsigned *)status, (long long)budget_cycles, arrive ? 1 : 0);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    gc_set_error(nullptr, "gc_selftest_wait_timeout: launch failed: %s", cudaGetErrorString(e));
    return GC_ERR_CUDA;
  }
  return GC_OK;
}
