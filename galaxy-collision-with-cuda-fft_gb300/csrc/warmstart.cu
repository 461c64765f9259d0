// Learned warm start: BF16 3-D convolutions on the fifth-generation tensor cores.
//
// This file holds the tensor-core kernels of the warm-start network (implicit-GEMM
// convolution forward / data-gradient / weight-gradient) and a single-tile GEMM
// used to check the shared-memory descriptor conventions on the device.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "umma.cuh"

// Clock budget of every mbarrier wait (about one second at 2 GHz).
#define WS_WAIT_BUDGET 2000000000LL
// Warps whose lane 0 issues tensor-core MMAs (each commits once per phase).
#define WS_ISSUERS 4
// Layers of the network.
#define WS_NL 11

// ------------------------------------------------------------------------------
// single-tile GEMM check: D (128 x N, f32) = A (128 x K) * B (N x K)^T
// ------------------------------------------------------------------------------
// A and B arrive row-major (bf16 bits) and are staged into shared memory in the
// no-swizzle canonical layout of the requested major-ness:
//   K-major,  R rows: byte(r,k) = (k/8)*R*16 + (r/8)*128 + (r%8)*16 + (k%8)*2
//   MN-major, R rows: byte(r,k) = (r/8)*(K/8)*128 + (k/8)*128 + (k%8)*16 + (r%8)*2
// `swap` exchanges the two byte offsets in the descriptor of MN-major operands.
__device__ __forceinline__ uint32_t st_offset(int r, int k, int R, int K, int mn) {
  return mn ? (uint32_t)((r >> 3) * (K >> 3) * 128 + (k >> 3) * 128 + (k & 7) * 16 + (r & 7) * 2)
            : (uint32_t)((k >> 3) * R * 16 + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

__global__ void __launch_bounds__(128) k_umma_selftest(const uint16_t *__restrict__ A, const uint16_t *__restrict__ B,
                                                       float *__restrict__ D, int N, int K, int a_mn, int b_mn,
                                                       int swap, unsigned *__restrict__ status) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t *sA = sm;
  uint8_t *sB = sm + 128 * K * 2;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sB + 256 * K * 2);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 128 * K; i += 128)
    *reinterpret_cast<uint16_t *>(sA + st_offset(i / K, i % K, 128, K, a_mn)) = A[i];
  for (int i = tid; i < N * K; i += 128)
    *reinterpret_cast<uint16_t *>(sB + st_offset(i / K, i % K, N, K, b_mn)) = B[i];
  if (warp == 0) {
    umma::tmem_alloc(tslot, 256);
    umma::tmem_relinquish();
  }
  if (tid == 0) {
    umma::mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::fence_async_smem();
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tslot;
  if (tid == 0) {
    const uint32_t a_lbo = a_mn ? 128u : 128u * 16u, a_sbo = a_mn ? (uint32_t)(K / 8) * 128u : 128u;
    const uint32_t b_lbo = b_mn ? 128u : (uint32_t)N * 16u, b_sbo = b_mn ? (uint32_t)(K / 8) * 128u : 128u;
    const uint32_t idesc = umma::idesc_bf16(128, N, a_mn, b_mn);
    for (int ks = 0; ks < K / 16; ++ks) {
      const uint32_t aoff = 2u * ks * a_lbo, boff = 2u * ks * b_lbo;  // two core matrices along K
      const uint64_t ad = (a_mn && swap) ? umma::sdesc(umma::smem_u32(sA) + aoff, a_sbo, a_lbo)
                                         : umma::sdesc(umma::smem_u32(sA) + aoff, a_lbo, a_sbo);
      const uint64_t bd = (b_mn && swap) ? umma::sdesc(umma::smem_u32(sB) + boff, b_sbo, b_lbo)
                                         : umma::sdesc(umma::smem_u32(sB) + boff, b_lbo, b_sbo);
      umma::mma_bf16(tmem, ad, bd, idesc, ks > 0 ? 1u : 0u);
    }
    umma::mma_commit(bar);
  }
  __syncwarp();
  const bool ok = umma::mbar_wait(bar, 0, WS_WAIT_BUDGET);
  if (!ok) {
    if (lane == 0) atomicOr(status, 1u);
    umma::mbar_wait(bar, 0, WS_WAIT_BUDGET);  // give in-flight MMAs a second chance before freeing TMEM
  }
  umma::tc_fence_after();
  if (ok) {
    for (int c = 0; c < N; c += 16) {
      uint32_t r[16];
      umma::tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c, r);
      umma::tmem_wait_ld();
      float *row = D + (size_t)(32 * warp + lane) * N + c;
#pragma unroll
      for (int j = 0; j < 16; ++j) row[j] = __uint_as_float(r[j]);
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

extern "C" int gc_ws_selftest_gemm(const void *A, const void *B, float *D, int N, int K, int a_mn, int b_mn, int swap,
                                   void *stream, unsigned *status) {
  if (!A || !B || !D || !status) return GC_ERR_ARG;
  if (N < 16 || N > 256 || (N % 16) || K < 16 || K > 64 || (K % 16)) return GC_ERR_ARG;
  const size_t smem = (size_t)128 * K * 2 + (size_t)256 * K * 2 + 64;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaFuncSetAttribute(k_umma_selftest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return GC_ERR_CUDA;
  k_umma_selftest<<<1, 128, smem, st>>>((const uint16_t *)A, (const uint16_t *)B, D, N, K, a_mn, b_mn, swap, status);
  return cudaGetLastError() == cudaSuccess ? GC_OK : GC_ERR_CUDA;
}

// ------------------------------------------------------------------------------
// activations and weights
// ------------------------------------------------------------------------------
// An activation with C channels on an R^3 grid is stored channel-chunk planar:
// chunk c (channels 8c..8c+7) is an R^3 array of 16-byte rows, one row per voxel
// (x fastest), i.e. element (ch, voxel) at ((ch/8)*R^3 + voxel)*8 + ch%8.
// Convolution weights (3x3x3, tap t = (dz+1)*9 + (dy+1)*3 + (dx+1)) for the
// forward pass are [27][Cin/8][Cout] 16-byte rows of 8 input channels.

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t bf_pack(float a, float b) {
  // round to nearest even, NaN kept quiet
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&p);
}
__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8]) {
  f[0] = bf_lo(v.x); f[1] = bf_hi(v.x); f[2] = bf_lo(v.y); f[3] = bf_hi(v.y);
  f[4] = bf_lo(v.z); f[5] = bf_hi(v.z); f[6] = bf_lo(v.w); f[7] = bf_hi(v.w);
}
template <int O, int N>
__device__ __forceinline__ uint4 pack8(const float (&f)[N]) {
  return make_uint4(bf_pack(f[O], f[O + 1]), bf_pack(f[O + 2], f[O + 3]), bf_pack(f[O + 4], f[O + 5]),
                    bf_pack(f[O + 6], f[O + 7]));
}

// ------------------------------------------------------------------------------
// convolution as implicit GEMM: out[v][co] = sum_t sum_ci in[v + off_t][ci] W[t][co][ci]
// ------------------------------------------------------------------------------
// A CTA owns BZ planes x BY lines x R voxels of the output. Its input tile with a
// one-voxel halo, (BZ+2) x (BY+2) x (R+2) voxels, is staged channel-chunk planar
// in shared memory: row L (padded linear voxel index) of chunk kc at byte
// (kc*V + L)*16. That is the K-major no-swizzle operand layout with 8-row groups
// 128 bytes apart, so the A operand of tap t for the 128 output rows starting
// at padded index s is simply the descriptor at row s + off_t: no im2col copy.
// Output rows are the padded linear range [L0, L1] cut into 128-row M tiles;
// rows that fall on halo voxels are computed and discarded. Accumulators live
// in Tensor Memory (M tile mt in columns mt*Cn ..). Weights stream through a
// two-slot ring of tap groups; completion of the MMAs is tracked by
// tcgen05.commit on one mbarrier per slot.
struct ConvFwd {
  CUtensorMap map;     // input: 8-channel rows of x, y, z, chunk; box one tile
  int use_map;         // the tile's lines fit a box (R <= 126)
  const uint4 *in;
  const uint4 *w;
  const float *bias;   // [Cout] or null
  const uint4 *skip;   // Cout channels or null: added before the activation
  const uint4 *mask;   // Cout channels or null: result zeroed where mask <= 0
  uint4 *out;          // Cout channels or null
  float *out_f32;      // channel 0 as f32 [R^3] or null
  unsigned *status;
  int R, Cin, Cout, BZ, BY;
  int Cn;              // output channels of a CTA (blockIdx.y is the slice)
  int relu;
  int tpg;             // taps per weight group
  int n_mt;
  uint32_t tmem_cols;
};

__host__ __device__ inline void conv_geom(int R, int BZ, int BY, int &W2, int &P, int &V, int &L0, int &L1) {
  W2 = R + 2;
  P = (BY + 2) * W2;
  V = (BZ + 2) * P;
  L0 = P + W2 + 1;
  L1 = V - 1 - L0;
}

__device__ __forceinline__ int tap_offset(int t, int P, int W2) {
  return (t / 9 - 1) * P + ((t / 3) % 3 - 1) * W2 + (t % 3 - 1);
}

// Copy the weights of tap group g (taps g*tpg .. min(27, (g+1)*tpg)), output channels
// c0 .. c0 + Cn, to dst.
__device__ __forceinline__ void load_taps(const uint4 *__restrict__ w, int g, int tpg, int kci, int Cout, int Cn, int c0,
                                          uint8_t *dst, int tid, int nthreads) {
  const int t0 = g * tpg, t1 = min(27, t0 + tpg);
  const uint4 *src = w + (size_t)t0 * kci * Cout + c0;
  uint4 *d = reinterpret_cast<uint4 *>(dst);
  const int n16 = (t1 - t0) * kci * Cn, sh = 31 - __clz(Cn);  // Cn is a power of two
  for (int i = tid; i < n16; i += nthreads)
    umma::cp_async16(d + i, src + (size_t)(i >> sh) * Cout + (i & (Cn - 1)), true);
}

// Mask rows (16 channels from c) of one voxel, read ahead of the accumulators.
template <class A>
__device__ __forceinline__ void conv_mask16(const A &a, int c, size_t vox, size_t R3, uint4 (&m)[2]) {
  if (a.mask) {
    m[0] = __ldg(a.mask + (size_t)(c >> 3) * R3 + vox);
    m[1] = __ldg(a.mask + (size_t)((c >> 3) + 1) * R3 + vox);
  }
}

// Bias, skip, activation, mask and stores of 16 channels (c ..) of one voxel; the bias
// is in shared memory (zeros where there is none).
template <class A>
__device__ __forceinline__ void conv_store16(const A &a, const uint32_t (&r)[16], const float *bias, const uint4 (&m)[2],
                                             int c, size_t vox, size_t R3) {
  float v[16];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 b4 = *reinterpret_cast<const float4 *>(bias + c + 4 * q);
    v[4 * q] = __uint_as_float(r[4 * q]) + b4.x;
    v[4 * q + 1] = __uint_as_float(r[4 * q + 1]) + b4.y;
    v[4 * q + 2] = __uint_as_float(r[4 * q + 2]) + b4.z;
    v[4 * q + 3] = __uint_as_float(r[4 * q + 3]) + b4.w;
  }
  if (a.skip) {
    float s0[8], s1[8];
    unpack8(__ldg(a.skip + (size_t)(c >> 3) * R3 + vox), s0);
    unpack8(__ldg(a.skip + (size_t)((c >> 3) + 1) * R3 + vox), s1);
#pragma unroll
    for (int j = 0; j < 8; ++j) { v[j] += s0[j]; v[8 + j] += s1[j]; }
  }
  if (a.relu) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.0f);
  }
  if (a.mask) {
    float m0[8], m1[8];
    unpack8(m[0], m0);
    unpack8(m[1], m1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = m0[j] > 0.0f ? v[j] : 0.0f;
      v[8 + j] = m1[j] > 0.0f ? v[8 + j] : 0.0f;
    }
  }
  if (a.out) {
    a.out[(size_t)(c >> 3) * R3 + vox] = pack8<0>(v);
    a.out[(size_t)((c >> 3) + 1) * R3 + vox] = pack8<8>(v);
  }
  if (a.out_f32 && c == 0) a.out_f32[vox] = v[0];
}

__global__ void __launch_bounds__(256) k_conv_fwd(const __grid_constant__ ConvFwd a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int R = a.R;
  int W2, P, V, L0, L1;
  conv_geom(R, a.BZ, a.BY, W2, P, V, L0, L1);
  const int kci = a.Cin >> 3;
  const size_t R3 = (size_t)R * R * R;
  const int nby = R / a.BY;
  const int z0 = (blockIdx.x / nby) * a.BZ, y0 = (blockIdx.x % nby) * a.BY;
  const uint32_t tile_bytes = (uint32_t)(kci * V + 128) * 16u;
  const int Cn = a.Cn, c0 = blockIdx.y * Cn;
  const uint32_t tap_bytes = (uint32_t)a.Cin * Cn * 2u;
  const uint32_t slot_bytes = (uint32_t)a.tpg * tap_bytes;
  uint8_t *tile = sm;
  uint8_t *ring = sm + ((tile_bytes + 1023u) & ~1023u);
  uint64_t *bars = reinterpret_cast<uint64_t *>(ring + 2u * slot_bytes);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + 3);
  float *bias = reinterpret_cast<float *>(bars + 8);
  const int ngroups = (27 + a.tpg - 1) / a.tpg;

  if (warp == 0) {
    umma::tmem_alloc(tslot, a.tmem_cols);
    umma::tmem_relinquish();
  }
  if (tid == 0) {  // one arrival per issuing warp (WS_ISSUERS commits per phase)
    umma::mbar_init(&bars[0], WS_ISSUERS);
    umma::mbar_init(&bars[1], WS_ISSUERS);
    umma::mbar_init(&bars[2], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  gc_after();  // (behind the allocation: a grid behind this one must not get Tensor Memory first)
  if (tid == 0 && a.use_map) {
    umma::fence_async_smem();
    umma::mbar_arrive_expect_tx(&bars[2], (uint32_t)(kci * V) * 16u);
    umma::tma_load_4d(sm, &a.map, -2, y0 - 1, z0 - 1, 0, &bars[2]);
  }
  if (tid < Cn) bias[tid] = a.bias ? a.bias[c0 + tid] : 0.0f;
  // input tile, zero outside the grid, plus a zero margin read by the last M tile: one
  // box of the tensor map (1.2k clk for 23 KB), or one warp per padded line with lanes
  // along x (10k clk) where a line is longer than a box may be
  uint4 *trow = reinterpret_cast<uint4 *>(tile);
  if (!a.use_map) {
    const int nzy = (a.BZ + 2) * (a.BY + 2), nrows = kci * nzy, nwarps = blockDim.x >> 5;
    for (int row = warp; row < nrows; row += nwarps) {
      const int kc = row / nzy, rr = row - kc * nzy;
      const int tz = rr / (a.BY + 2), ty = rr - tz * (a.BY + 2);
      const int gz = z0 - 1 + tz, gy = y0 - 1 + ty;
      const bool rowin = (unsigned)gz < (unsigned)R && (unsigned)gy < (unsigned)R;
      const uint4 *src = a.in + (size_t)kc * R3 + ((size_t)(rowin ? gz : 0) * R + (rowin ? gy : 0)) * R;
      uint4 *dst = trow + (size_t)kc * V + (size_t)rr * W2;
      for (int tx = lane; tx < W2; tx += 32) {
        const int gx = tx - 1;
        const bool in = rowin && (unsigned)gx < (unsigned)R;
        umma::cp_async16(dst + tx, in ? (const void *)(src + gx) : (const void *)a.in, in);
      }
    }
  }
  for (int i = tid; i < 128; i += blockDim.x) trow[kci * V + i] = make_uint4(0u, 0u, 0u, 0u);
  load_taps(a.w, 0, a.tpg, kci, a.Cout, Cn, c0, ring, tid, blockDim.x);
  umma::cp_async_wait_all();
  umma::fence_async_smem();
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma::idesc_bf16(128, Cn, 0, 0);
  const uint32_t a_lbo = (uint32_t)V * 16u, b_lbo = (uint32_t)Cn * 16u;
  const uint32_t tile_u32 = umma::smem_u32(tile), ring_u32 = umma::smem_u32(ring);
  uint32_t ph0 = 0u, ph1 = 0u;  // next completion parity of each slot's barrier
  int last = 0;                  // slot of the last commit
  bool fail = a.use_map && !umma::mbar_wait(&bars[2], 0, WS_WAIT_BUDGET);  // (then nothing is stored)
  for (int g = 0; g < ngroups; ++g) {
    const int s = g & 1;
    if (warp < WS_ISSUERS) {  // issuer w owns the M tiles mt = w (mod WS_ISSUERS)
      umma::tc_fence_after();
      const uint32_t lead = umma::elect_one();
      const int t0 = g * a.tpg, t1 = min(27, t0 + a.tpg);
      // descriptors differ only in the start address (bits 0..13, address / 16)
      const uint64_t ad0 = umma::sdesc(tile_u32, a_lbo, 128u), bd0 = umma::sdesc(ring_u32, b_lbo, 128u);
      // A warp feeds the tensor core an instruction every few tens of clocks: the whole
      // warp runs the loop on uniform values, the descriptors carried by additions only,
      // and one elected lane issues. With the address arithmetic in the inner loop of one
      // thread, the four issuers together took 59 clk an instruction at 128 x 16 x 16
      // (16 -> 16 channels, R = 128), so 40: the operand rows are 32 clk to read.
      const uint32_t kstep_a = (2u * a_lbo) >> 4, kstep_b = (2u * b_lbo) >> 4;
      const int nks = kci / 2;
      for (int t = t0; t < t1; ++t) {
        const uint64_t bd = bd0 + (((uint32_t)s * slot_bytes + (uint32_t)(t - t0) * tap_bytes) >> 4);
        uint64_t ad = ad0 + (uint32_t)(L0 + 128 * warp + tap_offset(t, P, W2));
        uint32_t td = tmem + (uint32_t)(warp * Cn);
#pragma unroll 4
        for (int mt = warp; mt < a.n_mt; mt += WS_ISSUERS, ad += 128u * WS_ISSUERS, td += (uint32_t)(WS_ISSUERS * Cn)) {
          umma::mma_bf16_if(lead, td, ad, bd, idesc, t > 0 ? 1u : 0u);
          for (int ks = 1; ks < nks; ++ks) umma::mma_bf16_if(lead, td, ad + ks * kstep_a, bd + ks * kstep_b, idesc, 1u);
        }
      }
      if (lead) umma::mma_commit(&bars[s]);
      __syncwarp();
    }
    last = s;
    if (g + 1 < ngroups) {
      const int s1 = (g + 1) & 1;
      if (g >= 1) {
        fail = !umma::mbar_wait(&bars[s1], s1 ? ph1 : ph0, WS_WAIT_BUDGET);
        if (s1) ph1 ^= 1u; else ph0 ^= 1u;
      }
      if (__syncthreads_or(fail)) { fail = true; break; }
      load_taps(a.w, g + 1, a.tpg, kci, a.Cout, Cn, c0, ring + (uint32_t)s1 * slot_bytes, tid, blockDim.x);
      umma::cp_async_wait_all();
      umma::fence_async_smem();
      __syncthreads();
    }
  }
  // completion of every MMA: the last commit (MMAs of one thread complete in order)
  if (!umma::mbar_wait(&bars[last], last ? ph1 : ph0, WS_WAIT_BUDGET)) fail = true;
  fail = __syncthreads_or(fail);
  umma::tc_fence_after();
  if (fail) {
    if (tid == 0) {
      atomicOr(a.status, 1u);
      // the box may still be on its way: it lands before the CTA leaves its shared memory
      if (a.use_map) umma::mbar_wait(&bars[2], 0, WS_WAIT_BUDGET);
    }
  } else {
    const int quad = warp & 3;
    for (int mt = warp >> 2; mt < a.n_mt; mt += (blockDim.x >> 7)) {
      const int L = L0 + 128 * mt + 32 * quad + lane;
      const int tz = L / P, rem = L - tz * P, ty = rem / W2, tx = rem - ty * W2;
      const bool valid = L <= L1 && tz >= 1 && tz <= a.BZ && ty >= 1 && ty <= a.BY && tx >= 1 && tx <= R;
      const size_t vox = ((size_t)(z0 + tz - 1) * R + (y0 + ty - 1)) * R + (tx - 1);
      for (int c = 0; c < Cn; c += 16) {
        uint32_t r[16];
        uint4 m[2] = {};
        umma::tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(mt * Cn + c), r);
        if (valid) conv_mask16(a, c0 + c, vox, R3, m);
        umma::tmem_wait_ld();
        if (!valid) continue;
        conv_store16(a, r, bias - c0, m, c0 + c, vox, R3);
      }
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, a.tmem_cols);
}

// ------------------------------------------------------------------------------
// the same convolution marching along z
// ------------------------------------------------------------------------------
// A CTA walks the planes of a strip of MA_LINES lines x BX voxels: a ring of input
// planes (with their one-voxel halo) is filled ahead by the TMA engine, the MMAs of a
// plane go to one half of Tensor Memory while the other half is read out, and all 27
// taps of the weights stay in shared memory. Loads, MMAs and epilogue therefore run
// beside each other; in k_conv_fwd they follow one another within a CTA, and its large
// input tile leaves room for one CTA on an SM (16 -> 16 channels, R = 128: 9.0k clk of
// loads, 20.6k of MMAs, 12.0k of epilogue for 2048 voxels). An M tile is 8 voxels of
// each of 16 lines: the 8-row groups of the operand lie one line apart (row order
// [line][chunk][x]), so every row is an output voxel and no halo row is computed
// (19 x 128 rows for 2048 voxels there). The accumulation order of an output is that
// of k_conv_fwd, taps outermost: results are the same bits.
// Measured (16 -> 16 channels): R = 128 155 -> 70 us, R = 64 18.5 -> 13.9. What is left
// is the MMAs: 9.1k clk a unit of 16 x 64 voxels against 216 x 40; each reads its 128
// operand rows from shared memory again (32 clk), and taps cannot share a read without
// another order of accumulation. A plane is one box of a tensor map: 0.8k clk for 36 KB
// with several in flight, where one bulk copy per line and chunk took 70 clk a copy
// (3.3k) and 16-byte asynchronous copies by a warp 13k.
// The units of work, (strip, plane) with the plane fastest, are dealt to the CTAs in
// equal contiguous runs; a run that enters a new strip reloads its first two planes.
struct ConvMarch {
  CUtensorMap map;  // input: 8-channel rows of x, chunk, y, z; box one slot
  const uint4 *w;
  const float *bias;  // as in ConvFwd, down to out_f32
  const uint4 *skip;
  const uint4 *mask;
  uint4 *out;
  float *out_f32;
  unsigned *status;
  int R, Cin, Cout, BX;
  int Cn;     // output channels of a CTA (blockIdx.y is the slice)
  int relu;
  int ns;     // ring slots (planes)
  int units;  // (R / BX) * (R / MA_LINES) * R
  uint32_t tmem_cols;
};

#define MA_LINES 16
#define MA_EPI 8  // epilogue warps, then WS_ISSUERS issuing warps, then one loading warp
#define MA_THREADS (32 * (MA_EPI + WS_ISSUERS + 1))
#define MA_MAX_SLOTS 6

static __host__ __device__ inline uint32_t march_slot_bytes(int Cin, int BX) {
  return ((uint32_t)((MA_LINES + 2) * (Cin >> 3) * (BX + 2)) * 16u + 127u) & ~127u;
}

__global__ void __launch_bounds__(MA_THREADS) k_conv_march(const __grid_constant__ ConvMarch a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int R = a.R, kci = a.Cin >> 3, W2 = a.BX + 2, ns = a.ns, n_mt = a.BX >> 3;
  const uint32_t slot_bytes = march_slot_bytes(a.Cin, a.BX);
  const int Cn = a.Cn, c0 = blockIdx.y * Cn;
  const uint32_t tap_bytes = (uint32_t)a.Cin * Cn * 2u, w_bytes = 27u * tap_bytes;
  uint8_t *wsm = sm + (uint32_t)ns * slot_bytes;
  uint64_t *full = reinterpret_cast<uint64_t *>(wsm + w_bytes);  // [ns] a plane has arrived
  uint64_t *empty = full + MA_MAX_SLOTS;                         // [ns] its last reader is done
  uint64_t *tfull = empty + MA_MAX_SLOTS;                        // [2] accumulators complete
  uint64_t *tempty = tfull + 2;                                  // [2] accumulators read out
  uint64_t *wbar = tempty + 2;                                   // weights have arrived
  uint64_t *done = wbar + 1;                                     // every MMA of the CTA is complete
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  float *bias = reinterpret_cast<float *>(full + 2 * MA_MAX_SLOTS + 8);
  if (warp == 0) {
    umma::tmem_alloc(tslot, a.tmem_cols);
    umma::tmem_relinquish();
  }
  if (tid == 32) {
    for (int s = 0; s < ns; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], WS_ISSUERS);
    }
    for (int b = 0; b < 2; ++b) {
      umma::mbar_init(&tfull[b], WS_ISSUERS);
      umma::mbar_init(&tempty[b], MA_EPI);
    }
    umma::mbar_init(wbar, 32 * MA_EPI);
    umma::mbar_init(done, WS_ISSUERS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tslot;
  gc_after();  // (behind the allocation: a grid behind this one must not get Tensor Memory first)
  // read after the weights have arrived, which these threads announce
  if (tid < Cn) bias[tid] = a.bias ? a.bias[c0 + tid] : 0.0f;
  const int nbx = R / a.BX;
  const int u0 = (int)((long long)a.units * blockIdx.x / gridDim.x);
  const int u1 = (int)((long long)a.units * (blockIdx.x + 1) / gridDim.x);
  bool ok = true;

  if (warp < MA_EPI) {
    // ---- epilogue: warp w reads lane quarter w % 4 of the M tiles w / 4, w / 4 + 2, ..
    const int quad = warp & 3, line = 4 * quad + (lane >> 3);
    const size_t R3 = (size_t)R * R * R;
    const int nc = Cn >> 4, nit = ((n_mt - (warp >> 2) + 1) >> 1) * nc;  // 16-channel pieces of this warp
    load_taps(a.w, 0, 27, kci, a.Cout, Cn, c0, wsm, tid, 32 * MA_EPI);
    umma::cp_async_wait_all();
    umma::fence_async_smem();
    umma::mbar_arrive(wbar);
    int n = 0;
    uint4 m[2] = {};  // mask rows of the next piece
    for (int u = u0; u < u1; ++u, ++n) {
      const int strip = u / R, z = u - strip * R, sy = strip / nbx;
      const int b = n & 1;
      const size_t vox0 = ((size_t)z * R + (MA_LINES * sy + line)) * R + (strip - sy * nbx) * a.BX + (lane & 7);
      int mt = warp >> 2, c = 0;
      if (nit) conv_mask16(a, c0, vox0 + 8 * mt, R3, m);
      ok = __all_sync(0xffffffffu, umma::mbar_wait(&tfull[b], (n >> 1) & 1, WS_WAIT_BUDGET));
      if (!ok) break;
      umma::tc_fence_after();
      for (int it = 0; it < nit; ++it) {
        uint32_t r[16];
        umma::tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)((b * n_mt + mt) * Cn + c), r);
        const int mt0 = mt, cc = c;
        const uint4 mc[2] = {m[0], m[1]};
        c += 16;
        if (c == Cn) { c = 0; mt += MA_EPI / 4; }
        if (it + 1 < nit) conv_mask16(a, c0 + c, vox0 + 8 * mt, R3, m);
        umma::tmem_wait_ld();
        conv_store16(a, r, bias - c0, mc, c0 + cc, vox0 + 8 * mt0, R3);
      }
      umma::tc_fence_before();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(&tempty[b]);
    }
  } else if (warp < MA_EPI + WS_ISSUERS) {
    // ---- issue: warp w owns the M tiles w, w + WS_ISSUERS, ..; its whole warp runs the
    // loop on uniform values and one elected lane issues
    const int w = warp - MA_EPI;
    const uint32_t lead = umma::elect_one();
    const uint32_t idesc = umma::idesc_bf16(128, Cn, 0, 0);
    const uint64_t ad0 = umma::sdesc(umma::smem_u32(sm), (uint32_t)W2 * 16u, (uint32_t)(kci * W2) * 16u);
    const uint64_t bd0 = umma::sdesc(umma::smem_u32(wsm), (uint32_t)Cn * 16u, 128u);
    const uint32_t kstep_a = 2u * (uint32_t)W2, kstep_b = 2u * (uint32_t)Cn;
    const int nks = kci / 2;
    ok = __all_sync(0xffffffffu, umma::mbar_wait(wbar, 0, WS_WAIT_BUDGET));
    int n = 0;
    int fs = 0;           // slot and phase of the first plane that the next unit reads
    uint32_t fph = 0u;
    for (int u = u0; u < u1 && ok;) {
      const int len = min(R - u % R, u1 - u);
      for (int i = 0; i < len && ok; ++i, ++n) {
        int sl[3];
        sl[0] = fs;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (d) sl[d] = sl[d - 1] + 1 < ns ? sl[d - 1] + 1 : 0;
        }
        const int b = n & 1;
        if (n >= 2) ok = ok && umma::mbar_wait(&tempty[b], ((n >> 1) - 1) & 1, WS_WAIT_BUDGET);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        umma::tc_fence_after();
        uint64_t bd = bd0;
        const uint32_t td0 = tmem + (uint32_t)((b * n_mt + w) * Cn);
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
          if (dz == 2 || i == 0) {  // the planes of a strip are waited for one by one
            ok = __all_sync(0xffffffffu, ok && umma::mbar_wait(&full[sl[dz]], fph ^ (sl[dz] < fs ? 1u : 0u), WS_WAIT_BUDGET));
            if (!ok) break;
          }
          for (int dy = 0; dy < 3; ++dy) {
            uint64_t al = ad0 + (uint32_t)(((uint32_t)sl[dz] * slot_bytes) >> 4) + (uint32_t)(dy * kci * W2 + 8 * w);
            for (int dx = 0; dx < 3; ++dx, ++al, bd += tap_bytes >> 4) {
              uint64_t ad = al;
              uint32_t td = td0;
              const uint32_t acc = (dz | dy | dx) ? 1u : 0u;
              for (int mt = w; mt < n_mt; mt += WS_ISSUERS, ad += 8u * WS_ISSUERS, td += (uint32_t)(WS_ISSUERS * Cn)) {
                umma::mma_bf16_if(lead, td, ad, bd, idesc, acc);
                for (int ks = 1; ks < nks; ++ks)
                  umma::mma_bf16_if(lead, td, ad + ks * kstep_a, bd + ks * kstep_b, idesc, 1u);
              }
            }
          }
        }
        if (lead) {
          umma::mma_commit(&tfull[b]);
          umma::mma_commit(&empty[sl[0]]);
          if (i == len - 1) {
            umma::mma_commit(&empty[sl[1]]);
            umma::mma_commit(&empty[sl[2]]);
          }
        }
        __syncwarp();
        const int adv = i == len - 1 ? 3 : 1;
        fs += adv;
        if (fs >= ns) { fs -= ns; fph ^= 1u; }
      }
      u += len;
    }
    if (lead) umma::mma_commit(done);
  } else {
    // ---- load: one box per plane
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)((MA_LINES + 2) * kci * W2) * 16u;
      int s = 0;
      uint32_t ph = 1u;  // the first round finds the slots empty
      for (int u = u0; u < u1 && ok;) {
        const int strip = u / R, z = u - strip * R, len = min(R - z, u1 - u), sy = strip / nbx;
        for (int p = z - 1; p <= z + len; ++p) {
          ok = umma::mbar_wait(&empty[s], ph, WS_WAIT_BUDGET);
          if (!ok) break;
          umma::mbar_arrive_expect_tx(&full[s], bytes);
          umma::tma_load_4d(sm + (uint32_t)s * slot_bytes, &a.map, 2 * ((strip - sy * nbx) * a.BX - 1), 0,
                            MA_LINES * sy - 1, p, &full[s]);
          if (++s == ns) { s = 0; ph ^= 1u; }
        }
        u += len;
      }
      if (!ok) {  // after a timeout: let the copies in flight land before the CTA ends
        for (int i = 0; i < ns; ++i) umma::mbar_wait(&full[i], i < s ? ph ^ 1u : ph, WS_WAIT_BUDGET);
      }
    }
  }
  if (!ok && lane == 0) atomicOr(a.status, 1u);
  if (warp == 0 && !umma::mbar_wait(done, 0, WS_WAIT_BUDGET) && lane == 0) atomicOr(a.status, 1u);
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, a.tmem_cols);
}

// ------------------------------------------------------------------------------
// weight gradient: dW[t][co][ci] = sum_v gy[v][co] x[v + off_t][ci]
// ------------------------------------------------------------------------------
// GEMM with M = co (64 or 128 rows), N = ci, K = voxels. The voxels are divided into
// blocks of BZ planes x BY lines x R, and the blocks over `nparts` partial sums (block b
// to partial b mod nparts), which are added in their order afterwards. Within a partial
// an accumulator takes its blocks one after another, 16 rows of the padded linear range
// [L0, L1] at a time: that order is part of the result's bits and is kept whatever runs
// beside what.
// A CTA takes the taps of one dz (blockIdx.x = dz and a share of its nine taps; the
// groups of a partial next to each other, so that the partials with a block more, which
// come first, start first), so its x tile is the block's BZ planes moved by dz, with the
// halo in y and x, staged as in the forward pass and as one box; read MN-major
// (8 channels of one voxel per 16-byte row), the B operand of a tap is again the tile
// shifted by some rows. gy arrives in stages of 128 rows, each row's 16-byte pieces
// (8 output channels) placed in groups of 8 rows so that every one of the M rows
// addresses shared memory of the stage (rows >= Cout are never read back). Rows outside
// the CTA's block are zero in gy. A CTA (partial, tap group) has warps that fill the
// ring of stages and at the end read the accumulators out, and warps that issue.
// With one loop that loaded a stage, synchronised and issued from four threads, M always
// 128, and the tap groups one after another, 16 -> 16 channels at R = 64 took 103 us and
// 128 -> 64 at R = 8 145 us; so they take 44 and 7.7.
struct ConvW {
  CUtensorMap map;  // x: 8-channel rows of x, y, z, chunk; box one tile
  int use_map;      // the tile's lines fit a box (R <= 126)
  int sub;          // groups of a dz
  const uint4 *x;   // layer input, Cin channels
  const uint4 *gy;  // gradient of the pre-activation output, Cout channels
  float *part;      // [nparts][27][Cout][Cin]
  unsigned *status;
  int R, Cin, Cout, BZ, BY;
  int nblocks;
  int tpg;   // taps of a group (dy3 = 0), or dx (dy3 = 1)
  int dy3;   // N = the three dy taps of one channel chunk (24 columns) instead of Cin
  int ns;    // stages
  uint32_t tmem_cols;
};

#define WG_ROWS 128  // rows of a stage
#define WG_LOAD 8    // warps that load (and read out), then WS_ISSUERS that issue
#define WG_THREADS (32 * (WG_LOAD + WS_ISSUERS))
#define WG_MAX_STAGES 8

__global__ void __launch_bounds__(WG_THREADS) k_conv_wgrad(const __grid_constant__ ConvW a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int R = a.R, ns = a.ns;
  int W2, P, V, L0, L1;
  conv_geom(R, a.BZ, a.BY, W2, P, V, L0, L1);
  const int kci = a.Cin >> 3, kco = a.Cout >> 3;
  const size_t R3 = (size_t)R * R * R;
  const int nby = R / a.BY;
  const int nst = (L1 - L0 + WG_ROWS) / WG_ROWS;
  const int M = a.Cout <= 64 ? 64 : 128;
  const uint32_t group_bytes = (uint32_t)M * 16u, stage_bytes = (WG_ROWS / 8) * group_bytes;
  const int Vt = a.BZ * P;  // rows of a chunk of the tile: planes 1 + dz .. BZ + dz of the padded block
  const uint32_t tile_bytes = ((uint32_t)(kci * Vt + 128) * 16u + 1023u) & ~1023u;
  uint8_t *tile = sm, *stg = sm + tile_bytes;
  uint64_t *full = reinterpret_cast<uint64_t *>(stg + (uint32_t)ns * stage_bytes);  // [ns] a stage is there
  uint64_t *empty = full + WG_MAX_STAGES;                                           // [ns] its MMAs are done
  uint64_t *tfull = empty + WG_MAX_STAGES;                                          // the x tile is there
  uint64_t *tempty = tfull + 1;                                                     // its MMAs are done
  uint64_t *done = tempty + 1;                                                      // every MMA is
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  // accumulators of this group: taps of a dz, or its dx of each chunk
  const int all = a.dy3 ? 3 : 9, dzi = blockIdx.x / a.sub;
  const int g0 = (blockIdx.x - dzi * a.sub) * a.tpg, g1 = min(all, g0 + a.tpg);
  const int N = a.dy3 ? 24 : a.Cin, nacc = (g1 - g0) * (a.dy3 ? kci : 1);
  if (warp == 0) {
    umma::tmem_alloc(tslot, a.tmem_cols);
    umma::tmem_relinquish();
  }
  if (tid == 32) {
    for (int s = 0; s < ns; ++s) {
      umma::mbar_init(&full[s], 32);
      umma::mbar_init(&empty[s], WS_ISSUERS);
    }
    umma::mbar_init(tfull, a.use_map ? 1 : 32 * WG_LOAD);
    umma::mbar_init(tempty, WS_ISSUERS);
    umma::mbar_init(done, WS_ISSUERS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // zero margin behind the tile, read by the last rows' shifts
  uint4 *trow = reinterpret_cast<uint4 *>(tile);
  for (int i = tid; i < 128; i += WG_THREADS) trow[kci * Vt + i] = make_uint4(0u, 0u, 0u, 0u);
  umma::fence_async_smem();
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tslot;
  gc_after();  // (behind the allocation: a grid behind this one must not get Tensor Memory first)
  bool ok = true;
  int nb = 0;  // blocks done: parity of the tile's barriers

  if (warp < WG_LOAD) {
    // ---- load: warp w fills every WG_LOAD-th stage
    int f = 0, s = 0;
    uint32_t ph = 1u;  // the first round finds the stages empty
    // quotients by P and W2 as high products with ceil(2^32 / d), exact for rows and
    // divisors below 2^16 (four divisions a lane, one after another, took 2.8k clk a stage)
    const uint32_t mP = 0xffffffffu / (uint32_t)P + 1u, mW = 0xffffffffu / (uint32_t)W2 + 1u;
    for (int b = blockIdx.y; b < a.nblocks && ok; b += gridDim.y, ++nb) {
      const int z0 = (b / nby) * a.BZ, y0 = (b % nby) * a.BY;
      if (!a.use_map || warp == 0) {  // the tile, when the last block's MMAs are done with it
        if (nb) ok = __all_sync(0xffffffffu, umma::mbar_wait(tempty, (nb - 1) & 1, WS_WAIT_BUDGET));
        if (!ok) break;
      }
      if (a.use_map) {
        if (tid == 0) {
          umma::mbar_arrive_expect_tx(tfull, (uint32_t)(kci * Vt) * 16u);
          umma::tma_load_4d(tile, &a.map, -2, y0 - 1, z0 - 1 + dzi, 0, tfull);
        }
        __syncwarp();
      } else {
        const int nzy = a.BZ * (a.BY + 2), nrows = kci * nzy;
        for (int row = warp; row < nrows; row += WG_LOAD) {
          const int kc = row / nzy, rr = row - kc * nzy;
          const int tz = rr / (a.BY + 2), ty = rr - tz * (a.BY + 2);
          const int gz = z0 - 1 + dzi + tz, gy_ = y0 - 1 + ty;
          const bool rowin = (unsigned)gz < (unsigned)R && (unsigned)gy_ < (unsigned)R;
          const uint4 *src = a.x + (size_t)kc * R3 + ((size_t)(rowin ? gz : 0) * R + (rowin ? gy_ : 0)) * R;
          uint4 *dst = trow + (size_t)kc * Vt + (size_t)rr * W2;
          for (int tx = lane; tx < W2; tx += 32) {
            const int gx = tx - 1;
            const bool in = rowin && (unsigned)gx < (unsigned)R;
            umma::cp_async16(dst + tx, in ? (const void *)(src + gx) : (const void *)a.x, in);
          }
        }
        umma::cp_async_wait_all();
        umma::fence_async_smem();
        umma::mbar_arrive(tfull);
      }
      for (int st = 0; st < nst; ++st, ++f) {
        // every warp waits for every stage in turn (a wait by parity must not fall a phase behind)
        ok = __all_sync(0xffffffffu, umma::mbar_wait(&empty[s], ph, WS_WAIT_BUDGET));
        if (!ok) break;
        if (f % WG_LOAD == warp) {
          uint8_t *sbuf = stg + (uint32_t)s * stage_bytes;
#pragma unroll
          for (int r = lane; r < WG_ROWS; r += 32) {
            const int L = L0 + WG_ROWS * st + r;
            const int tz = (int)__umulhi((uint32_t)L, mP), rem = L - tz * P;
            const int ty = (int)__umulhi((uint32_t)rem, mW), tx = rem - ty * W2;
            const bool valid = L <= L1 && ty >= 1 && ty <= a.BY && tx >= 1 && tx <= R;
            const uint4 *src = valid ? a.gy + ((size_t)(z0 + tz - 1) * R + (y0 + ty - 1)) * R + (tx - 1) : a.gy;
            uint8_t *d = sbuf + (uint32_t)(r >> 3) * group_bytes + (r & 7) * 16;
            for (int c = 0; c < kco; ++c) umma::cp_async16(d + c * 128, valid ? src + (size_t)c * R3 : a.gy, valid);
          }
          umma::cp_async_wait_all();
          umma::fence_async_smem();
          umma::mbar_arrive(&full[s]);
        }
        if (++s == ns) { s = 0; ph ^= 1u; }
      }
    }
    // ---- every MMA complete: accumulators out
    ok = __all_sync(0xffffffffu, ok && umma::mbar_wait(done, 0, WS_WAIT_BUDGET));
    umma::tc_fence_after();
    if (ok) {
      const int quad = warp & 3, co = M == 64 ? 16 * quad + lane : 32 * quad + lane;
      const bool mine = co < a.Cout && (M == 128 || lane < 16);
      const int ncol8 = nacc * (N / 8);  // columns in pieces of 8
      float *base = a.part + (size_t)blockIdx.y * 27 * a.Cout * a.Cin + (size_t)co * a.Cin;
      for (int q = 2 * (warp >> 2); q < ncol8; q += 4) {
        uint32_t r[16];
        umma::tmem_ld16(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(8 * q), r);
        umma::tmem_wait_ld();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c8 = q + h;
          if (!mine || c8 >= ncol8) continue;
          int t, ci;
          if (a.dy3) {
            const int u = c8 / 3, dy = c8 - 3 * u;
            t = 9 * dzi + 3 * dy + g0 + u / kci;
            ci = 8 * (u % kci);
          } else {
            t = 9 * dzi + g0 + c8 / kci;
            ci = 8 * (c8 % kci);
          }
          float4 *dst = reinterpret_cast<float4 *>(base + (size_t)t * a.Cout * a.Cin + ci);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            dst[j] = make_float4(__uint_as_float(r[8 * h + 4 * j]), __uint_as_float(r[8 * h + 4 * j + 1]),
                                 __uint_as_float(r[8 * h + 4 * j + 2]), __uint_as_float(r[8 * h + 4 * j + 3]));
        }
      }
    }
  } else {
    // ---- issue: warp w feeds the accumulators w, w + WS_ISSUERS, ..
    const int w = warp - WG_LOAD;
    const uint32_t lead = umma::elect_one();
    const uint32_t idesc = umma::idesc_bf16(M, N, 1, 1);
    const uint64_t ad0 = umma::sdesc_mn(umma::smem_u32(stg), group_bytes, 128u);
    const uint64_t bd0 = umma::sdesc_mn(umma::smem_u32(tile), 128u, a.dy3 ? (uint32_t)W2 * 16u : (uint32_t)Vt * 16u);
    const uint32_t kstep = (2u * group_bytes) >> 4;
    int s = 0;
    uint32_t ph = 0u, accum = 0u;
    for (int b = blockIdx.y; b < a.nblocks && ok; b += gridDim.y, ++nb) {
      ok = __all_sync(0xffffffffu, umma::mbar_wait(tfull, nb & 1, WS_WAIT_BUDGET));
      for (int st = 0; st < nst && ok; ++st) {
        ok = __all_sync(0xffffffffu, umma::mbar_wait(&full[s], ph, WS_WAIT_BUDGET));
        if (!ok) break;
        umma::tc_fence_after();
        const uint64_t ad = ad0 + (((uint32_t)s * stage_bytes) >> 4);
        const uint64_t bs = bd0 + (uint32_t)(L0 - P + WG_ROWS * st);
        for (int q = w; q < nacc; q += WS_ISSUERS) {
          int off;  // dy W2 + dx; dy = -1 is the first of the three column groups
          if (a.dy3)
            off = (g0 + q / kci - 1) - W2 + (q % kci) * Vt;
          else
            off = ((g0 + q) / 3 - 1) * W2 + (g0 + q) % 3 - 1;
          const uint64_t bd = bs + (uint64_t)(int64_t)off;
          const uint32_t td = tmem + (uint32_t)(q * N);
          umma::mma_bf16_if(lead, td, ad, bd, idesc, accum);
#pragma unroll
          for (int ks = 1; ks < WG_ROWS / 16; ++ks)
            umma::mma_bf16_if(lead, td, ad + ks * kstep, bd + 16u * ks, idesc, 1u);
        }
        accum = 1u;
        if (lead) {
          umma::mma_commit(&empty[s]);
          if (st == nst - 1) umma::mma_commit(tempty);
        }
        __syncwarp();
        if (++s == ns) { s = 0; ph ^= 1u; }
      }
    }
    if (lead) umma::mma_commit(done);
  }
  if (!ok && lane == 0) atomicOr(a.status, 1u);
  if (warp == 0) {  // after a timeout too, MMAs and copies in flight end first
    if (!umma::mbar_wait(done, 0, WS_WAIT_BUDGET) && lane == 0) atomicOr(a.status, 1u);
    if (!ok && a.use_map) umma::mbar_wait(tfull, nb & 1, WS_WAIT_BUDGET);
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, a.tmem_cols);
}

// out[e] = sum over c of part[c*nelem + e] for few elements and many partials:
// one block per element, a fixed strided split and a fixed tree (deterministic).
__device__ __forceinline__ void reduce_col(const float *__restrict__ part, int nparts, int nelem, int e,
                                           float *__restrict__ out) {
  __shared__ float red[256];
  float s = 0.0f;
  for (int c = threadIdx.x; c < nparts; c += 256) s += part[(size_t)c * nelem + e];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[e] = red[0];
}
__global__ void __launch_bounds__(256) k_reduce_cols(const float *__restrict__ part, int nparts, int nelem,
                                                     float *__restrict__ out) {
  gc_after();
  reduce_col(part, nparts, nelem, blockIdx.x, out);
}

// dW[e] = sum over partials in their order, for several layers (blockIdx.y): one chain of
// additions per element, U partials' loads of it in flight. A launch per layer took 4.6
// us each at R = 64, all eleven in one 29.
struct WgReduce {
  struct Layer {
    const float *part;
    float *out;
    int nparts, nelem;
  } l[WS_NL];
};
template <int U>
__device__ __forceinline__ void reduce_run(const float *__restrict__ p, size_t stride, int n, int &c, float &s) {
  for (; c + U <= n; c += U) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = __ldcg(p + (size_t)u * stride);
    p += (size_t)U * stride;
#pragma unroll
    for (int u = 0; u < U; ++u) s += v[u];
  }
}
__global__ void __launch_bounds__(64) k_wgrad_reduce(const __grid_constant__ WgReduce d) {
  gc_after();
  const WgReduce::Layer &L = d.l[blockIdx.y];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < L.nelem; e += gridDim.x * blockDim.x) {
    float s = 0.0f;
    int c = 0;
    reduce_run<32>(L.part + e, L.nelem, L.nparts, c, s);
    reduce_run<8>(L.part + (size_t)c * L.nelem + e, L.nelem, L.nparts, c, s);
    reduce_run<1>(L.part + (size_t)c * L.nelem + e, L.nelem, L.nparts, c, s);
    L.out[e] = s;
  }
}

// ------------------------------------------------------------------------------
// elementwise network stages (bf16 chunk-planar activations)
// ------------------------------------------------------------------------------
// Coarse voxel (I,J,K) of an R/2 grid covers fine voxels (2I..2I+1, 2J.., 2K..).
// The elementwise kernels run one thread per voxel of a line: blockIdx.z = chunk *
// planes + plane, blockIdx.y = line, the voxel from blockIdx.x.
__device__ __forceinline__ size_t child_index(int R, int I, int J, int K, int c) {
  return ((size_t)(2 * I + (c >> 2)) * R + (2 * J + ((c >> 1) & 1))) * R + (2 * K + (c & 1));
}

static dim3 line_grid(int Rl, int kc, int tpb) { return dim3((Rl + tpb - 1) / tpb, Rl, Rl * kc); }
static dim3 quad_grid(int R, int kc, int tpb) { return dim3((R + tpb - 1) / tpb, R / 2, R / 2 * kc); }

// out (R/2) = mean of the 8 children of in (R)
__global__ void __launch_bounds__(64) k_pool2(const uint4 *__restrict__ in, uint4 *__restrict__ out, int R) {
  gc_after();
  const int Rc = R >> 1;
  const int K = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y, c = blockIdx.z / Rc, I = blockIdx.z - c * Rc;
  if (K >= Rc) return;
  const size_t R3 = (size_t)R * R * R, Rc3 = (size_t)Rc * Rc * Rc;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    float f[8];
    unpack8(__ldg(in + c * R3 + child_index(R, I, J, K, ch)), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += f[j];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] *= 0.125f;
  out[c * Rc3 + ((size_t)I * Rc + J) * Rc + K] = pack8<0>(acc);
}

// Two passes over a level's fine grid that add a parent's value to its eight children:
// a thread takes the four children of a parent at its x (blockIdx.z = chunk * R/2 + X,
// blockIdx.y = Y: two lines of two planes), so that each load of the warp is one
// stretch, four (eight) are on their way at once and the parent is read once a line.
// With a voxel per thread (65536 blocks of 64 threads at R = 128, which the chip is slow
// to hand out) the upsampling took 50.7 us on its three levels at R = 128; so 30.4.
__device__ __forceinline__ size_t quad_index(int R, int X, int Y, int q, int z) {
  return ((size_t)(2 * X + (q >> 1)) * R + (2 * Y + (q & 1))) * R + z;
}

// out (R) = relu(u[parent] + skip)
__global__ void __launch_bounds__(64) k_up_add_relu(const uint4 *__restrict__ u, const uint4 *__restrict__ skip,
                                                    uint4 *__restrict__ out, int R) {
  gc_after();
  const int Rc = R >> 1;
  const int z = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y, c = blockIdx.z / Rc, X = blockIdx.z - c * Rc;
  if (z >= R) return;
  const size_t R3 = (size_t)R * R * R, Rc3 = (size_t)Rc * Rc * Rc;
  uint4 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = __ldg(skip + c * R3 + quad_index(R, X, Y, q, z));
  float a[8];
  unpack8(__ldg(u + c * Rc3 + ((size_t)X * Rc + Y) * Rc + (z >> 1)), a);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float b[8];
    unpack8(v[q], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] = fmaxf(a[j] + b[j], 0.0f);
    out[c * R3 + quad_index(R, X, Y, q, z)] = pack8<0>(b);
  }
}

// out (R/2) = sum of the 8 children of g (R): adjoint of the nearest-neighbour upsample
__global__ void __launch_bounds__(64) k_up_adjoint(const uint4 *__restrict__ g, uint4 *__restrict__ out, int R) {
  gc_after();
  const int Rc = R >> 1;
  const int K = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y, c = blockIdx.z / Rc, I = blockIdx.z - c * Rc;
  if (K >= Rc) return;
  const size_t R3 = (size_t)R * R * R, Rc3 = (size_t)Rc * Rc * Rc;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    float f[8];
    unpack8(__ldg(g + c * R3 + child_index(R, I, J, K, ch)), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += f[j];
  }
  out[c * Rc3 + ((size_t)I * Rc + J) * Rc + K] = pack8<0>(acc);
}

// out (R) = (skipgrad + gp[parent] / 8) where act > 0, else 0: the gradient of an
// encoder activation that feeds both a skip connection and the average pool.
__global__ void __launch_bounds__(64) k_pool_adj_add_mask(const uint4 *__restrict__ skipgrad,
                                                          const uint4 *__restrict__ gp, const uint4 *__restrict__ act,
                                                          uint4 *__restrict__ out, int R) {
  gc_after();
  const int Rc = R >> 1;
  const int z = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y, c = blockIdx.z / Rc, X = blockIdx.z - c * Rc;
  if (z >= R) return;
  const size_t R3 = (size_t)R * R * R, Rc3 = (size_t)Rc * Rc * Rc;
  uint4 vs[4], vm[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) vs[q] = __ldg(skipgrad + c * R3 + quad_index(R, X, Y, q, z));
#pragma unroll
  for (int q = 0; q < 4; ++q) vm[q] = __ldg(act + c * R3 + quad_index(R, X, Y, q, z));
  float p[8];
  unpack8(__ldg(gp + c * Rc3 + ((size_t)X * Rc + Y) * Rc + (z >> 1)), p);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float s[8], m[8];
    unpack8(vs[q], s);
    unpack8(vm[q], m);
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = m[j] > 0.0f ? s[j] + 0.125f * p[j] : 0.0f;
    out[c * R3 + quad_index(R, X, Y, q, z)] = pack8<0>(s);
  }
}

// Bias gradients of all layers: per-block partial channel sums of g (C = 8*kc channels),
// part[block][C], nb blocks for each chunk of each layer; then the sums
// of the partials. Two launches where a pair per layer took 2 us a launch.
struct WsBias {
  struct Layer {
    const uint4 *g;
    float *part, *out;
    size_t R3;
    int kc, nb, first;  // chunks, blocks of each, first block of the layer in the grid
  } l[WS_NL];
};
__global__ void __launch_bounds__(256) k_chan_sum(const __grid_constant__ WsBias d) {
  gc_after();
  __shared__ float red[8][8];  // [warp][channel of the chunk]
  int layer = 0;
  while (layer + 1 < WS_NL && (int)blockIdx.x >= d.l[layer + 1].first) ++layer;
  const WsBias::Layer &L = d.l[layer];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kc = L.kc;
  const int c = ((int)blockIdx.x - L.first) / L.nb, blk = (int)blockIdx.x - L.first - c * L.nb;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (size_t v = blk * (size_t)blockDim.x + tid; v < L.R3; v += (size_t)L.nb * blockDim.x) {
    float f[8];
    unpack8(__ldg(L.g + (size_t)c * L.R3 + v), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += f[j];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  }
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) red[warp][j] = acc[j];
  }
  __syncthreads();
  if (tid < 8) {
    float s = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w][tid];
    L.part[(size_t)blk * (8 * kc) + 8 * c + tid] = s;
  }
}
__global__ void __launch_bounds__(256) k_chan_finish(const __grid_constant__ WsBias d) {
  gc_after();
  const WsBias::Layer &L = d.l[blockIdx.y];
  if ((int)blockIdx.x < 8 * L.kc) reduce_col(L.part, L.nb, 8 * L.kc, blockIdx.x, L.out);
}

// Network input: channels 0..3 from f16 planar features [4][R^3]; channels 4..15 zero.
__global__ void __launch_bounds__(256) k_pack_input(const __half *__restrict__ feat, uint4 *__restrict__ x0, size_t R3) {
  gc_after();
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < R3; v += (size_t)gridDim.x * blockDim.x) {
    float f[8] = {__half2float(feat[v]), __half2float(feat[R3 + v]), __half2float(feat[2 * R3 + v]),
                  __half2float(feat[3 * R3 + v]), 0, 0, 0, 0};
    x0[v] = pack8<0>(f);
    x0[R3 + v] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// Loss 0.5 * mean((y - t)^2) over R^3 and its gradient dL/dy (channel 0 of a
// 16-channel bf16 tensor, other channels zero). Per-block partial loss sums.
__global__ void __launch_bounds__(256) k_mse(const float *__restrict__ y, const __half *__restrict__ t, size_t R3,
                                             uint4 *__restrict__ gy, float *__restrict__ part) {
  gc_after();
  __shared__ float red[8];
  const float inv_n = 1.0f / (float)R3;
  float acc = 0.0f;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < R3; v += (size_t)gridDim.x * blockDim.x) {
    const float d = y[v] - __half2float(t[v]);
    acc += d * d;
    float f[8] = {d * inv_n, 0, 0, 0, 0, 0, 0, 0};
    gy[v] = pack8<0>(f);
    gy[R3 + v] = make_uint4(0u, 0u, 0u, 0u);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    part[blockIdx.x] = 0.5f * s * inv_n;
  }
}

// ------------------------------------------------------------------------------
// parameters: Adam and the bf16 packing of the weights
// ------------------------------------------------------------------------------
// Where a layer's parameters and packed weights lie.
struct WsPack {
  struct Layer {
    uint16_t *wf, *wb;
    int off, Cin, Cout;  // W (f32 [27][Cout][Cin]) at params[off], the bias behind it
  } l[WS_NL];
};

// W -> forward operand [27][Cin/8][Cout][8] and data-gradient operand
// [27][Cout/8][Cin][8] with the tap mirrored (t' = 26 - t).
__device__ __forceinline__ void pack_weight(const WsPack::Layer &L, int i, float v) {
  const int t = i / (L.Cout * L.Cin), rem = i - t * L.Cout * L.Cin, co = rem / L.Cin, ci = rem - co * L.Cin;
  const uint16_t u = (uint16_t)(bf_pack(v, 0.0f) & 0xffffu);
  L.wf[(((size_t)t * (L.Cin >> 3) + (ci >> 3)) * L.Cout + co) * 8 + (ci & 7)] = u;
  L.wb[(((size_t)(26 - t) * (L.Cout >> 3) + (co >> 3)) * L.Cin + ci) * 8 + (co & 7)] = u;
}

// All layers' weights in one launch (blockIdx.y is the layer).
__global__ void __launch_bounds__(256) k_pack_weights(const float *__restrict__ p, const __grid_constant__ WsPack d) {
  gc_after();
  const WsPack::Layer &L = d.l[blockIdx.y];
  const int n = 27 * L.Cout * L.Cin;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) pack_weight(L, i, p[L.off + i]);
}

// One Adam step and the packing of the new weights. Every parameter is read, updated and
// packed in one pass: Adam (7.7 us) and eleven packing launches of 1.9 us took 28, this 12.
__global__ void __launch_bounds__(256) k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                                              float *__restrict__ v, const __grid_constant__ WsPack d, float lr, float b1,
                                              float b2, float eps, float bc1, float bc2) {
  gc_after();
  const WsPack::Layer &L = d.l[blockIdx.y];
  const int nw = 27 * L.Cout * L.Cin, n = nw + L.Cout;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int i = L.off + j;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p[i] = pi;
    if (j < nw) pack_weight(L, j, pi);
  }
}

// ------------------------------------------------------------------------------
// the network object
// ------------------------------------------------------------------------------
// Encoder-decoder over 4 levels (R, R/2, R/4, R/8) with 16-32-64-128 channels:
//   e0 = relu(A x0)            p1 = pool(e0)   e1 = relu(B p1)   p2 = pool(e1)
//   e2 = relu(C p2)            p3 = pool(e2)   e3 = relu(D p3)
//   u2 = E e3                  d2 = relu(up(u2) + e2)            f2 = relu(F d2)
//   u1 = G f2                  d1 = relu(up(u1) + e1)            f1 = relu(H d1)
//   u0 = I f1                  d0 = relu(up(u0) + e0)            f0 = relu(J d0)
//   y  = K f0 (channel 0)
// every capital a 3x3x3 convolution with bias (zero padding), pool a 2x2x2 mean,
// up a nearest-neighbour doubling. x0 has 16 channels, 3 in use.
static const int kWsLayer[WS_NL][4] = {  // cin, cout, level, relu
    {16, 16, 0, 1}, {16, 32, 1, 1}, {32, 64, 2, 1}, {64, 128, 3, 1}, {128, 64, 3, 0}, {64, 64, 2, 1},
    {64, 32, 2, 0}, {32, 32, 1, 1}, {32, 16, 1, 0}, {16, 16, 0, 1}, {16, 16, 0, 0}};

struct FwdPlan {
  int BX;  // 0: blocks of whole lines (k_conv_fwd); else strips of BX voxels (k_conv_march)
  int BZ, BY, tpg, n_mt, grid;
  int ns;
  int Cn;  // output channels of a CTA
  uint32_t cols;
  size_t smem;
};
struct WgPlan {
  int BZ, BY, nblocks;
  int grid;         // partial sums
  int groups, sub, tpg;  // tap groups beside each other, of a dz, and taps (or dx) in each
  int dy3, ns;
  uint32_t cols;
  size_t smem;
};

struct gc_ws {
  int R;
  int device;
  cudaStream_t stream;
  size_t nparams;
  size_t w_off[WS_NL], b_off[WS_NL];
  float *params, *grads, *adam_m, *adam_v;
  uint16_t *wf[WS_NL], *wb[WS_NL];
  FwdPlan pf[WS_NL], pb[WS_NL];
  WgPlan pw[WS_NL];
  void *arena;
  uint4 *x0, *e0, *d0, *f0, *gy, *g_f0, *g_d0, *g_e0;
  uint4 *p1, *e1, *u0, *d1, *f1, *g_u0, *g_f1, *g_d1, *g_p1, *g_e1;
  uint4 *p2, *e2, *u1, *d2, *f2, *g_u1, *g_f2, *g_d2, *g_p2, *g_e2;
  uint4 *p3, *e3, *u2, *g_u2, *g_e3, *g_p3;
  float *y;
  float *part;          // weight-gradient partials ..
  size_t pofs[WS_NL];   // .. each layer's behind the other
  WgReduce pend;        // layers whose partials wait for their sums
  int npend;
  float *cpart;
  float *lpart;
  float *loss;
  unsigned *status;
  int sm_count;
  char err[256];
};

static int ws_fail(gc_ws *ws, int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(ws->err, sizeof(ws->err), fmt, ap);
  va_end(ap);
  return code;
}
#define WS_CUDA(ws, call)                                                                        \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess) return ws_fail(ws, GC_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

// Launch on the object's stream; every kernel of the network begins with gc_after() (see
// gc_launch_after).
template <typename... KArgs, typename... Args>
static void ws_launch(gc_ws *ws, void (*k)(KArgs...), dim3 grid, int block, size_t smem, Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ws->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(std::forward<Args>(args))...);
}
static uint32_t pow2_cols(int c) {
  uint32_t n = 32;
  while ((int)n < c) n <<= 1;
  return n;
}

// Shared memory that leaves at most `k` CTAs on an SM (so their Tensor Memory fits).
static size_t smem_for_residency(size_t smem, int k) {
  const size_t per_sm = 233472, reserve = 1024;
  const size_t need = per_sm / (size_t)(k + 1) - reserve + 1;
  return std::max(smem, need);
}

static const size_t WS_SMEM_MAX = 232448;
static const size_t WS_BARS = 64 + 512;  // barriers and the bias of k_conv_fwd

// Tile plans of the convolution. Every feasible block (BZ, BY) and marching strip (BX)
// is enumerated, each for every split of the output channels over CTAs; the default pick
// minimises an estimate in clocks, from clocks taken inside the kernels: staging moves
// 40 bytes a clock and SM, an MMA takes 40 clk (32 to read its 128 operand rows), or Cn / 2
// where that is more, or 57 from a single issuing warp, the epilogue 1000 clk per 16
// channels and pair of M tiles. In a block these follow one another and co-resident CTAs
// share the busiest of them; in a strip they overlap. gc_ws_autotune replaces the pick by
// the fastest measured candidate.
// Where the families meet, forward pass, strips against blocks: 16 -> 16 channels R = 128
// 70 / 155 us, R = 64 13.9 / 18.5; 64 -> 32 R = 16 7.8 / 14.8. Strips want R to be a
// multiple of MA_LINES and all taps in shared memory; splitting the channels makes room
// for the weights of the deep levels (128 -> 64, R = 8: 17.4 us, 25.4 unsplit).
static std::vector<FwdPlan> enum_fwd(int R, int Cin, int Cout, int sm_count, std::vector<double> *costs) {
  std::vector<FwdPlan> out;
  const int bys[] = {32, 16, 8, 4, 2, 1};
  const int bzs[] = {1, 2, 4, 8};
  for (int Cn = Cout; Cn >= 16; Cn >>= 1) {
    const size_t tap = (size_t)Cin * Cn * 2;
    const double mma1 = std::max(40.0, 0.5 * Cn);
    for (int BY : bys) {
      if (BY > R || R % BY) continue;
      for (int BZ : bzs) {
        if (BZ > R || R % BZ) continue;
        int W2, P, V, L0, L1;
        conv_geom(R, BZ, BY, W2, P, V, L0, L1);
        const int n_mt = (L1 - L0 + 128) / 128;
        if (n_mt * Cn > 512) continue;
        const size_t tile = (((size_t)(Cin / 8) * V + 128) * 16 + 1023) & ~(size_t)1023;
        if (tile + 2 * tap + WS_BARS > WS_SMEM_MAX) continue;
        const int tpg = (int)std::min<size_t>(27, (WS_SMEM_MAX - tile - WS_BARS) / (2 * tap));
        const int ngroups = (27 + tpg - 1) / tpg;
        const int tpg_even = (27 + ngroups - 1) / ngroups;
        const size_t smem = tile + 2 * (size_t)tpg_even * tap + WS_BARS;
        FwdPlan p = {};
        p.BZ = BZ; p.BY = BY; p.tpg = tpg_even; p.n_mt = n_mt; p.grid = (R / BZ) * (R / BY);
        p.Cn = Cn;
        p.cols = pow2_cols(n_mt * Cn);
        p.smem = smem_for_residency(smem, (int)(512 / p.cols));
        out.push_back(p);
        if (costs) {
          const int occ = std::max(1, std::min(8, (int)(233472 / (p.smem + 1024))));
          const double load = ((double)(Cin / 8) * V * 16 + 27.0 * tap) / 40.0;
          const double mma = 27.0 * n_mt * (Cin / 16) * (n_mt == 1 ? std::max(57.0, mma1) : mma1) + 1200.0 * ngroups;
          const double epi = 1000.0 * ((n_mt + 1) / 2) * (Cn / 16);
          const double per_cta = load + mma + epi + 2000.0;
          const double busiest = std::max(load, std::max(mma, epi));
          const double ctas = (double)p.grid * (Cout / Cn);
          const double together = std::min<double>(occ, std::ceil(ctas / sm_count));
          costs->push_back(std::ceil(ctas / (sm_count * together)) * (per_cta + (together - 1.0) * busiest));
        }
      }
    }
    // marching strips: MA_LINES lines x BX voxels, all weights in shared memory
    const int bxs[] = {64, 32, 16, 8};  // a line of a box is at most 128 rows
    for (int BX : bxs) {
      if (R % MA_LINES || BX > R || R % BX) continue;
      const int n_mt = BX / 8;
      if (2 * n_mt * Cn > 512) continue;
      const size_t slot = march_slot_bytes(Cin, BX), fixed = 27 * tap + (2 * MA_MAX_SLOTS + 8) * 8 + 512;
      if (fixed + 3 * slot > WS_SMEM_MAX) continue;
      const int units = (R / BX) * (R / MA_LINES) * R, split = Cout / Cn;
      FwdPlan p = {};
      p.BX = BX; p.BZ = 1; p.BY = MA_LINES; p.tpg = 27; p.n_mt = n_mt;
      p.Cn = Cn;
      p.ns = (int)std::min<size_t>(MA_MAX_SLOTS, (WS_SMEM_MAX - fixed) / slot);
      p.cols = pow2_cols(2 * n_mt * Cn);
      p.smem = smem_for_residency(fixed + p.ns * slot, 1);
      p.grid = std::min(units, std::max(1, sm_count / split));
      out.push_back(p);
      if (costs) {
        const int per = (units + p.grid - 1) / p.grid;
        const double load = (double)slot / 40.0;
        const double mma = 27.0 * n_mt * (Cin / 16) * (n_mt == 1 ? std::max(57.0, mma1) : mma1);
        const double epi = 500.0 * ((n_mt + 1) / 2) * (Cn / 16);
        costs->push_back(3000.0 + 27.0 * tap / 40.0 + load + per * std::max(mma + 600.0, std::max(load, epi)) + epi);
      }
    }
  }
  return out;
}

static bool plan_fwd(int R, int Cin, int Cout, int sm_count, FwdPlan &best) {
  std::vector<double> cost;
  const std::vector<FwdPlan> c = enum_fwd(R, Cin, Cout, sm_count, &cost);
  if (c.empty()) return false;
  size_t k = 0;
  for (size_t i = 1; i < c.size(); ++i)
    if (cost[i] < cost[k]) k = i;
  best = c[k];
  return true;
}

// Blocks of the weight gradient and how they run. (BZ, BY) and the number of partials
// belong to the result's bits and follow a score of useful rows, filled SMs and tile
// reuse; how many taps a CTA takes, and how deep its ring is, do not. The taps are divided
// by an estimate in clocks: a CTA's fixed 5000 (measured: set-up, first tile and stage)
// and its products or its stages of gy at 900 each, whichever is more, over the waves
// that shared memory and Tensor Memory make of them. At 16 channels a product takes the
// three dy taps of a channel chunk: 24 columns and 18 products per 16 rows where 27 of 16
// columns need 1.5 times as long.
static std::vector<WgPlan> enum_wgrad(int R, int Cin, int Cout, int sm_count, std::vector<double> *scores) {
  std::vector<WgPlan> out;
  const int bys[] = {32, 16, 8, 4, 2, 1};
  const int bzs[] = {1, 2, 4};
  for (int BY : bys) {
    if (BY > R || R % BY) continue;
    for (int BZ : bzs) {
      if (BZ > R || R % BZ) continue;
      int W2, P, V, L0, L1;
      conv_geom(R, BZ, BY, W2, P, V, L0, L1);
      const size_t tile = (((size_t)(Cin / 8) * V + 128) * 16 + 1023) & ~(size_t)1023;
      // partials: as many as CTAs of one tile and two stages of 32 KB that hold 512 / Cin
      // taps fit the chip
      const size_t ref = tile + 2 * 32768 + 64;
      if (ref > WS_SMEM_MAX) continue;
      const int nst = (L1 - L0 + WG_ROWS) / WG_ROWS;
      const size_t ref_res = smem_for_residency(ref, (int)(512 / pow2_cols(std::min(27, 512 / Cin) * Cin)));
      WgPlan p = {};
      p.BZ = BZ; p.BY = BY; p.nblocks = (R / BZ) * (R / BY);
      p.grid = std::min(p.nblocks, sm_count * std::max(1, (int)(233472 / (ref_res + 1024))));
      p.dy3 = Cin == 16 && Cout <= 64;
      const int all = p.dy3 ? 3 : 9, acc = p.dy3 ? 24 * (Cin / 8) : Cin;  // columns of one of them
      const size_t stage = (size_t)WG_ROWS * 2 * (Cout <= 64 ? 64 : 128), bars = (2 * WG_MAX_STAGES + 5) * 8;
      const size_t dtile = (((size_t)(Cin / 8) * BZ * P + 128) * 16 + 1023) & ~(size_t)1023;  // one dz
      const int most = (p.nblocks + p.grid - 1) / p.grid;  // blocks of a partial
      const int N = p.dy3 ? 24 : Cin;
      const double clk = std::max(0.5 * N, Cout <= 64 ? 24.0 : 32.0 + 0.25 * N);
      double best = 0.0;
      for (int sub = 1; sub <= all; ++sub) {
        const int tpg = (all + sub - 1) / sub;
        if (tpg * acc > 512 || (sub > 1 && tpg == (all + sub - 2) / (sub - 1))) continue;
        const uint32_t cols = pow2_cols(tpg * acc);
        int ns = (int)std::min<size_t>(std::min(WG_MAX_STAGES, most * nst), (WS_SMEM_MAX - dtile - bars) / stage);
        if (ns > 4) ns = 4;
        const size_t smem = smem_for_residency(dtile + ns * stage + bars, (int)(512 / cols));
        const int res = std::max(1, std::min(4, (int)(233472 / (smem + 1024))));
        const double prod = (double)most * nst * (WG_ROWS / 16) * tpg * (p.dy3 ? Cin / 8 : 1) * clk;
        const double waves = std::ceil(3.0 * p.grid * sub / ((double)sm_count * res));
        const double cost = waves * std::max(5000.0 + std::max(prod, 900.0 * most * nst), res * prod);
        if (best == 0.0 || cost < best) {
          best = cost;
          p.sub = sub; p.tpg = tpg; p.groups = 3 * sub; p.cols = cols; p.ns = ns; p.smem = smem;
        }
      }
      if (best == 0.0) continue;
      out.push_back(p);
      if (scores) {
        const double useful = (double)BZ * BY * R / (128.0 * nst);
        const double fill = std::min(1.0, (double)p.nblocks / (double)sm_count);
        const double reload = (double)(BZ * BY) / ((BZ + 2.0) * (BY + 2.0));
        scores->push_back(useful * fill * (0.5 + 0.5 * reload));
      }
    }
  }
  return out;
}

static bool plan_wgrad(int R, int Cin, int Cout, int sm_count, WgPlan &best) {
  std::vector<double> sc;
  const std::vector<WgPlan> c = enum_wgrad(R, Cin, Cout, sm_count, &sc);
  if (c.empty()) return false;
  size_t k = 0;
  for (size_t i = 1; i < c.size(); ++i)
    if (sc[i] > sc[k]) k = i;
  best = c[k];
  return true;
}

static unsigned ew_blocks(size_t n, int sm_count) {
  size_t b = (n + 255) / 256;
  const size_t cap = (size_t)sm_count * 8;
  if (b > cap) b = cap;
  return (unsigned)std::max<size_t>(1, b);
}

// Tensor map over a channel-chunk planar activation (kci chunks of R^3 16-byte rows).
// A row is two 8-byte elements, so a box spans up to 128 voxels along x and x
// coordinates are even, 16-byte aligned. `order` names the dimensions after x, nearest
// first. The encoder is reached through the runtime: the library does not link the
// driver. `base` belongs to the network object; maps are made for each launch (below a
// microsecond) and not kept.
enum WsDim { WS_Y, WS_Z, WS_C };
static int ws_tmap(gc_ws *ws, CUtensorMap *map, const uint4 *base, int R, int kci, const WsDim (&order)[3], int bx, int b1,
                   int b2, int b3) {
  typedef CUresult (*encode_t)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                               const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const encode_t encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return (encode_t)fn;
  }();
  if (!encode) return ws_fail(ws, GC_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t n = (cuuint64_t)R, size[3] = {n, n, (cuuint64_t)kci}, stride[3] = {n * 16, n * n * 16, n * n * n * 16};
  const cuuint64_t dims[4] = {2 * n, size[order[0]], size[order[1]], size[order[2]]};
  const cuuint64_t strides[3] = {stride[order[0]], stride[order[1]], stride[order[2]]};
  const cuuint32_t box[4] = {2u * (cuuint32_t)bx, (cuuint32_t)b1, (cuuint32_t)b2, (cuuint32_t)b3};
  const cuuint32_t one[4] = {1, 1, 1, 1};
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<uint4 *>(base), dims, strides, box, one,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return ws_fail(ws, GC_ERR_CUDA, "cuTensorMapEncodeTiled failed (R = %d, %d chunks)", R, kci);
  return GC_OK;
}

static int ws_conv(gc_ws *ws, const FwdPlan &p, int R, int Cin, int Cout, const uint4 *in, const uint16_t *w,
                   const float *bias, const uint4 *skip, const uint4 *mask, uint4 *out, float *out_f32, int relu) {
  if (p.BX) {
    ConvMarch m = {};
    const int st = ws_tmap(ws, &m.map, in, R, Cin / 8, {WS_C, WS_Y, WS_Z}, p.BX + 2, Cin / 8, MA_LINES + 2, 1);
    if (st) return st;
    m.w = reinterpret_cast<const uint4 *>(w); m.bias = bias; m.skip = skip; m.mask = mask;
    m.out = out; m.out_f32 = out_f32; m.status = ws->status;
    m.R = R; m.Cin = Cin; m.Cout = Cout; m.BX = p.BX; m.Cn = p.Cn; m.relu = relu; m.ns = p.ns;
    m.units = (R / p.BX) * (R / MA_LINES) * R;
    m.tmem_cols = p.cols;
    ws_launch(ws, k_conv_march, dim3(p.grid, Cout / p.Cn), MA_THREADS, p.smem, m);
    WS_CUDA(ws, cudaGetLastError());
    return GC_OK;
  }
  ConvFwd a = {};
  a.use_map = R <= 126;
  if (a.use_map) {
    const int st = ws_tmap(ws, &a.map, in, R, Cin / 8, {WS_Y, WS_Z, WS_C}, R + 2, p.BY + 2, p.BZ + 2, Cin / 8);
    if (st) return st;
  }
  a.in = in; a.w = reinterpret_cast<const uint4 *>(w); a.bias = bias; a.skip = skip; a.mask = mask;
  a.out = out; a.out_f32 = out_f32; a.status = ws->status;
  a.R = R; a.Cin = Cin; a.Cout = Cout; a.BZ = p.BZ; a.BY = p.BY; a.Cn = p.Cn; a.relu = relu; a.tpg = p.tpg; a.n_mt = p.n_mt;
  a.tmem_cols = p.cols;
  ws_launch(ws, k_conv_fwd, dim3(p.grid, Cout / p.Cn), 256, p.smem, a);
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

static int ws_wgrad(gc_ws *ws, int l, const uint4 *x, const uint4 *gy) {
  const int Cin = kWsLayer[l][0], Cout = kWsLayer[l][1], R = ws->R >> kWsLayer[l][2];
  const WgPlan &p = ws->pw[l];
  ConvW a = {};
  a.use_map = R <= 126;
  if (a.use_map) {
    const int st = ws_tmap(ws, &a.map, x, R, Cin / 8, {WS_Y, WS_Z, WS_C}, R + 2, p.BY + 2, p.BZ, Cin / 8);
    if (st) return st;
  }
  a.x = x; a.gy = gy; a.part = ws->part + ws->pofs[l]; a.status = ws->status;
  a.R = R; a.Cin = Cin; a.Cout = Cout; a.BZ = p.BZ; a.BY = p.BY; a.nblocks = p.nblocks;
  a.tpg = p.tpg; a.sub = p.sub; a.dy3 = p.dy3; a.ns = p.ns; a.tmem_cols = p.cols;
  ws_launch(ws, k_conv_wgrad, dim3(p.groups, p.grid), WG_THREADS, p.smem, a);
  WS_CUDA(ws, cudaGetLastError());
  ws->pend.l[ws->npend++] = {a.part, ws->grads + ws->w_off[l], p.grid, 27 * Cout * Cin};
  return GC_OK;
}

// The sums of the layers that wait for them.
static int ws_wgrad_finish(gc_ws *ws) {
  int most = 0;
  for (int i = 0; i < ws->npend; ++i) most = std::max(most, ws->pend.l[i].nelem);
  const unsigned nb = std::min<unsigned>((unsigned)(most + 63) / 64, (unsigned)ws->sm_count * 8u);
  if (ws->npend) ws_launch(ws, k_wgrad_reduce, dim3(nb, ws->npend), 64, 0, ws->pend);
  ws->npend = 0;
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

// Bias gradients of every layer, from the output gradients of a whole backward pass.
static int ws_bias_grads(gc_ws *ws) {
  const uint4 *g[WS_NL] = {ws->g_e0, ws->g_e1, ws->g_e2, ws->g_e3, ws->g_u2, ws->g_f2, ws->g_u1, ws->g_f1, ws->g_u0,
                           ws->g_f0, ws->gy};
  WsBias d;
  int blocks = 0;
  for (int l = 0; l < WS_NL; ++l) {
    const size_t R = (size_t)(ws->R >> kWsLayer[l][2]), R3 = R * R * R;
    const int nb = (int)std::min<unsigned>(ew_blocks(R3, ws->sm_count), 1024u), kc = kWsLayer[l][1] / 8;
    d.l[l] = {g[l], ws->cpart + (size_t)l * 1024 * 128, ws->grads + ws->b_off[l], R3, kc, nb, blocks};
    blocks += nb * kc;
  }
  ws_launch(ws, k_chan_sum, dim3(blocks), 256, 0, d);
  ws_launch(ws, k_chan_finish, dim3(128, WS_NL), 256, 0, d);
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

static int ws_fwd_layer(gc_ws *ws, int l, const uint4 *in, const uint4 *skip, uint4 *out, float *out_f32) {
  const int R = ws->R >> kWsLayer[l][2];
  return ws_conv(ws, ws->pf[l], R, kWsLayer[l][0], kWsLayer[l][1], in, ws->wf[l], ws->params + ws->b_off[l], skip,
                 nullptr, out, out_f32, kWsLayer[l][3]);
}

// data gradient of layer l: conv of g (Cout channels) with the mirrored weights,
// optionally masked by (act > 0)
static int ws_dgrad(gc_ws *ws, int l, const uint4 *g, const uint4 *mask_act, uint4 *out) {
  const int R = ws->R >> kWsLayer[l][2];
  return ws_conv(ws, ws->pb[l], R, kWsLayer[l][1], kWsLayer[l][0], g, ws->wb[l], nullptr, nullptr, mask_act, out,
                 nullptr, 0);
}

extern "C" int gc_ws_layer_info(int layer, int *cin, int *cout, int *level, int *relu) {
  if (layer < 0 || layer >= WS_NL) return GC_ERR_ARG;
  if (cin) *cin = kWsLayer[layer][0];
  if (cout) *cout = kWsLayer[layer][1];
  if (level) *level = kWsLayer[layer][2];
  if (relu) *relu = kWsLayer[layer][3];
  return GC_OK;
}

extern "C" int gc_ws_create(gc_ws **out, int R) {
  if (!out) return GC_ERR_ARG;
  *out = nullptr;
  if (R < 16 || R > 512 || (R % 8)) return GC_ERR_ARG;
  gc_ws *ws = new (std::nothrow) gc_ws();
  if (!ws) return GC_ERR_CUDA;
  memset(ws, 0, sizeof(*ws));
  ws->R = R;
  cudaGetDevice(&ws->device);
  cudaDeviceGetAttribute(&ws->sm_count, cudaDevAttrMultiProcessorCount, ws->device);
  if (ws->sm_count <= 0) ws->sm_count = (int)gc_sms();
  size_t off = 0;
  for (int l = 0; l < WS_NL; ++l) {
    ws->w_off[l] = off;
    off += (size_t)27 * kWsLayer[l][0] * kWsLayer[l][1];
    ws->b_off[l] = off;
    off += kWsLayer[l][1];
  }
  ws->nparams = off;
  size_t wbytes = 0;
  for (int l = 0; l < WS_NL; ++l) wbytes += (size_t)27 * kWsLayer[l][0] * kWsLayer[l][1] * 2 * 2;
  int rc = GC_OK;
  auto fail = [&](const char *what) {
    snprintf(ws->err, sizeof(ws->err), "gc_ws_create: %s", what);
    rc = GC_ERR_CUDA;
  };
  if (cudaMalloc(&ws->params, 4 * ws->nparams * sizeof(float)) != cudaSuccess) fail("parameters");
  if (rc == GC_OK) {
    ws->grads = ws->params + ws->nparams;
    ws->adam_m = ws->grads + ws->nparams;
    ws->adam_v = ws->adam_m + ws->nparams;
    cudaMemset(ws->params, 0, 4 * ws->nparams * sizeof(float));
  }
  uint16_t *wall = nullptr;
  if (rc == GC_OK && cudaMalloc(&wall, wbytes) != cudaSuccess) fail("bf16 weights");
  if (rc == GC_OK) {
    cudaMemset(wall, 0, wbytes);
    for (int l = 0; l < WS_NL; ++l) {
      const size_t nw = (size_t)27 * kWsLayer[l][0] * kWsLayer[l][1];
      ws->wf[l] = wall;
      ws->wb[l] = wall + nw;
      wall += 2 * nw;
    }
  }
  // activations
  const size_t R3[4] = {(size_t)R * R * R, (size_t)R * R * R / 8, (size_t)R * R * R / 64, (size_t)R * R * R / 512};
  struct Req { uint4 **p; int ch; int lev; };
  const Req reqs[] = {
      {&ws->x0, 16, 0}, {&ws->e0, 16, 0}, {&ws->d0, 16, 0}, {&ws->f0, 16, 0}, {&ws->gy, 16, 0}, {&ws->g_f0, 16, 0},
      {&ws->g_d0, 16, 0}, {&ws->g_e0, 16, 0},
      {&ws->p1, 16, 1}, {&ws->e1, 32, 1}, {&ws->u0, 16, 1}, {&ws->d1, 32, 1}, {&ws->f1, 32, 1}, {&ws->g_u0, 16, 1},
      {&ws->g_f1, 32, 1}, {&ws->g_d1, 32, 1}, {&ws->g_p1, 16, 1}, {&ws->g_e1, 32, 1},
      {&ws->p2, 32, 2}, {&ws->e2, 64, 2}, {&ws->u1, 32, 2}, {&ws->d2, 64, 2}, {&ws->f2, 64, 2}, {&ws->g_u1, 32, 2},
      {&ws->g_f2, 64, 2}, {&ws->g_d2, 64, 2}, {&ws->g_p2, 32, 2}, {&ws->g_e2, 64, 2},
      {&ws->p3, 64, 3}, {&ws->e3, 128, 3}, {&ws->u2, 64, 3}, {&ws->g_u2, 64, 3}, {&ws->g_e3, 128, 3},
      {&ws->g_p3, 64, 3}};
  size_t abytes = 0;
  for (const Req &q : reqs) abytes += ((R3[q.lev] * (q.ch / 8) * 16 + 255) & ~(size_t)255);
  abytes += ((R3[0] * 4 + 255) & ~(size_t)255);  // y
  if (rc == GC_OK && cudaMalloc(&ws->arena, abytes) != cudaSuccess) fail("activations");
  if (rc == GC_OK) {
    cudaMemset(ws->arena, 0, abytes);
    uint8_t *p = (uint8_t *)ws->arena;
    for (const Req &q : reqs) {
      *q.p = (uint4 *)p;
      p += ((R3[q.lev] * (q.ch / 8) * 16 + 255) & ~(size_t)255);
    }
    ws->y = (float *)p;
  }
  // plans
  for (int l = 0; l < WS_NL && rc == GC_OK; ++l) {
    const int Rl = R >> kWsLayer[l][2];
    if (!plan_fwd(Rl, kWsLayer[l][0], kWsLayer[l][1], ws->sm_count, ws->pf[l]) ||
        !plan_fwd(Rl, kWsLayer[l][1], kWsLayer[l][0], ws->sm_count, ws->pb[l]) ||
        !plan_wgrad(Rl, kWsLayer[l][0], kWsLayer[l][1], ws->sm_count, ws->pw[l])) {
      snprintf(ws->err, sizeof(ws->err), "gc_ws_create: no tile plan for layer %d", l);
      rc = GC_ERR_ARG;
    }
  }
  size_t part = 0;  // weight-gradient partials: the most any candidate plan of a layer may use
  for (int l = 0; l < WS_NL && rc == GC_OK; ++l) {
    const int Rl = R >> kWsLayer[l][2];
    size_t most = 0;
    for (const WgPlan &c : enum_wgrad(Rl, kWsLayer[l][0], kWsLayer[l][1], ws->sm_count, nullptr))
      most = std::max(most, (size_t)c.grid * 27 * kWsLayer[l][0] * kWsLayer[l][1]);
    ws->pofs[l] = part;
    part += (most + 63) & ~(size_t)63;
  }
  if (rc == GC_OK && cudaMalloc(&ws->part, part * sizeof(float) + (size_t)(WS_NL * 1024 * 128 + 1024 + 16) * sizeof(float) +
                                               64) != cudaSuccess)
    fail("partials");
  if (rc == GC_OK) {
    ws->cpart = ws->part + part;
    ws->lpart = ws->cpart + WS_NL * 1024 * 128;
    ws->loss = ws->lpart + 1024;
    ws->status = (unsigned *)(ws->loss + 8);
    cudaMemset(ws->status, 0, sizeof(unsigned));
  }
  if (rc == GC_OK) {
    if (cudaFuncSetAttribute(k_conv_march, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_MAX) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_conv_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_MAX) != cudaSuccess ||
        cudaFuncSetAttribute(k_conv_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM_MAX) !=
            cudaSuccess)
      fail("shared memory attribute");
  }
  if (rc != GC_OK) {
    char msg[256];
    memcpy(msg, ws->err, sizeof(msg));
    gc_ws_destroy(ws);
    fprintf(stderr, "%s\n", msg);
    return rc;
  }
  *out = ws;
  return GC_OK;
}

extern "C" int gc_ws_destroy(gc_ws *ws) {
  if (!ws) return GC_OK;
  if (ws->params) cudaFree(ws->params);
  if (ws->wf[0]) cudaFree(ws->wf[0]);
  if (ws->arena) cudaFree(ws->arena);
  if (ws->part) cudaFree(ws->part);
  delete ws;
  return GC_OK;
}

extern "C" const char *gc_ws_last_error(const gc_ws *ws) { return ws ? ws->err : "null warm-start object"; }

extern "C" int gc_ws_set_stream(gc_ws *ws, void *stream) {
  if (!ws) return GC_ERR_ARG;
  ws->stream = (cudaStream_t)stream;
  return GC_OK;
}

extern "C" int gc_ws_num_params(const gc_ws *ws, int64_t *n) {
  if (!ws || !n) return GC_ERR_ARG;
  *n = (int64_t)ws->nparams;
  return GC_OK;
}

static WsPack ws_pack_desc(const gc_ws *ws) {
  WsPack d;
  for (int l = 0; l < WS_NL; ++l) d.l[l] = {ws->wf[l], ws->wb[l], (int)ws->w_off[l], kWsLayer[l][0], kWsLayer[l][1]};
  return d;
}

static int ws_repack(gc_ws *ws) {
  ws_launch(ws, k_pack_weights, dim3(512, WS_NL), 256, 0, ws->params, ws_pack_desc(ws));
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

extern "C" int gc_ws_set_params(gc_ws *ws, const float *params) {
  if (!ws || !params) return GC_ERR_ARG;
  WS_CUDA(ws, cudaMemcpyAsync(ws->params, params, ws->nparams * sizeof(float), cudaMemcpyDeviceToDevice, ws->stream));
  WS_CUDA(ws, cudaMemsetAsync(ws->adam_m, 0, 2 * ws->nparams * sizeof(float), ws->stream));
  return ws_repack(ws);
}

extern "C" int gc_ws_get_params(gc_ws *ws, float *params) {
  if (!ws || !params) return GC_ERR_ARG;
  WS_CUDA(ws, cudaMemcpyAsync(params, ws->params, ws->nparams * sizeof(float), cudaMemcpyDeviceToDevice, ws->stream));
  return GC_OK;
}

extern "C" int gc_ws_get_grads(gc_ws *ws, float *grads) {
  if (!ws || !grads) return GC_ERR_ARG;
  WS_CUDA(ws, cudaMemcpyAsync(grads, ws->grads, ws->nparams * sizeof(float), cudaMemcpyDeviceToDevice, ws->stream));
  return GC_OK;
}

extern "C" int gc_ws_status(gc_ws *ws, unsigned *flags, int clear) {
  if (!ws || !flags) return GC_ERR_ARG;
  WS_CUDA(ws, cudaMemcpyAsync(flags, ws->status, sizeof(unsigned), cudaMemcpyDeviceToHost, ws->stream));
  WS_CUDA(ws, cudaStreamSynchronize(ws->stream));
  if (clear) WS_CUDA(ws, cudaMemsetAsync(ws->status, 0, sizeof(unsigned), ws->stream));
  return GC_OK;
}

static int ws_forward_packed(gc_ws *ws, float *y_out) {
  const int R = ws->R;
  int s;
  if ((s = ws_fwd_layer(ws, 0, ws->x0, nullptr, ws->e0, nullptr))) return s;
  ws_launch(ws, k_pool2, dim3(line_grid(R / 2, 2, 64)), 64, 0, ws->e0, ws->p1, R);
  if ((s = ws_fwd_layer(ws, 1, ws->p1, nullptr, ws->e1, nullptr))) return s;
  ws_launch(ws, k_pool2, dim3(line_grid(R / 4, 4, 64)), 64, 0, ws->e1, ws->p2, R / 2);
  if ((s = ws_fwd_layer(ws, 2, ws->p2, nullptr, ws->e2, nullptr))) return s;
  ws_launch(ws, k_pool2, dim3(line_grid(R / 8, 8, 64)), 64, 0, ws->e2, ws->p3, R / 4);
  if ((s = ws_fwd_layer(ws, 3, ws->p3, nullptr, ws->e3, nullptr))) return s;
  if ((s = ws_fwd_layer(ws, 4, ws->e3, nullptr, ws->u2, nullptr))) return s;
  ws_launch(ws, k_up_add_relu, dim3(quad_grid(R / 4, 8, 64)), 64, 0, ws->u2, ws->e2, ws->d2, R / 4);
  if ((s = ws_fwd_layer(ws, 5, ws->d2, nullptr, ws->f2, nullptr))) return s;
  if ((s = ws_fwd_layer(ws, 6, ws->f2, nullptr, ws->u1, nullptr))) return s;
  ws_launch(ws, k_up_add_relu, dim3(quad_grid(R / 2, 4, 64)), 64, 0, ws->u1, ws->e1, ws->d1, R / 2);
  if ((s = ws_fwd_layer(ws, 7, ws->d1, nullptr, ws->f1, nullptr))) return s;
  if ((s = ws_fwd_layer(ws, 8, ws->f1, nullptr, ws->u0, nullptr))) return s;
  ws_launch(ws, k_up_add_relu, dim3(quad_grid(R, 2, 64)), 64, 0, ws->u0, ws->e0, ws->d0, R);
  if ((s = ws_fwd_layer(ws, 9, ws->d0, nullptr, ws->f0, nullptr))) return s;
  if ((s = ws_fwd_layer(ws, 10, ws->f0, nullptr, nullptr, y_out ? y_out : ws->y))) return s;
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

extern "C" int gc_ws_forward(gc_ws *ws, const void *feat, float *y_out) {
  if (!ws || !feat) return GC_ERR_ARG;
  const size_t R3 = (size_t)ws->R * ws->R * ws->R;
  ws_launch(ws, k_pack_input, dim3(ew_blocks(R3, ws->sm_count)), 256, 0, (const __half *)feat, ws->x0, R3);
  WS_CUDA(ws, cudaGetLastError());
  int s = ws_forward_packed(ws, ws->y);
  if (s) return s;
  if (y_out) WS_CUDA(ws, cudaMemcpyAsync(y_out, ws->y, R3 * sizeof(float), cudaMemcpyDeviceToDevice, ws->stream));
  return GC_OK;
}

extern "C" int gc_ws_backward(gc_ws *ws, const void *target, float *loss_out) {
  if (!ws || !target) return GC_ERR_ARG;
  const int R = ws->R;
  const size_t R3 = (size_t)R * R * R;
  const int sm = ws->sm_count;
  int s;
  const unsigned nl = std::min<unsigned>(ew_blocks(R3, sm), 1024u);
  ws->npend = 0;
  ws_launch(ws, k_mse, dim3(nl), 256, 0, ws->y, (const __half *)target, R3, ws->gy, ws->lpart);
  ws_launch(ws, k_reduce_cols, dim3(1), 256, 0, ws->lpart, (int)nl, 1, ws->loss);
  WS_CUDA(ws, cudaGetLastError());
  // K, J
  if ((s = ws_wgrad(ws, 10, ws->f0, ws->gy))) return s;
  if ((s = ws_dgrad(ws, 10, ws->gy, ws->f0, ws->g_f0))) return s;
  if ((s = ws_wgrad(ws, 9, ws->d0, ws->g_f0))) return s;
  if ((s = ws_dgrad(ws, 9, ws->g_f0, ws->d0, ws->g_d0))) return s;
  ws_launch(ws, k_up_adjoint, dim3(line_grid(R / 2, 2, 64)), 64, 0, ws->g_d0, ws->g_u0, R);
  // I, H
  if ((s = ws_wgrad(ws, 8, ws->f1, ws->g_u0))) return s;
  if ((s = ws_dgrad(ws, 8, ws->g_u0, ws->f1, ws->g_f1))) return s;
  if ((s = ws_wgrad(ws, 7, ws->d1, ws->g_f1))) return s;
  if ((s = ws_dgrad(ws, 7, ws->g_f1, ws->d1, ws->g_d1))) return s;
  ws_launch(ws, k_up_adjoint, dim3(line_grid(R / 4, 4, 64)), 64, 0, ws->g_d1, ws->g_u1, R / 2);
  // G, F
  if ((s = ws_wgrad(ws, 6, ws->f2, ws->g_u1))) return s;
  if ((s = ws_dgrad(ws, 6, ws->g_u1, ws->f2, ws->g_f2))) return s;
  if ((s = ws_wgrad(ws, 5, ws->d2, ws->g_f2))) return s;
  if ((s = ws_dgrad(ws, 5, ws->g_f2, ws->d2, ws->g_d2))) return s;
  ws_launch(ws, k_up_adjoint, dim3(line_grid(R / 8, 8, 64)), 64, 0, ws->g_d2, ws->g_u2, R / 4);
  // E, D
  if ((s = ws_wgrad(ws, 4, ws->e3, ws->g_u2))) return s;
  if ((s = ws_dgrad(ws, 4, ws->g_u2, ws->e3, ws->g_e3))) return s;
  if ((s = ws_wgrad(ws, 3, ws->p3, ws->g_e3))) return s;
  if ((s = ws_dgrad(ws, 3, ws->g_e3, nullptr, ws->g_p3))) return s;
  ws_launch(ws, k_pool_adj_add_mask, dim3(quad_grid(R / 4, 8, 64)), 64, 0, ws->g_d2, ws->g_p3, ws->e2, ws->g_e2, R / 4);
  // C
  if ((s = ws_wgrad(ws, 2, ws->p2, ws->g_e2))) return s;
  if ((s = ws_dgrad(ws, 2, ws->g_e2, nullptr, ws->g_p2))) return s;
  ws_launch(ws, k_pool_adj_add_mask, dim3(quad_grid(R / 2, 4, 64)), 64, 0, ws->g_d1, ws->g_p2, ws->e1, ws->g_e1, R / 2);
  // B
  if ((s = ws_wgrad(ws, 1, ws->p1, ws->g_e1))) return s;
  if ((s = ws_dgrad(ws, 1, ws->g_e1, nullptr, ws->g_p1))) return s;
  ws_launch(ws, k_pool_adj_add_mask, dim3(quad_grid(R, 2, 64)), 64, 0, ws->g_d0, ws->g_p1, ws->e0, ws->g_e0, R);
  // A
  if ((s = ws_wgrad(ws, 0, ws->x0, ws->g_e0))) return s;
  if ((s = ws_wgrad_finish(ws)) || (s = ws_bias_grads(ws))) return s;
  WS_CUDA(ws, cudaGetLastError());
  if (loss_out) WS_CUDA(ws, cudaMemcpyAsync(loss_out, ws->loss, sizeof(float), cudaMemcpyDeviceToDevice, ws->stream));
  return GC_OK;
}

// ---- autotuner --------------------------------------------------------------------
// Buffers each layer reads and writes in the forward, data-gradient and
// weight-gradient passes (the autotuner times candidates on them).
struct WsBufs {
  const uint4 *in;
  uint4 *out;
  const uint4 *mask;
  float *outf;
};
static WsBufs fwd_bufs(gc_ws *ws, int l) {
  const uint4 *in[WS_NL] = {ws->x0, ws->p1, ws->p2, ws->p3, ws->e3, ws->d2, ws->f2, ws->d1, ws->f1, ws->d0, ws->f0};
  uint4 *out[WS_NL] = {ws->e0, ws->e1, ws->e2, ws->e3, ws->u2, ws->f2, ws->u1, ws->f1, ws->u0, ws->f0, nullptr};
  return {in[l], out[l], nullptr, l == WS_NL - 1 ? ws->y : nullptr};
}
static WsBufs dgrad_bufs(gc_ws *ws, int l) {  // l >= 1
  const uint4 *in[WS_NL] = {nullptr, ws->g_e1, ws->g_e2, ws->g_e3, ws->g_u2, ws->g_f2, ws->g_u1, ws->g_f1, ws->g_u0,
                            ws->g_f0, ws->gy};
  uint4 *out[WS_NL] = {nullptr, ws->g_p1, ws->g_p2, ws->g_p3, ws->g_e3, ws->g_d2, ws->g_f2, ws->g_d1, ws->g_f1,
                       ws->g_d0, ws->g_f0};
  const uint4 *mask[WS_NL] = {nullptr, nullptr, nullptr, nullptr, ws->e3, ws->d2, ws->f2, ws->d1, ws->f1, ws->d0,
                              ws->f0};
  return {in[l], out[l], mask[l], nullptr};
}
static WsBufs wgrad_bufs(gc_ws *ws, int l) {  // in = layer input, mask = output gradient
  const uint4 *x[WS_NL] = {ws->x0, ws->p1, ws->p2, ws->p3, ws->e3, ws->d2, ws->f2, ws->d1, ws->f1, ws->d0, ws->f0};
  const uint4 *g[WS_NL] = {ws->g_e0, ws->g_e1, ws->g_e2, ws->g_e3, ws->g_u2, ws->g_f2, ws->g_u1, ws->g_f1, ws->g_u0,
                           ws->g_f0, ws->gy};
  return {x[l], nullptr, g[l], nullptr};
}

// Time every feasible tile plan of every layer's three passes (CUDA events,
// `iters` launches after one untimed) and keep the fastest. Activations are
// overwritten. ms_out (host, nullable) receives the best time per pass,
// [layer][forward, data gradient, weight gradient], 0 where a pass does not exist.
extern "C" int gc_ws_autotune(gc_ws *ws, int iters, float *ms_out) {
  if (!ws || iters < 1) return GC_ERR_ARG;
  cudaEvent_t ev0, ev1;
  WS_CUDA(ws, cudaEventCreate(&ev0));
  WS_CUDA(ws, cudaEventCreate(&ev1));
  int rc = GC_OK;
  for (int l = 0; l < WS_NL && rc == GC_OK; ++l) {
    const int Cin = kWsLayer[l][0], Cout = kWsLayer[l][1], R = ws->R >> kWsLayer[l][2];
    for (int kind = 0; kind < 3 && rc == GC_OK; ++kind) {
      float best = 3.0e38f;
      if (kind == 2) {
        const std::vector<WgPlan> c = enum_wgrad(R, Cin, Cout, ws->sm_count, nullptr);
        const WsBufs b = wgrad_bufs(ws, l);
        WgPlan keep = ws->pw[l];
        for (const WgPlan &p : c) {
          ws->pw[l] = p;
          if ((rc = ws_wgrad(ws, l, b.in, b.mask)) || (rc = ws_wgrad_finish(ws))) break;
          cudaEventRecord(ev0, ws->stream);
          for (int i = 0; i < iters && rc == GC_OK; ++i)
            if (!(rc = ws_wgrad(ws, l, b.in, b.mask))) rc = ws_wgrad_finish(ws);
          cudaEventRecord(ev1, ws->stream);
          cudaEventSynchronize(ev1);
          float ms = 0.0f;
          cudaEventElapsedTime(&ms, ev0, ev1);
          if (ms < best) { best = ms; keep = p; }
        }
        ws->pw[l] = keep;
      } else {
        if (kind == 1 && l == 0) { if (ms_out) ms_out[3 * l + kind] = 0.0f; continue; }
        const int ci = kind == 0 ? Cin : Cout, co = kind == 0 ? Cout : Cin;
        const std::vector<FwdPlan> c = enum_fwd(R, ci, co, ws->sm_count, nullptr);
        const WsBufs b = kind == 0 ? fwd_bufs(ws, l) : dgrad_bufs(ws, l);
        FwdPlan &slot = kind == 0 ? ws->pf[l] : ws->pb[l];
        FwdPlan keep = slot;
        const uint16_t *w = kind == 0 ? ws->wf[l] : ws->wb[l];
        const float *bias = kind == 0 ? ws->params + ws->b_off[l] : nullptr;
        const int relu = kind == 0 ? kWsLayer[l][3] : 0;
        for (const FwdPlan &p : c) {
          if ((rc = ws_conv(ws, p, R, ci, co, b.in, w, bias, nullptr, b.mask, b.out, b.outf, relu))) break;
          cudaEventRecord(ev0, ws->stream);
          for (int i = 0; i < iters && rc == GC_OK; ++i)
            rc = ws_conv(ws, p, R, ci, co, b.in, w, bias, nullptr, b.mask, b.out, b.outf, relu);
          cudaEventRecord(ev1, ws->stream);
          cudaEventSynchronize(ev1);
          float ms = 0.0f;
          cudaEventElapsedTime(&ms, ev0, ev1);
          if (ms < best) { best = ms; keep = p; }
        }
        slot = keep;
      }
      if (ms_out) ms_out[3 * l + kind] = best < 3.0e38f ? best / (float)iters : 0.0f;
    }
  }
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  if (rc == GC_OK) WS_CUDA(ws, cudaGetLastError());
  return rc;
}

static int ws_cout(int l, int kind) { return kWsLayer[l][kind == 0 ? 1 : 0]; }

// The plan in use: out[0..4] = BZ, BY, taps per group (or per pass), CTAs, M tiles
// (0 for the weight gradient). kind 0 forward, 1 data gradient, 2 weight gradient.
extern "C" int gc_ws_plan_info(const gc_ws *ws, int layer, int kind, int *out) {
  if (!ws || !out || layer < 0 || layer >= WS_NL || kind < 0 || kind > 2) return GC_ERR_ARG;
  if (kind == 2) {
    const WgPlan &p = ws->pw[layer];
    out[0] = p.BZ; out[1] = p.BY; out[2] = p.dy3 ? 3 * p.tpg : p.tpg; out[3] = p.grid * p.groups; out[4] = 0;
  } else {
    const FwdPlan &p = kind == 0 ? ws->pf[layer] : ws->pb[layer];
    out[0] = p.BZ; out[1] = p.BY; out[2] = p.tpg; out[3] = p.grid * ws_cout(layer, kind) / p.Cn; out[4] = p.n_mt;
  }
  return GC_OK;
}

// Take candidate `index` of the plans of (layer, kind); *count receives how many there
// are. A negative index only counts.
extern "C" int gc_ws_set_plan(gc_ws *ws, int layer, int kind, int index, int *count) {
  if (!ws || layer < 0 || layer >= WS_NL || kind < 0 || kind > 2) return GC_ERR_ARG;
  const int Cin = kWsLayer[layer][0], Cout = kWsLayer[layer][1], R = ws->R >> kWsLayer[layer][2];
  if (kind == 2) {
    const std::vector<WgPlan> c = enum_wgrad(R, Cin, Cout, ws->sm_count, nullptr);
    if (count) *count = (int)c.size();
    if (index >= (int)c.size()) return GC_ERR_ARG;
    if (index >= 0) ws->pw[layer] = c[index];
  } else {
    const std::vector<FwdPlan> c = enum_fwd(R, kind ? Cout : Cin, kind ? Cin : Cout, ws->sm_count, nullptr);
    if (count) *count = (int)c.size();
    if (index >= (int)c.size()) return GC_ERR_ARG;
    if (index >= 0) (kind ? ws->pb[layer] : ws->pf[layer]) = c[index];
  }
  return GC_OK;
}

extern "C" int gc_ws_adam(gc_ws *ws, float lr, float beta1, float beta2, float eps, int step) {
  if (!ws || step < 1 || !(lr >= 0.0f)) return GC_ERR_ARG;
  const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
  ws_launch(ws, k_adam, dim3(512, WS_NL), 256, 0, ws->params, ws->grads, ws->adam_m, ws->adam_v, ws_pack_desc(ws), lr,
                                                  beta1, beta2, eps, bc1, bc2);
  WS_CUDA(ws, cudaGetLastError());
  return GC_OK;
}

// ------------------------------------------------------------------------------
// engine hook: history, input features, applying the prediction
// ------------------------------------------------------------------------------
// Initial guess of step n from the previous potentials:
//   plain        phi(n-1)                                   (the reference's warm start)
//   extrapolate  phi(n-1) + d(n-1),  d(k) = phi(k) - phi(k-1) at full resolution
//   learned      the extrapolation + s * trilinear(y): the network predicts the
//                next second difference dd(n) = d(n) - d(n-1) on the (G/2)^3 grid
//                in units of s = rms(dd_c(n-1)); a zero output is the extrapolation.
// The coarse grid has R = G/2 cells per axis; cell (I,J,K) is the mean of the
// fine nodes (2I..2I+1, 2J.., 2K..), centred at fine coordinate 2I + 0.5.
// Coarse history per context: phi_c(n-1), d_c(n-1), dd_c(n-1). Features of step
// n (f16 [4][R^3]): log(1 + rho_c / mean rho_c), phi_c / rms, d_c / rms(d_c),
// dd_c / rms(dd_c); training target dd_c(n) / rms(dd_c(n-1)).
__global__ void __launch_bounds__(64) k_ws_coarsen(const float *__restrict__ f, int G, float *__restrict__ out) {
  gc_after();
  const int R = G >> 1;
  const int K = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y, I = blockIdx.z;
  if (K >= R) return;
  float s = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += __ldg(f + child_index(G, I, J, K, c));
  out[((size_t)I * R + J) * R + K] = 0.125f * s;
}

// per-block sums: rho_c, phi_c^2, d_c^2, dd_c^2
__global__ void __launch_bounds__(256) k_ws_stats(const float *__restrict__ rho, const float *__restrict__ phi,
                                                  const float *__restrict__ dlt, const float *__restrict__ ddl,
                                                  size_t n, float *__restrict__ part) {
  gc_after();
  __shared__ float red[4][8];
  float a = 0.0f, b = 0.0f, c = 0.0f, e = 0.0f;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    a += rho[v];
    b += phi[v] * phi[v];
    c += dlt[v] * dlt[v];
    e += ddl[v] * ddl[v];
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { red[0][w] = a; red[1][w] = b; red[2][w] = c; red[3][w] = e; }
  __syncthreads();
  if (threadIdx.x < 4) {
    float s = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[threadIdx.x][i];
    part[4 * blockIdx.x + threadIdx.x] = s;
  }
}

// scal: [0] mean rho_c, [1] rms phi_c, [2] rms d_c, [3] d usable, [4] rms dd_c, [5] dd usable
// One block of 256 threads; fixed strided split and tree over the partials.
__global__ void __launch_bounds__(256) k_ws_scales(const float *__restrict__ part, int nb, size_t n, int hist,
                                                   float *__restrict__ scal) {
  gc_after();
  __shared__ double red[4][256];
  const int t = threadIdx.x;
  double ta = 0.0, tb = 0.0, tc = 0.0, te = 0.0;
  for (int i = t; i < nb; i += 256) { ta += part[4 * i]; tb += part[4 * i + 1]; tc += part[4 * i + 2]; te += part[4 * i + 3]; }
  red[0][t] = ta; red[1][t] = tb; red[2][t] = tc; red[3][t] = te;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
#pragma unroll
      for (int k = 0; k < 4; ++k) red[k][t] += red[k][t + w];
    }
    __syncthreads();
  }
  if (t != 0) return;
  const double a = red[0][0], b = red[1][0], c = red[2][0], e = red[3][0];
  const double mr = a / (double)n, rp = sqrt(b / (double)n), rd = sqrt(c / (double)n), rdd = sqrt(e / (double)n);
  const double tiny = 1e-30 * (rp > 0.0 ? rp : 1.0);
  scal[0] = mr > 0.0 ? (float)mr : 1.0f;
  scal[1] = (hist >= 1 && rp > 0.0) ? (float)rp : 1.0f;
  const bool dok = hist >= 2 && rd > tiny;
  scal[2] = dok ? (float)rd : 1.0f;
  scal[3] = dok ? 1.0f : 0.0f;
  const bool ddok = hist >= 3 && rdd > tiny;
  scal[4] = ddok ? (float)rdd : 1.0f;
  scal[5] = ddok ? 1.0f : 0.0f;
}

__global__ void __launch_bounds__(256) k_ws_features(const float *__restrict__ rho, const float *__restrict__ phi,
                                                     const float *__restrict__ dlt, const float *__restrict__ ddl,
                                                     const float *__restrict__ scal, int hist, size_t n,
                                                     __half *__restrict__ feat, __half *__restrict__ rec) {
  gc_after();
  const float ir = 1.0f / scal[0], ip = 1.0f / scal[1], id = 1.0f / scal[2], idd = 1.0f / scal[4];
  const bool has_p = hist >= 1, has_d = scal[3] != 0.0f, has_dd = scal[5] != 0.0f;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const __half a = __float2half_rn(log1pf(fmaxf(rho[v] * ir, 0.0f)));
    const __half b = __float2half_rn(has_p ? phi[v] * ip : 0.0f);
    const __half c = __float2half_rn(has_d ? dlt[v] * id : 0.0f);
    const __half e = __float2half_rn(has_dd ? ddl[v] * idd : 0.0f);
    feat[v] = a; feat[n + v] = b; feat[2 * n + v] = c; feat[3 * n + v] = e;
    if (rec) { rec[v] = a; rec[n + v] = b; rec[2 * n + v] = c; rec[3 * n + v] = e; }
  }
}

// Initial guess on every fine node: prev holds phi(n-2) on entry and phi(n-1)
// on exit; hi/lo (phi(n-1) on entry) get + d(n-1) when use_d (extrapolating,
// with two solves in the history) and + s * trilinear(yc) when yc is given.
__global__ void __launch_bounds__(128) k_ws_apply(const float *__restrict__ yc, const float *__restrict__ scal,
                                                  int use_d, int G, float *__restrict__ hi, float *__restrict__ lo,
                                                  float *__restrict__ prev) {
  gc_after();
  const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
  if (k >= G) return;
  // the face nodes are the multipole faces' (computed beside this pass)
  if (i == 0 || j == 0 || k == 0 || i == G - 1 || j == G - 1 || k == G - 1) return;
  const int R = G >> 1;
  const size_t v = ((size_t)i * G + j) * G + k;
  const float h = hi[v], l = lo[v];
  float corr = 0.0f;
  if (use_d) corr = __fsub_rn(h, prev[v]);
  if (yc && scal[5] != 0.0f) {
    int i0[3];
    float f[3];
    const int ii[3] = {i, j, k};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float c = 0.5f * (float)ii[a] - 0.25f;
      int b = (int)floorf(c);
      b = b < 0 ? 0 : (b > R - 2 ? R - 2 : b);
      i0[a] = b;
      f[a] = fminf(fmaxf(c - (float)b, 0.0f), 1.0f);
    }
    float acc = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int dx = c >> 2, dy = (c >> 1) & 1, dz = c & 1;
      const float w = (dx ? f[0] : 1.0f - f[0]) * (dy ? f[1] : 1.0f - f[1]) * (dz ? f[2] : 1.0f - f[2]);
      acc += w * __ldg(yc + ((size_t)(i0[0] + dx) * R + (i0[1] + dy)) * R + (i0[2] + dz));
    }
    corr += scal[4] * acc;
  }
  prev[v] = h;
  if (corr != 0.0f) {
    float sh, eh;
    df_two_sum(h, corr, sh, eh);
    float h2, l2;
    df_fast_two_sum(sh, __fadd_rn(l, eh), h2, l2);
    hi[v] = h2;
    lo[v] = l2;
  }
}

// after the solve: new phi_c, its first and second differences, the training
// target, history update
__global__ void __launch_bounds__(64) k_ws_post(const float *__restrict__ hi, int G, float *__restrict__ phi,
                                                float *__restrict__ dlt, float *__restrict__ ddl,
                                                const float *__restrict__ scal, int hist, __half *__restrict__ rec) {
  gc_after();
  const int R = G >> 1;
  const int K = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y, I = blockIdx.z;
  if (K >= R) return;
  const size_t R3 = (size_t)R * R * R;
  const size_t v = ((size_t)I * R + J) * R + K;
  const float idd = 1.0f / scal[4];
  const bool has_dd = scal[5] != 0.0f;
  float s = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += __ldg(hi + child_index(G, I, J, K, c));
  const float nw = 0.125f * s;
  const float d = hist >= 1 ? nw - phi[v] : 0.0f;
  const float dd = hist >= 2 ? d - dlt[v] : 0.0f;
  if (rec) rec[4 * R3 + v] = __float2half_rn(has_dd ? dd * idd : 0.0f);
  phi[v] = nw;
  dlt[v] = d;
  ddl[v] = dd;
}

static int ws_hook_buffers(gc_ctx *ctx) {
  const int R = ctx->G / 2;
  const size_t R3 = (size_t)R * R * R, G3 = (size_t)ctx->G * ctx->G * ctx->G;
  const size_t need = 5 * R3 + 2 * R3 + 16 + 4 * 1024 + G3;
  if (ctx->ws_buf && ctx->ws_buf_cap >= need) return GC_OK;
  cudaFree(ctx->ws_buf);
  ctx->ws_buf = nullptr;
  GC_CUDA(ctx, cudaMalloc(&ctx->ws_buf, need * sizeof(float)));
  GC_CUDA(ctx, cudaMemsetAsync(ctx->ws_buf, 0, need * sizeof(float), ctx->stream));
  ctx->ws_buf_cap = need;
  return GC_OK;
}

struct WsViews {
  float *rho, *phi, *dlt, *ddl, *y, *scal, *part, *prev;
  __half *feat;
};
static WsViews ws_views(gc_ctx *ctx) {
  const int R = ctx->G / 2;
  const size_t R3 = (size_t)R * R * R;
  WsViews w;
  w.rho = ctx->ws_buf;
  w.phi = w.rho + R3;
  w.dlt = w.phi + R3;
  w.ddl = w.dlt + R3;
  w.y = w.ddl + R3;
  w.feat = reinterpret_cast<__half *>(w.y + R3);  // 4 R^3 halves
  w.scal = w.y + 3 * R3;
  w.part = w.scal + 16;
  w.prev = w.part + 4 * 1024;
  return w;
}

int gc_ws_pre_solve(gc_ctx *ctx, int warm, int mode) {
  ctx->ws_skip = 0;
  if (!ctx->ws_track && !ctx->ws_record) return GC_OK;
  if (ctx->G % 2) return GC_OK;
  // a PRIME after a CLOSE solves at the positions of the last solve again: it
  // neither uses nor extends the history
  if (mode == GC_STEP_PRIME && ctx->ws_hist > 0 && warm) {
    ctx->ws_skip = 1;
    return GC_OK;
  }
  if (!warm) ctx->ws_hist = 0;  // a cold solve restarts the history
  int s;
  if ((s = ws_hook_buffers(ctx))) return s;
  const WsViews w = ws_views(ctx);
  const int R = ctx->G / 2;
  const size_t R3 = (size_t)R * R * R;
  unsigned nb = (unsigned)std::min<size_t>((R3 + 255) / 256, 1024);
  // the coarse history and the network features: for the learned guess, for
  // recording, or when tracking was asked for (the extrapolation needs neither)
  const bool coarse = ctx->ws_coarse || ctx->ws_record;
  if (coarse) {
  gc_launch_after(ctx, GK_WARMSTART, k_ws_coarsen, dim3((R + 63) / 64, R, R), dim3(64), 0, (const float *)ctx->b0, ctx->G,
            w.rho);
  gc_launch_after(ctx, GK_WARMSTART, k_ws_stats, dim3(nb), dim3(256), 0, (const float *)w.rho, (const float *)w.phi,
            (const float *)w.dlt, (const float *)w.ddl, R3, w.part);
  gc_launch_after(ctx, GK_WARMSTART, k_ws_scales, dim3(1), dim3(256), 0, (const float *)w.part, (int)nb, R3, ctx->ws_hist,
            w.scal);
  gc_launch_after(ctx, GK_WARMSTART, k_ws_features, dim3(nb), dim3(256), 0, (const float *)w.rho, (const float *)w.phi,
            (const float *)w.dlt, (const float *)w.ddl, (const float *)w.scal, ctx->ws_hist, R3, w.feat,
            (__half *)ctx->ws_record);
  GC_LAUNCH_CHECK(ctx, "warm-start features");
  }
  if (!warm || ctx->ws_hist < 1) return GC_OK;
  const float *yc = nullptr;
  if (ctx->ws_mode == GC_WS_LEARNED && ctx->ws_hist >= 3) {
    gc_ws *ws = ctx->ws;
    if (!ws || ws->R != R) {
      gc_set_error(ctx, "learned warm start needs a network with R = G/2 = %d", R);
      return GC_ERR_STATE;
    }
    ws->stream = ctx->stream;
    // the network's convolutions are timed as one warm-start interval (they
    // launch on the network object, not through the context's launcher)
    const int slot = ctx->prof.enabled && !ctx->capturing ? gc_prof_slot(ctx, GK_WARMSTART) : -1;
    if (slot >= 0) cudaEventRecord(ctx->prof.ev[2 * slot], ctx->stream);
    if ((s = gc_ws_forward(ws, w.feat, w.y))) {
      gc_set_error(ctx, "warm-start network: %s", ws->err);
      return s;
    }
    if (slot >= 0) cudaEventRecord(ctx->prof.ev[2 * slot + 1], ctx->stream);
    ctx->prof.launches[GK_WARMSTART] += 18;
    yc = w.y;
  }
  const int use_d = ctx->ws_mode != GC_WS_PLAIN && ctx->ws_hist >= 2;
  gc_launch_after(ctx, GK_WARMSTART, k_ws_apply, dim3((ctx->G + 127) / 128, ctx->G, ctx->G), dim3(128), 0, yc,
            (const float *)w.scal, use_d, ctx->G, ctx->hi, ctx->lo, w.prev);
  GC_LAUNCH_CHECK(ctx, "warm-start apply");
  return GC_OK;
}

int gc_ws_post_solve(gc_ctx *ctx) {
  if (!ctx->ws_track && !ctx->ws_record) return GC_OK;
  if (ctx->G % 2 || ctx->ws_skip) return GC_OK;
  if (!ctx->ws_coarse && !ctx->ws_record) {
    ctx->ws_hist = ctx->ws_hist < 3 ? ctx->ws_hist + 1 : 3;
    return GC_OK;
  }
  const WsViews w = ws_views(ctx);
  const int R = ctx->G / 2;
  gc_launch_after(ctx, GK_WARMSTART, k_ws_post, dim3((R + 63) / 64, R, R), dim3(64), 0, (const float *)ctx->hi, ctx->G,
            w.phi, w.dlt, w.ddl, (const float *)w.scal, ctx->ws_hist, (__half *)ctx->ws_record);
  GC_LAUNCH_CHECK(ctx, "warm-start history");
  ctx->ws_hist = ctx->ws_hist < 3 ? ctx->ws_hist + 1 : 3;
  ctx->ws_record = nullptr;
  return GC_OK;
}

extern "C" int gc_pm_set_warmstart(gc_ctx *ctx, gc_ws *ws, int mode, int track) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, mode == GC_WS_PLAIN || mode == GC_WS_LEARNED || mode == GC_WS_EXTRAPOLATE,
             "gc_pm_set_warmstart: bad mode %d", mode);
  GC_REQUIRE(ctx, mode != GC_WS_LEARNED || ws, "gc_pm_set_warmstart: learned mode needs a network");
  GC_REQUIRE(ctx, ctx->G % 2 == 0 || (mode == GC_WS_PLAIN && !track),
             "gc_pm_set_warmstart: the coarse history needs an even grid size");
  GC_REQUIRE(ctx, !ws || ws->R == ctx->G / 2, "gc_pm_set_warmstart: network R=%d, grid needs R=%d", ws ? ws->R : 0,
             ctx->G / 2);
  const int tr = (track || mode != GC_WS_PLAIN) ? 1 : 0;
  const int coarse = (track || mode == GC_WS_LEARNED) ? 1 : 0;
  // the history restarts when what it holds changes
  if ((tr && !ctx->ws_track) || (coarse && !ctx->ws_coarse) || mode != ctx->ws_mode) ctx->ws_hist = 0;
  ctx->ws = ws;
  ctx->ws_mode = mode;
  ctx->ws_track = tr;
  ctx->ws_coarse = coarse;
  return GC_OK;
}

extern "C" int gc_pm_record_sample(gc_ctx *ctx, void *out) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, ctx->G % 2 == 0, "gc_pm_record_sample: the coarse grid needs an even grid size");
  GC_REQUIRE(ctx, ctx->ws_coarse, "gc_pm_record_sample: set the warm start with track = 1 first");
  ctx->ws_record = out;
  return GC_OK;
}
