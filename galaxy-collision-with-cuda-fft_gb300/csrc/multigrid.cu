// Open-boundary multigrid Poisson solver for laplacian(phi) = 4 pi G rho.
//
// The discrete problem is the reference's (src/galaxy_collision/solver/multigrid.py):
// 7-point Laplacian on the finest node grid, Dirichlet faces from the monopole +
// quadrupole of rho about its centre of mass (multigrid.py:261-295), residual
// ||rhs - L phi||_2 against ||rhs||_2 (multigrid.py:473-485). Only the finest
// level defines the answer (multigrid.py:8-15), so the hierarchy is free:
//
//  * Level l has its far face at p_l = (G-1)/2^l (in level-l node units). Coarse
//    node J <-> fine node 2J. When p_l is fractional the last interior node J_l
//    uses a Shortley-Weller stencil with the Dirichlet face at distance
//    delta = p_l - J_l, and the transfer operators interpolate to that face. The
//    reference instead cuts the coarse grid at fine node 2(n/2)-2 and converges
//    at ~0.6-0.7 per V-cycle; this hierarchy converges at ~0.1.
//  * The finest level relaxes the potential itself as a double-float pair
//    (hi + lo, both FP32): each red-black Gauss-Seidel update is computed from
//    an accurate local residual (exact neighbour differences summed with
//    error-free transforms), so the residual can be driven below the FP32 floor
//    (~6e-5 relative in the reference) with FP32 arithmetic only. This is the
//    defect-correction loop: coarse levels relax FP32 corrections of that
//    residual, the coarsest level is solved in FP64.
//  * All arrays are C-order [i][j][k], k fastest. Right-hand sides are stored
//    h^2-scaled (b = h^2 * rhs) so stencils need no division by h^2.
#include "common.cuh"

#include <math.h>
#include <stdlib.h>

#define RB_TX 32
#define RB_TY 8

// ------------------------------------------------------------------------------
// level geometry
// ------------------------------------------------------------------------------
int gc_mg_build_levels(gc_ctx *ctx) {
  const int G = ctx->G;
  ctx->nlev = 0;
  ctx->tail = 0;
  if (G - 2 < 1) return GC_OK;  // no interior node: the solve is the boundary alone
  LevelGeom g0;
  g0.n = G;
  g0.J = G - 2;
  g0.a = 1.0f;
  g0.dB = 2.0f;
  g0.p = (float)(G - 1);
  ctx->lev[0] = g0;
  int nl = 1;
  for (int l = 1; l < GC_MAX_LEVELS; ++l) {
    double p = (double)(G - 1) / (double)(1 << l);
    int J = (int)ceil(p) - 1;
    if (J < 1) break;
    double delta = p - (double)J;
    LevelGeom g;
    g.n = J + 2;
    g.J = J;
    g.a = (float)(2.0 / (1.0 + delta));
    g.dB = (float)(2.0 / delta);
    g.p = (float)p;
    ctx->lev[nl++] = g;
  }
  ctx->nlev = nl;
  int tail = nl;
  for (int l = 1; l < nl; ++l) {
    if (ctx->lev[l].n <= GC_TAIL_MAX_N) {
      tail = l;
      break;
    }
  }
  ctx->tail = tail;
  return GC_OK;
}

static bool finest_blocks(const gc_ctx *ctx, const gc_mg_params *p);
static bool finest_planes(const gc_ctx *ctx, const gc_mg_params *p);

// (cleared on the context's own stream and waited for: the caller's stream may be under
// capture, and need not be ordered after the default one)
static int alloc_zero(gc_ctx *ctx, float **a, size_t n) {
  if (*a) return GC_OK;
  if (!ctx->cap) GC_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->cap, cudaStreamNonBlocking));
  float *p = nullptr;
  GC_CUDA(ctx, cudaMalloc(&p, n * sizeof(float)));
  cudaError_t e = cudaMemsetAsync(p, 0, n * sizeof(float), ctx->cap);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->cap);
  if (e != cudaSuccess) {
    cudaFree(p);
    GC_CUDA(ctx, e);
  }
  *a = p;
  return GC_OK;
}

// The finest level's correction and residual as the solve with these parameters keeps
// them (allocated on first use; faces stay zero): natural layout (in blocks, or
// GC_MG_NATURAL_LAYOUT) or colour-split, and the scratch of the paths that store the
// correction's residual.
static int mg_alloc_finest(gc_ctx *ctx, const gc_mg_params *p) {
  if (ctx->nlev == 0) return GC_OK;
  const size_t g3 = (size_t)ctx->G * ctx->G * ctx->G;
  const bool blocks = finest_blocks(ctx, p);
  int s;
  if (blocks || (p->flags & GC_MG_NATURAL_LAYOUT)) {
    if ((s = alloc_zero(ctx, &ctx->e0n, g3)) || (s = alloc_zero(ctx, &ctx->r0n, g3))) return s;
  } else {
    if ((s = alloc_zero(ctx, &ctx->e0s, 2 * ctx->half0)) || (s = alloc_zero(ctx, &ctx->r0s, 2 * ctx->half0))) return s;
  }
  return ctx->nlev > 1 && !blocks && !finest_planes(ctx, p) ? alloc_zero(ctx, &ctx->r0, g3) : GC_OK;
}

int gc_mg_alloc(gc_ctx *ctx) {
  const size_t G = ctx->G;
  const size_t g3 = G * G * G;
  ctx->H0 = (ctx->G + 1) / 2;
  ctx->half0 = G * G * (size_t)ctx->H0;
  GC_CUDA(ctx, cudaMalloc(&ctx->hi, g3 * sizeof(float)));
  GC_CUDA(ctx, cudaMalloc(&ctx->lo, g3 * sizeof(float)));
  GC_CUDA(ctx, cudaMalloc(&ctx->b0, g3 * sizeof(float)));
  GC_CUDA(ctx, cudaMemset(ctx->hi, 0, g3 * sizeof(float)));
  GC_CUDA(ctx, cudaMemset(ctx->lo, 0, g3 * sizeof(float)));
  GC_CUDA(ctx, cudaMemset(ctx->b0, 0, g3 * sizeof(float)));
  // the coarse levels' arrays in one block (each on a 256-byte boundary): e and b, the
  // black nodes of the way down (ed) above the tail, and a residual scratch
  size_t need = 0, rc_n = 0;
  auto take = [&](float **p, size_t n) {
    if (p) *p = ctx->coarse + need;
    need += (n + 63) & ~(size_t)63;
  };
  for (int pass = 0; pass < 2; ++pass) {
    need = 0;
    for (int l = 1; l < ctx->nlev; ++l) {
      const size_t n3 = (size_t)ctx->lev[l].n * ctx->lev[l].n * ctx->lev[l].n;
      take(pass ? &ctx->e[l] : nullptr, n3);
      take(pass ? &ctx->b[l] : nullptr, n3);
      if (l < ctx->tail) {
        take(pass ? &ctx->ed[l] : nullptr, n3);
        if (n3 > rc_n) rc_n = n3;
      }
    }
    if (rc_n) take(pass ? &ctx->rc : nullptr, rc_n);
    if (!pass && need) {
      GC_CUDA(ctx, cudaMalloc(&ctx->coarse, need * sizeof(float)));
      GC_CUDA(ctx, cudaMemset(ctx->coarse, 0, need * sizeof(float)));
    }
  }
  // the finest level's arrays of the default parameters' path
  gc_mg_params p;
  gc_mg_default_params(&p);
  return mg_alloc_finest(ctx, &p);
}

void gc_mg_free(gc_ctx *ctx) {
  cudaFree(ctx->hi); cudaFree(ctx->lo);
  cudaFree(ctx->b0); cudaFree(ctx->r0);
  cudaFree(ctx->e0s); cudaFree(ctx->r0s); cudaFree(ctx->e0n); cudaFree(ctx->r0n);
  for (int l = 1; l < GC_MAX_LEVELS; ++l) ctx->e[l] = ctx->b[l] = ctx->ed[l] = nullptr;
  cudaFree(ctx->coarse);
  ctx->coarse = nullptr;
  ctx->hi = ctx->lo = ctx->b0 = ctx->r0 = ctx->rc = nullptr;
  ctx->e0s = ctx->r0s = ctx->e0n = ctx->r0n = nullptr;
}

// ------------------------------------------------------------------------------
// reductions: per-block partials written in a fixed order, then one block sums them
// ------------------------------------------------------------------------------
// Sum nparts rows of nv partials into dst[0..nv), deterministically (a fixed
// association for given nparts and nv). FP64 runs at a small fraction of the
// f32 rate on this GPU (16 clk an SM for a warp's addition), so the adds are spread:
// warp w of one block sums value w (lanes take rows lane, lane + 32, ...); a single
// value takes one block of 256 threads, and a long list is first cut into
// GC_FIN_CHUNKS contiguous chunks summed by as many blocks.
#define GC_FIN_NV 32
#define GC_FIN_CHUNKS 128
__global__ void __launch_bounds__(1024)
    k_fin_warps(const double *__restrict__ parts, int nparts, int nv, double *__restrict__ dst) {
  const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
  if (v >= nv) return;
  double s = 0.0;
#pragma unroll 8
  for (int i = lane; i < nparts; i += 32) s += parts[(size_t)i * nv + v];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) dst[v] = s;
}

// The stopping rule of a device-decided solve (the host loop of gc_mg_run), evaluated
// where the residual's norm is finished (on = 0: the sum alone): the cycle count lives in
// dsmall[GC_S_CYCLES]; the loop continues while fewer than max_c cycles ran and not (at
// least max(1, min_c) cycles ran and ||r|| < tol ||b|| with ||b|| > 0). The verdict goes
// to the conditional node that repeats the V-cycle body, the converged flag to
// dsmall[GC_S_CONVERGED].
struct MgDecide {
  cudaGraphConditionalHandle h;
  double tol;
  int on, min_c, max_c, first, count;
};

__device__ __forceinline__ void mg_decide(const MgDecide &d, double *__restrict__ small, double r2) {
  const int c = d.first ? 0 : (int)small[GC_S_CYCLES] + 1;
  const double b2 = small[GC_S_BNORM2];
  small[GC_S_CYCLES] = (double)c;
  const int minc = d.min_c > 1 ? d.min_c : 1;
  const bool conv = c >= minc && b2 > 0.0 && sqrt(r2) < d.tol * sqrt(b2);
  small[GC_S_CONVERGED] = conv ? 1.0 : 0.0;
  const bool more = !conv && c < d.max_c;
  if (!more && d.count) {  // the solve ends here: count it
    small[GC_S_SOLVES] += 1.0;
    small[GC_S_CYC_TOTAL] += (double)c;
    const double rel2 = b2 > 0.0 ? r2 / b2 : 0.0;
    if (rel2 > small[GC_S_MAXREL2]) small[GC_S_MAXREL2] = rel2;
  }
  cudaGraphSetConditional(d.h, more ? 1u : 0u);
}

// One value: 256 threads with up to 16 loads in flight each, then the stopping rule in
// the same launch. Latency is all there is: one warp over 2048 partials took 5.3 us and
// the rule another launch of 2.5 (64^3, one V-cycle of 90 us); together here 4.5 (97^3:
// 9.2 + 2.7 -> 4.9). Loading the rule's operands ahead and sparing its square roots
// changed nothing.
__global__ void __launch_bounds__(256)
    k_fin_one(const double *__restrict__ parts, int nparts, double *__restrict__ dst, double *__restrict__ small,
              const __grid_constant__ MgDecide d) {
  gc_after();
  __shared__ double sh[8];
  const int tid = threadIdx.x;
  double x[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i0 = tid; i0 < nparts; i0 += 4096) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = i0 + 256 * u < nparts ? __ldcg(parts + i0 + 256 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < 16; ++u)
      if (256 * u < nparts) x[u & 3] += v[u];
  }
  double s = (x[0] + x[1]) + (x[2] + x[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) sh[tid >> 5] = s;
  __syncthreads();
  if (tid != 0) return;
  const double r = ((sh[0] + sh[1]) + (sh[2] + sh[3])) + ((sh[4] + sh[5]) + (sh[6] + sh[7]));
  *dst = r;
  if (d.on) mg_decide(d, small, r);
}

__global__ void __launch_bounds__(256)
    k_fin_chunks(const double *__restrict__ parts, int nparts, double *__restrict__ out) {
  gc_after();
  __shared__ double sh[8];
  const int per = (nparts + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per, i1 = min(nparts, i0 + per);
  double s = 0.0;
  for (int i = i0 + (int)threadIdx.x; i < i1; i += 256) s += parts[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0.0;
    for (int w = 0; w < 8; ++w) x += sh[w];
    out[blockIdx.x] = x;
  }
}

// ------------------------------------------------------------------------------
// finest level: double-float red-black Gauss-Seidel, residual, prolongation
// ------------------------------------------------------------------------------
// Accurate residual r = b - L_h2(hi + lo) at an interior node (h^2 units) from
// the pair at the node (hc, lc) and at its six neighbours in the order
// i+1, i-1, j+1, j-1, k+1, k-1: exact neighbour differences summed with
// error-free transforms, the lo parts' Laplacian added in f32.
__device__ __forceinline__ float df_residual_v(float hc, float lc, const float (&h)[6], const float (&l)[6],
                                               float bc) {
  const float d0 = __fsub_rn(h[0], hc);
  const float d1 = __fsub_rn(h[1], hc);
  const float d2 = __fsub_rn(h[2], hc);
  const float d3 = __fsub_rn(h[3], hc);
  const float d4 = __fsub_rn(h[4], hc);
  const float d5 = __fsub_rn(h[5], hc);
  float s, e, t;
  df_two_sum(d0, d1, s, e);
  df_two_sum(s, d2, s, t); e = __fadd_rn(e, t);
  df_two_sum(s, d3, s, t); e = __fadd_rn(e, t);
  df_two_sum(s, d4, s, t); e = __fadd_rn(e, t);
  df_two_sum(s, d5, s, t); e = __fadd_rn(e, t);
  const float ln = ((((l[0] + l[1]) + l[2]) + l[3]) + l[4]) + l[5];
  const float ll = __fsub_rn(ln, __fmul_rn(6.0f, lc));
  float r1, r1e;
  df_two_sum(bc, -s, r1, r1e);
  return __fadd_rn(r1, __fsub_rn(r1e, __fadd_rn(e, ll)));
}

__device__ __forceinline__ float df_residual(const float *__restrict__ hi, const float *__restrict__ lo,
                                             float bc, size_t c, size_t sj, size_t si, float &hc_out,
                                             float &lc_out) {
  const float h[6] = {hi[c + si], hi[c - si], hi[c + sj], hi[c - sj], hi[c + 1], hi[c - 1]};
  const float l[6] = {lo[c + si], lo[c - si], lo[c + sj], lo[c - sj], lo[c + 1], lo[c - 1]};
  hc_out = hi[c];
  lc_out = lo[c];
  return df_residual_v(hc_out, lc_out, h, l, bc);
}

// FP64 verification residual: phi = (double)hi + (double)lo, or hi alone when lo is NULL.
__global__ void __launch_bounds__(256)
    k_resid64(const float *__restrict__ hi, const float *__restrict__ lo, const float *__restrict__ b,
              double *__restrict__ parts, int G) {
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  double acc[1] = {0.0};
  if (k <= G - 2 && j <= G - 2) {
    const size_t sj = (size_t)G, si = (size_t)G * G;
    const size_t c = (size_t)i * si + (size_t)j * sj + k;
    auto P = [&](size_t q) { return lo ? (double)hi[q] + (double)lo[q] : (double)hi[q]; };
    const double pc = P(c);
    const double lap = (P(c + si) - pc) + (P(c - si) - pc) + (P(c + sj) - pc) + (P(c - sj) - pc) +
                       (P(c + 1) - pc) + (P(c - 1) - pc);
    const double rv = (double)b[c] - lap;
    acc[0] = rv * rv;
  }
  const size_t bid = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  block_partials<1>(acc, parts + bid);
}

// ------------------------------------------------------------------------------
// coarse levels (FP32 corrections, Shortley-Weller far faces)
// ------------------------------------------------------------------------------
struct AxisTerm {
  float s;  // weighted neighbour sum along the axis
  float d;  // diagonal contribution
};

__device__ __forceinline__ AxisTerm sw_axis(const float *__restrict__ e, size_t c, size_t stride, int idx,
                                            const LevelGeom &g) {
  AxisTerm t;
  if (idx == g.J) {
    t.s = g.a * e[c - stride];
    t.d = g.dB;
  } else {
    t.s = e[c + stride] + e[c - stride];
    t.d = 2.0f;
  }
  return t;
}

__device__ __forceinline__ void sw_stencil(const float *__restrict__ e, size_t c, int i, int j, int k,
                                           const LevelGeom &g, float &sum, float &diag) {
  const size_t n = (size_t)g.n;
  const AxisTerm ax = sw_axis(e, c, n * n, i, g);
  const AxisTerm ay = sw_axis(e, c, n, j, g);
  const AxisTerm az = sw_axis(e, c, 1, k, g);
  sum = (ax.s + ay.s) + az.s;
  diag = (ax.d + ay.d) + az.d;
}

// Gauss-Seidel value (sum - b) / diag. The common diagonal 6 (every node off a
// Shortley-Weller face) multiplies by the correctly rounded 1/6 instead of
// dividing; every smoother of every level and layout uses this one rule, with
// explicitly rounded products so that no contraction can differ between them.
#define GC_SIXTH 0.16666667f
__device__ __forceinline__ float gs_value(float sum, float b, float diag) {
  return diag == 6.0f ? __fmul_rn(sum - b, GC_SIXTH) : (sum - b) / diag;
}

__global__ void __launch_bounds__(RB_TX *RB_TY)
    k_smooth(float *__restrict__ e, const float *__restrict__ b, LevelGeom g, int color) {
  const int kk = blockIdx.x * RB_TX + threadIdx.x;
  const int j = blockIdx.y * RB_TY + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (j > g.J) return;
  const int k = 2 * kk + ((color + i + j) & 1);
  if (k < 1 || k > g.J) return;
  const size_t n = g.n;
  const size_t c = ((size_t)i * n + j) * n + k;
  float sum, diag;
  sw_stencil(e, c, i, j, k, g, sum, diag);
  e[c] = gs_value(sum, b[c], diag);
}

__global__ void __launch_bounds__(256)
    k_resid(const float *__restrict__ e, const float *__restrict__ b, float *__restrict__ r, LevelGeom g) {
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (k > g.J || j > g.J) return;
  const size_t n = g.n;
  const size_t c = ((size_t)i * n + j) * n + k;
  float sum, diag;
  sw_stencil(e, c, i, j, k, g, sum, diag);
  r[c] = b[c] - (sum - diag * e[c]);
}

// 1-D restriction weight of fine node 2J'+o into coarse node J' (transpose of the prolongation / 2).
__device__ __forceinline__ float restrict_w(int Jc, int o, const LevelGeom &f, const LevelGeom &cg) {
  const int i = 2 * Jc + o;
  if (i < 1 || i > f.J) return 0.0f;
  if (o == 0) return 0.5f;
  if (o < 0) return 0.25f;
  if (Jc < cg.J) return 0.25f;
  return 0.5f * (f.p - (float)i) / (f.p - (float)(2 * Jc));
}

// b_c = 4 * R(r_f) at coarse node (I, Jj, K): full weighting (transpose of
// trilinear prolongation), summed separably: the three k terms of each of the
// nine (i, j) fine rows, then the rows' j weights, then the i weights. Terms of
// weight zero (fine nodes on a face) are not read.
__device__ __forceinline__ void restrict_node(const float *__restrict__ rf, const LevelGeom &f,
                                              float *__restrict__ bc, const LevelGeom &cg, int I, int Jj, int K) {
  float wi[3], wj[3], wk[3];
#pragma unroll
  for (int o = -1; o <= 1; ++o) {
    wi[o + 1] = restrict_w(I, o, f, cg);
    wj[o + 1] = restrict_w(Jj, o, f, cg);
    wk[o + 1] = restrict_w(K, o, f, cg);
  }
  const size_t n = f.n;
  const float *base = rf + ((size_t)(2 * I - 1) * n + (size_t)(2 * Jj - 1)) * n + (size_t)(2 * K - 1);
  float acc = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (wi[a] == 0.0f) continue;
    float ta = 0.0f;
#pragma unroll
    for (int bb = 0; bb < 3; ++bb) {
      if (wj[bb] == 0.0f) continue;
      const float *row = base + ((size_t)a * n + (size_t)bb) * n;
      float sab = wk[1] * row[1];
      if (wk[0] != 0.0f) sab += wk[0] * row[0];
      if (wk[2] != 0.0f) sab += wk[2] * row[2];
      ta += wj[bb] * sab;
    }
    acc += wi[a] * ta;
  }
  const size_t m = cg.n;
  bc[((size_t)I * m + Jj) * m + K] = 4.0f * acc;
}

__global__ void __launch_bounds__(256)
    k_restrict(const float *__restrict__ rf, LevelGeom f, float *__restrict__ bc, LevelGeom cg) {
  gc_after();
  const int K = blockIdx.x * 32 + threadIdx.x + 1;
  const int Jj = blockIdx.y * 8 + threadIdx.y + 1;
  const int I = blockIdx.z + 1;
  if (K > cg.J || Jj > cg.J) return;
  restrict_node(rf, f, bc, cg, I, Jj, K);
}

// 1-D prolongation weights of fine node i from the coarse level.
__device__ __forceinline__ int prolong_w(int i, const LevelGeom &f, const LevelGeom &cg, int &c0, float &w0,
                                         float &w1) {
  c0 = i >> 1;
  if ((i & 1) == 0) {
    w0 = 1.0f;
    w1 = 0.0f;
    return 1;
  }
  if (c0 + 1 <= cg.J) {
    w0 = 0.5f;
    w1 = 0.5f;
    return 2;
  }
  w0 = (f.p - (float)i) / (f.p - (float)(2 * c0));
  w1 = 0.0f;
  return 1;
}

// P(e_c) at fine node (i, j, k); coarse node (I, J, K) at ec[I si + J sj + K].
__device__ __forceinline__ float prolong_at(const float *__restrict__ ec, int si, int sj, int i, int j, int k,
                                            const LevelGeom &f, const LevelGeom &cg) {
  int ci, cj, ck;
  float wi0, wi1, wj0, wj1, wk0, wk1;
  const int ni = prolong_w(i, f, cg, ci, wi0, wi1);
  const int nj = prolong_w(j, f, cg, cj, wj0, wj1);
  const int nk = prolong_w(k, f, cg, ck, wk0, wk1);
  float val = 0.0f;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const float wa = a ? wi1 : wi0;
#pragma unroll
    for (int bb = 0; bb < 2; ++bb) {
      if (a >= ni || bb >= nj) continue;
      const float wb = bb ? wj1 : wj0;
      const float *row = ec + (ci + a) * si + (cj + bb) * sj + ck;
      const float wab = wa * wb;
      val += wab * wk0 * row[0];
      if (nk == 2) val += wab * wk1 * row[1];
    }
  }
  return val;
}

__device__ __forceinline__ float prolong_value(const float *__restrict__ ec, int i, int j, int k,
                                               const LevelGeom &f, const LevelGeom &cg) {
  return prolong_at(ec, cg.n * cg.n, cg.n, i, j, k, f, cg);  // coarse levels have < 2^31 nodes
}

__global__ void __launch_bounds__(256)
    k_prolong(const float *__restrict__ ec, LevelGeom cg, float *__restrict__ ef, LevelGeom f) {
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (k > f.J || j > f.J) return;
  const size_t n = f.n;
  ef[((size_t)i * n + j) * n + k] += prolong_value(ec, i, j, k, f, cg);
}

// ------------------------------------------------------------------------------
// finest level: defect correction with FP32 corrections in colour-split storage
// ------------------------------------------------------------------------------
// Each V-cycle solves L e = r for a correction e of the current potential
// (phi = hi + lo, double-float) with FP32 red-black Gauss-Seidel, then adds it:
// phi += e, and forms the new residual r = b - L phi accurately from the pair.
// The correction and the residual are stored colour-split: node (i,j,k) of
// colour c = (i+j+k)&1 lives in half c at s = (i*G + j)*H + (k>>1), H = (G+1)/2
// (the same-colour nodes of a row are every other k, so k>>1 is unique). A
// half-sweep of colour c then reads only the other colour's half and its own
// right-hand side and writes its own half: a Gauss-Seidel update does not use
// the node's old value. Neighbours of node s of colour c in the other half:
// i +- 1 at s +- G*H, j +- 1 at s +- H, k +- 1 at s + p and s + p - 1 with
// p = k & 1. Face nodes are never written and stay zero (homogeneous
// correction). The arithmetic is that of k_smooth / k_resid / k_prolong on the
// level-0 geometry in natural layout (GC_MG_NATURAL_LAYOUT runs those), term for
// term, so both layouts give identical potentials.
struct Split0 {
  int G, H;
  size_t half;  // nodes per colour half: G * G * H
};

__device__ __forceinline__ float split_nbr_sum(const float *__restrict__ o, size_t s, size_t GH, int H, int p) {
  const float ax = o[s + GH] + o[s - GH];
  const float ay = o[s + H] + o[s - H];
  const float az = o[s + p] + o[s + p - 1];
  return (ax + ay) + az;
}

// One half-sweep of colour `color` on the interior; FIRST: the correction
// starts at zero, so e = (0 - r)/6 and nothing is read but r.
template <bool FIRST>
__global__ void __launch_bounds__(256)
    k_rb0(float *__restrict__ e, const float *__restrict__ r, Split0 d, int color) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (kk >= d.H || j > d.G - 2) return;
  const int p = (color + i + j) & 1;
  const int k = 2 * kk + p;
  if (k < 1 || k > d.G - 2) return;
  const size_t s = ((size_t)i * d.G + j) * d.H + kk;
  float *own = e + (size_t)color * d.half;
  const float *oth = e + (size_t)(color ^ 1) * d.half;
  const float rv = r[(size_t)color * d.half + s];
  const float sum = FIRST ? 0.0f : split_nbr_sum(oth, s, (size_t)d.G * d.H, d.H, p);
  own[s] = __fmul_rn(sum - rv, GC_SIXTH);
}

// (h, l) += ev: double-float add (or a plain f32 add).
template <bool PLAIN>
__device__ __forceinline__ void phi_sum(float &h, float &l, float ev) {
  if (PLAIN) {
    h = __fadd_rn(h, ev);
  } else {
    float s1, e1;
    df_two_sum(h, ev, s1, e1);
    df_fast_two_sum(s1, __fadd_rn(l, e1), h, l);
  }
}

// phi += e at natural node c.
template <bool PLAIN>
__device__ __forceinline__ void phi_add(float *__restrict__ hi, float *__restrict__ lo, size_t c, float ev) {
  float h = hi[c], l = PLAIN ? 0.0f : lo[c];
  phi_sum<PLAIN>(h, l, ev);
  hi[c] = h;
  if (!PLAIN) lo[c] = l;
}

// The last half-sweep (black) fused with the update phi += e: thread kk of row
// (i,j) relaxes the black node 2kk + pb and adds the final corrections of that
// node and of the red node 2kk + (1 - pb) into the potential. The correction is
// dead afterwards, so the black value is not stored.
template <bool PLAIN>
__global__ void __launch_bounds__(256)
    k_rb0_last(const float *__restrict__ e, const float *__restrict__ r, float *__restrict__ hi,
               float *__restrict__ lo, Split0 d) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (kk >= d.H || j > d.G - 2) return;
  const int pb = (1 + i + j) & 1;
  const int kb = 2 * kk + pb, kr = 2 * kk + (pb ^ 1);
  const size_t s = ((size_t)i * d.G + j) * d.H + kk;
  const size_t row = ((size_t)i * d.G + j) * d.G;
  if (kb >= 1 && kb <= d.G - 2) {
    const float sum = split_nbr_sum(e, s, (size_t)d.G * d.H, d.H, pb);
    const float eb = __fmul_rn(sum - r[d.half + s], GC_SIXTH);
    phi_add<PLAIN>(hi, lo, row + kb, eb);
  }
  if (kr >= 1 && kr <= d.G - 2) phi_add<PLAIN>(hi, lo, row + kr, e[s]);
}

// phi += e at every interior node (natural-layout correction), the update of
// the natural-layout path and of cycles without post-smoothing.
template <bool PLAIN, bool SPLIT>
__global__ void __launch_bounds__(256)
    k_update0(const float *__restrict__ e, float *__restrict__ hi, float *__restrict__ lo, Split0 d) {
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (k > d.G - 2 || j > d.G - 2) return;
  const size_t c = ((size_t)i * d.G + j) * d.G + k;
  const float ev = SPLIT ? e[(size_t)((i + j + k) & 1) * d.half + ((size_t)i * d.G + j) * d.H + (k >> 1)] : e[c];
  phi_add<PLAIN>(hi, lo, c, ev);
}

// Plain FP32 residual b - L(hi) (the reference's left-to-right neighbour sum).
__device__ __forceinline__ float f32_residual(const float *__restrict__ hi, float bc, size_t c, size_t sj, size_t si) {
  const float s6 = ((((hi[c + si] + hi[c - si]) + hi[c + sj]) + hi[c - sj]) + hi[c + 1]) + hi[c - 1];
  return bc - (s6 - 6.0f * hi[c]);
}

// Residual r = b - L phi of the potential (double-float, or f32 when PLAIN) at
// every interior node, stored colour-split (SPLIT) or natural; block partials of
// sum r^2. With e_first (split only), the first half-sweep of the next cycle's
// pre-smoothing (red, from a zero correction) is written as well.
template <bool PLAIN, bool SPLIT>
__global__ void __launch_bounds__(256)
    k_resid0(const float *__restrict__ hi, const float *__restrict__ lo, const float *__restrict__ b,
             float *__restrict__ rout, float *__restrict__ e_first, double *__restrict__ parts, Split0 d) {
  gc_after();
  const int G = d.G;
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  float acc = 0.0f;
  if (k <= G - 2 && j <= G - 2) {
    const size_t sj = (size_t)G, si = (size_t)G * G;
    const size_t c = (size_t)i * si + (size_t)j * sj + k;
    float rv;
    if (PLAIN) {
      rv = f32_residual(hi, b[c], c, sj, si);
    } else {
      float hc, lc;
      rv = df_residual(hi, lo, b[c], c, sj, si, hc, lc);
    }
    if (SPLIT) {
      const int col = (i + j + k) & 1;
      const size_t s = ((size_t)i * G + j) * d.H + (k >> 1);
      rout[(size_t)col * d.half + s] = rv;
      if (e_first && col == 0) e_first[s] = __fmul_rn(0.0f - rv, GC_SIXTH);
    } else {
      rout[c] = rv;
    }
    acc = rv * rv;
  }
  const size_t bid = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  block_sum_f32(acc, parts + bid);
}

// Residual of the correction equation, r - L e (e, r colour-split), written in
// natural layout for the restriction: the arithmetic of k_resid on level 0.
__global__ void __launch_bounds__(256)
    k_resid0e(const float *__restrict__ e, const float *__restrict__ r, float *__restrict__ rc, Split0 d) {
  const int G = d.G;
  const int k = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (k > G - 2 || j > G - 2) return;
  const int col = (i + j + k) & 1;
  const size_t s = ((size_t)i * G + j) * d.H + (k >> 1);
  const float *own = e + (size_t)col * d.half;
  const float *oth = e + (size_t)(col ^ 1) * d.half;
  const float sum = split_nbr_sum(oth, s, (size_t)G * d.H, d.H, k & 1);
  const float diag = 6.0f;
  rc[((size_t)i * G + j) * G + k] = r[(size_t)col * d.half + s] - (sum - diag * own[s]);
}

// Add the level-1 correction into the colour-split level-0 correction: black
// nodes only when a red half-sweep follows (it overwrites the red half without
// reading it), both colours otherwise.
__global__ void __launch_bounds__(256)
    k_prolong0s(const float *__restrict__ ec, LevelGeom cg, float *__restrict__ e, LevelGeom f, Split0 d,
                int both) {
  const int kk = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (kk >= d.H || j > d.G - 2) return;
  const size_t s = ((size_t)i * d.G + j) * d.H + kk;
  for (int col = both ? 0 : 1; col < 2; ++col) {
    const int k = 2 * kk + ((col + i + j) & 1);
    if (k < 1 || k > d.G - 2) continue;
    e[(size_t)col * d.half + s] += prolong_value(ec, i, j, k, f, cg);
  }
}

// ---- the same finest-level kernels, vectorised (G % 4 == 0) --------------------
// With G a multiple of 4 the split row length H = G/2 is even, so slot pairs
// (2t, 2t+1) start on 8-byte boundaries, and natural rows of G nodes split into
// 16-byte quads. Each thread then handles two slots of one colour (half-sweeps,
// prolongation) or four consecutive nodes (residuals, update) with vector
// loads; the arithmetic of every node is that of the scalar kernels above.
__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st2(float *p, float a, float b) { *reinterpret_cast<float2 *>(p) = make_float2(a, b); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float f4get(const float4 &v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }
__device__ __forceinline__ void f4set(float4 &v, int q, float x) {
  if (q == 0) v.x = x; else if (q == 1) v.y = x; else if (q == 2) v.z = x; else v.w = x;
}

// Half-sweep of colour `color`, slots 2t and 2t+1 of a row. Face slots (k = 0 or
// G-1) are written back as zero, their value in the homogeneous correction.
template <bool FIRST>
__global__ void __launch_bounds__(256)
    k_rb0x2(float *__restrict__ e, const float *__restrict__ r, Split0 d, int color) {
  gc_after();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  const int kk0 = 2 * t;
  if (kk0 >= d.H || j > d.G - 2) return;
  const int p = (color + i + j) & 1;
  const int k0 = 2 * kk0 + p;  // the pair's nodes are k0 and k0 + 2
  const size_t s = ((size_t)i * d.G + j) * d.H + kk0;
  const float2 rv = ld2(r + (size_t)color * d.half + s);
  float v0, v1;
  if (FIRST) {
    v0 = __fmul_rn(0.0f - rv.x, GC_SIXTH);
    v1 = __fmul_rn(0.0f - rv.y, GC_SIXTH);
  } else {
    const float *o = e + (size_t)(color ^ 1) * d.half;
    const size_t GH = (size_t)d.G * d.H;
    const float2 xp = ld2(o + s + GH), xm = ld2(o + s - GH), yp = ld2(o + s + d.H), ym = ld2(o + s - d.H);
    const float2 zc = ld2(o + s);
    const float zo = p ? o[s + 2] : o[s - 1];
    const float az0 = p ? zc.y + zc.x : zc.x + zo;  // (k+1) + (k-1) of node k0
    const float az1 = p ? zo + zc.y : zc.y + zc.x;  // ... of node k0 + 2
    const float sum0 = ((xp.x + xm.x) + (yp.x + ym.x)) + az0;
    const float sum1 = ((xp.y + xm.y) + (yp.y + ym.y)) + az1;
    v0 = __fmul_rn(sum0 - rv.x, GC_SIXTH);
    v1 = __fmul_rn(sum1 - rv.y, GC_SIXTH);
  }
  if (k0 < 1) v0 = 0.0f;
  if (k0 + 2 > d.G - 2) v1 = 0.0f;
  st2(e + (size_t)color * d.half + s, v0, v1);
}

// Last (black) half-sweep fused with phi += e on four consecutive nodes
// 4t .. 4t+3 of a row: the black slots 2t, 2t+1 and the red ones beside them.
template <bool PLAIN>
__global__ void __launch_bounds__(256)
    k_rb0_lastx4(const float *__restrict__ e, const float *__restrict__ r, float *__restrict__ hi,
                 float *__restrict__ lo, Split0 d) {
  gc_after();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  const int kk0 = 2 * t;
  if (kk0 >= d.H || j > d.G - 2) return;
  const int pb = (1 + i + j) & 1;  // k parity of the black nodes of the row
  const size_t s = ((size_t)i * d.G + j) * d.H + kk0;
  const size_t GH = (size_t)d.G * d.H;
  const float *o = e;  // red half: the neighbours of the black nodes, and the red corrections
  const float2 xp = ld2(o + s + GH), xm = ld2(o + s - GH), yp = ld2(o + s + d.H), ym = ld2(o + s - d.H);
  const float2 zc = ld2(o + s);
  const float zo = pb ? o[s + 2] : o[s - 1];
  const float az0 = pb ? zc.y + zc.x : zc.x + zo;
  const float az1 = pb ? zo + zc.y : zc.y + zc.x;
  const float2 rb = ld2(r + d.half + s);
  const float eb0 = __fmul_rn((((xp.x + xm.x) + (yp.x + ym.x)) + az0) - rb.x, GC_SIXTH);
  const float eb1 = __fmul_rn((((xp.y + xm.y) + (yp.y + ym.y)) + az1) - rb.y, GC_SIXTH);
  const size_t c0 = ((size_t)i * d.G + j) * d.G + 2 * kk0;
  float4 h = ld4(hi + c0);
  float4 l = PLAIN ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(lo + c0);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = 2 * kk0 + q;
    if (k < 1 || k > d.G - 2) continue;
    const bool black = (q & 1) == pb;
    const float ev = black ? (q < 2 ? eb0 : eb1) : (q < 2 ? zc.x : zc.y);
    if (PLAIN) {
      f4set(h, q, __fadd_rn(f4get(h, q), ev));
    } else {
      float s1, e1, hh, llo;
      df_two_sum(f4get(h, q), ev, s1, e1);
      const float ln = __fadd_rn(f4get(l, q), e1);
      df_fast_two_sum(s1, ln, hh, llo);
      f4set(h, q, hh);
      f4set(l, q, llo);
    }
  }
  st4(hi + c0, h);
  if (!PLAIN) st4(lo + c0, l);
}

// Residual of the potential on four consecutive nodes 4t .. 4t+3 (see k_resid0).
template <bool PLAIN, bool SPLIT>
__global__ void __launch_bounds__(256)
    k_resid0x4(const float *__restrict__ hi, const float *__restrict__ lo, const float *__restrict__ b,
               float *__restrict__ rout, float *__restrict__ e_first, double *__restrict__ parts, Split0 d) {
  gc_after();
  const int G = d.G;
  const int t = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  float acc = 0.0f;
  if (4 * t < G && j <= G - 2) {
    const size_t sj = (size_t)G, si = (size_t)G * G;
    const size_t c0 = (size_t)i * si + (size_t)j * sj + 4 * t;
    const float4 hc = ld4(hi + c0), hxp = ld4(hi + c0 + si), hxm = ld4(hi + c0 - si), hyp = ld4(hi + c0 + sj),
                 hym = ld4(hi + c0 - sj);
    const float hzm = hi[c0 - 1], hzp = hi[c0 + 4];
    float4 lc = make_float4(0.f, 0.f, 0.f, 0.f), lxp = lc, lxm = lc, lyp = lc, lym = lc;
    float lzm = 0.f, lzp = 0.f;
    if (!PLAIN) {
      lc = ld4(lo + c0); lxp = ld4(lo + c0 + si); lxm = ld4(lo + c0 - si); lyp = ld4(lo + c0 + sj);
      lym = ld4(lo + c0 - sj);
      lzm = lo[c0 - 1]; lzp = lo[c0 + 4];
    }
    const float4 bv = ld4(b + c0);
    float rv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float hk = f4get(hc, q);
      const float hkp = q < 3 ? f4get(hc, q + 1) : hzp, hkm = q > 0 ? f4get(hc, q - 1) : hzm;
      if (PLAIN) {
        const float s6 = ((((f4get(hxp, q) + f4get(hxm, q)) + f4get(hyp, q)) + f4get(hym, q)) + hkp) + hkm;
        rv[q] = f4get(bv, q) - (s6 - 6.0f * hk);
      } else {
        const float lkp = q < 3 ? f4get(lc, q + 1) : lzp, lkm = q > 0 ? f4get(lc, q - 1) : lzm;
        const float h6[6] = {f4get(hxp, q), f4get(hxm, q), f4get(hyp, q), f4get(hym, q), hkp, hkm};
        const float l6[6] = {f4get(lxp, q), f4get(lxm, q), f4get(lyp, q), f4get(lym, q), lkp, lkm};
        rv[q] = df_residual_v(hk, f4get(lc, q), h6, l6, f4get(bv, q));
      }
      const int k = 4 * t + q;
      if (k < 1 || k > G - 2) rv[q] = 0.0f;  // faces: no residual, zero correction
    }
    if (SPLIT) {
      // nodes 4t, 4t+2 share a colour (slots 2t, 2t+1), as do 4t+1, 4t+3
      const int c0col = (i + j) & 1;  // colour of node 4t
      const size_t sl = ((size_t)i * G + j) * d.H + 2 * t;
      st2(rout + (size_t)c0col * d.half + sl, rv[0], rv[2]);
      st2(rout + (size_t)(c0col ^ 1) * d.half + sl, rv[1], rv[3]);
      if (e_first) {  // red = colour 0
        if (c0col == 0) st2(e_first + sl, __fmul_rn(0.0f - rv[0], GC_SIXTH), __fmul_rn(0.0f - rv[2], GC_SIXTH));
        else st2(e_first + sl, __fmul_rn(0.0f - rv[1], GC_SIXTH), __fmul_rn(0.0f - rv[3], GC_SIXTH));
      }
    } else {
      st4(rout + c0, make_float4(rv[0], rv[1], rv[2], rv[3]));
    }
    acc = ((rv[0] * rv[0] + rv[1] * rv[1]) + rv[2] * rv[2]) + rv[3] * rv[3];
  }
  const size_t bid = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  block_sum_f32(acc, parts + bid);
}

// Residual of the correction equation on four consecutive nodes, natural output.
__global__ void __launch_bounds__(256)
    k_resid0ex4(const float *__restrict__ e, const float *__restrict__ r, float *__restrict__ rc, Split0 d) {
  gc_after();
  const int G = d.G;
  const int t = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  if (4 * t >= G || j > G - 2) return;
  const int ca = (i + j) & 1;  // colour of nodes 4t, 4t+2 (half A); 4t+1, 4t+3 are half B
  const size_t s0 = ((size_t)i * G + j) * d.H + 2 * t;
  const size_t GH = (size_t)G * d.H;
  const float *A = e + (size_t)ca * d.half, *B = e + (size_t)(ca ^ 1) * d.half;
  const float2 a0 = ld2(A + s0), axp = ld2(A + s0 + GH), axm = ld2(A + s0 - GH), ayp = ld2(A + s0 + d.H),
               aym = ld2(A + s0 - d.H);
  const float a2 = A[s0 + 2];
  const float2 b0 = ld2(B + s0), bxp = ld2(B + s0 + GH), bxm = ld2(B + s0 - GH), byp = ld2(B + s0 + d.H),
               bym = ld2(B + s0 - d.H);
  const float bm = B[s0 - 1];
  const float2 ra = ld2(r + (size_t)ca * d.half + s0), rb = ld2(r + (size_t)(ca ^ 1) * d.half + s0);
  // node q: own value, other-colour sums (i, j, k) in split_nbr_sum's order
  const float sum0 = ((bxp.x + bxm.x) + (byp.x + bym.x)) + (b0.x + bm);
  const float sum1 = ((axp.x + axm.x) + (ayp.x + aym.x)) + (a0.y + a0.x);
  const float sum2 = ((bxp.y + bxm.y) + (byp.y + bym.y)) + (b0.y + b0.x);
  const float sum3 = ((axp.y + axm.y) + (ayp.y + aym.y)) + (a2 + a0.y);
  const float diag = 6.0f;
  float4 out;
  out.x = ra.x - (sum0 - diag * a0.x);
  out.y = rb.x - (sum1 - diag * b0.x);
  out.z = ra.y - (sum2 - diag * a0.y);
  out.w = rb.y - (sum3 - diag * b0.y);
  if (4 * t == 0) out.x = 0.0f;           // face k = 0
  if (4 * t + 3 == G - 1) out.w = 0.0f;  // face k = G-1
  st4(rc + ((size_t)i * G + j) * G + 4 * t, out);
}

// Level-1 correction into the black half, slots 2t and 2t+1 of a row (the two
// nodes share their i and j weights).
__global__ void __launch_bounds__(256)
    k_prolong0bx2(const float *__restrict__ ec, LevelGeom cg, float *__restrict__ e, LevelGeom f, Split0 d) {
  gc_after();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int i = blockIdx.z + 1;
  const int kk0 = 2 * t;
  if (kk0 >= d.H || j > d.G - 2) return;
  const int pb = (1 + i + j) & 1;
  const int k0 = 2 * kk0 + pb, k1 = k0 + 2;
  int ci, cj, ck0, ck1;
  float wi0, wi1, wj0, wj1, a0, a1, b0, b1;
  const int ni = prolong_w(i, f, cg, ci, wi0, wi1);
  const int nj = prolong_w(j, f, cg, cj, wj0, wj1);
  const int nk0 = prolong_w(k0, f, cg, ck0, a0, a1);
  const int nk1 = prolong_w(k1, f, cg, ck1, b0, b1);
  const size_t m = cg.n;
  float v0 = 0.0f, v1 = 0.0f;
  for (int a = 0; a < ni; ++a) {
    const float wa = a ? wi1 : wi0;
    for (int bb = 0; bb < nj; ++bb) {
      const float wb = bb ? wj1 : wj0;
      const size_t row = ((size_t)(ci + a) * m + (cj + bb)) * m;
      const float wab = wa * wb;
      v0 += wab * a0 * ec[row + ck0];
      if (nk0 == 2) v0 += wab * a1 * ec[row + ck0 + 1];
      v1 += wab * b0 * ec[row + ck1];
      if (nk1 == 2) v1 += wab * b1 * ec[row + ck1 + 1];
    }
  }
  if (k0 < 1) v0 = 0.0f;
  if (k1 > d.G - 2) v1 = 0.0f;
  float *blk = e + d.half + ((size_t)i * d.G + j) * d.H + kk0;
  const float2 old = ld2(blk);
  st2(blk, old.x + v0, old.y + v1);
}

// ------------------------------------------------------------------------------
// finest level: the way down and the way up as one pass each over the planes
// ------------------------------------------------------------------------------
// k_fine_down: three half-sweeps, the residual of the correction and its restriction
// (the first red half-sweep, from zero, included). k_fine_up: the prolongation, four
// half-sweeps and phi += e. Instead of one pass over memory per half-sweep, a CTA takes
// all k of a strip of rows and marches along i: at plane p it relaxes the newest plane
// for the first time, plane p-1 for the second time, and so on, so that a plane
// leaves the pipeline four planes later and is read and written once. Rows at the
// strip's edges (four each side) and the planes at the ends of its march are relaxed
// by its neighbours too. The arithmetic of every node is that of k_rb0x2,
// k_resid0ex4, k_restrict, k_prolong0bx2 and k_rb0_lastx4: identical potentials.
//
// A thread owns four nodes along k (two slots of each colour) of FL_RJ neighbouring
// rows and keeps, for each stage, the other colour's values at its nodes on the last
// two planes (z: plane q, x: plane q - 1) in registers; plane q + 1 is what the stage
// before has just produced. So the i neighbours, and the j neighbours inside its rows,
// cost nothing; the others come from shared memory, where every stage publishes its
// plane for the next step. One barrier per plane. With rows starting on odd j the
// k parity of the active nodes is the same in every stage of a step and alternates
// with the row and the plane: compile-time constants in a loop over plane pairs.
//
// The next step's right-hand sides are loaded at the end of a step, all together: loads
// issued among the stages held up every later wait (a warp has few scoreboards) and
// took a quarter longer. Bound by instruction issue and latency (12 warps an SM: 168
// registers each; issue slots 51 % and LSU 53 % busy, DRAM 14 to 46 %), with 24 rows of
// which 14 (down) or 16 (up) are a strip's own. Measured at 256^3: 95 us down and 99 us
// up, against 126 us for three half-sweeps, the residual and the restriction and 146 us
// for the prolongation, three half-sweeps and the last one with the update; the
// residual kernel also no longer writes the first half-sweep (69 -> 65 us).
#define FL_RJ 4
#define FL_THREADS 384
struct FL {
  static constexpr int W = 2;                         // warps along k: 128 nodes each
  static constexpr int NG = FL_THREADS / 32 / W, ROWS = FL_RJ * NG, PH = 64 * W + 4;
  static constexpr int plane = ROWS * PH;             // floats of one published half plane
  static constexpr int NJ = (ROWS - 10) / 2;          // coarse rows of a strip on the way down
  static constexpr int NR = ROWS - 8;                 // rows of a strip on the way up
  static constexpr int CR = ROWS / 2 + 2;             // coarse rows under a strip on the way up
  // a margin row, two sets of four published planes, then the pass's own
  static constexpr int pub = PH + 8 * plane;
  static constexpr size_t smem_down = sizeof(float) * (pub + 2 * ROWS * 32 * W + 2 * NG * 64 * W);
  static constexpr size_t smem_up = sizeof(float) * (pub + 2 * CR * PH + 16 * FL_RJ * FL_THREADS);
};

struct FlThread {
  int t, g, j0;        // quad, row group, first row
  bool first, last;    // quad 0, the quad of k = G - 1
  int at[FL_RJ];       // (j H + 2 t) of the row, rows and quads clamped to the grid's
  float six[FL_RJ];    // 1/6 on interior rows, else 0: results off the interior are zero
};

// The neighbour sums of the active nodes; pa: their k parity.
__device__ __forceinline__ float2 fl_sum(float2 xp, float2 xm, float2 yp, float2 ym, float2 z, float zo, int pa) {
  const float az0 = pa ? __fadd_rn(z.y, z.x) : __fadd_rn(z.x, zo);
  const float az1 = pa ? __fadd_rn(zo, z.y) : __fadd_rn(z.y, z.x);
  return make_float2(__fadd_rn(__fadd_rn(__fadd_rn(xp.x, xm.x), __fadd_rn(yp.x, ym.x)), az0),
                     __fadd_rn(__fadd_rn(__fadd_rn(xp.y, xm.y), __fadd_rn(yp.y, ym.y)), az1));
}
// (sum - r) / 6, zero on the faces k = 0 and k = G - 1 (six: 1/6, or 0 off the
// interior rows and planes)
__device__ __forceinline__ float2 fl_relax(float2 s, float2 r, float six, const FlThread &T, int pa) {
  float2 v = make_float2(__fmul_rn(__fsub_rn(s.x, r.x), six), __fmul_rn(__fsub_rn(s.y, r.y), six));
  if (pa == 0) v.x = T.first ? 0.0f : v.x;
  else v.y = T.last ? 0.0f : v.y;
  return v;
}

// One stage on all rows of the thread: the neighbour sums of its active nodes from
// xp (plane q + 1), z and x (planes q and q - 1) and, outside its rows, the plane q
// that the stage before published (buf: this thread's first slot in row 0 of the
// strip). The strip's outermost rows read whatever lies beside them: their results
// are not used.
template <int PH>
__device__ __forceinline__ void fl_sums(const float2 (&xp)[FL_RJ], const float2 (&x)[FL_RJ], const float2 (&z)[FL_RJ],
                                        const float *buf, const FlThread &T, int par, float2 (&sum)[FL_RJ]) {
  const float2 below = ld2(buf - PH), above = ld2(buf + FL_RJ * PH);
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a) {
    const int pa = (par + a) & 1;
    const float zo = buf[a * PH + (pa ? 2 : -1)];
    const float2 yp = a + 1 < FL_RJ ? z[a + 1 < FL_RJ ? a + 1 : a] : above;
    const float2 ym = a > 0 ? z[a > 0 ? a - 1 : a] : below;
    sum[a] = fl_sum(xp[a], x[a], yp, ym, z[a], zo, pa);
  }
}

template <int PH>
__device__ __forceinline__ void fl_publish(float *buf, const float2 (&v)[FL_RJ]) {
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a) st2(buf + a * PH, v[a].x, v[a].y);
}

__device__ __forceinline__ void fl_shift(float2 (&x)[FL_RJ], float2 (&z)[FL_RJ], const float2 (&v)[FL_RJ]) {
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a) {
    x[a] = z[a];
    z[a] = v[a];
  }
}

__device__ __forceinline__ FlThread fl_thread(int jb, const Split0 &d) {
  FlThread T;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T.t = 32 * (w % FL::W) + lane;
  T.g = w / FL::W;
  T.j0 = jb + FL_RJ * T.g;
  T.first = T.t == 0;
  T.last = 4 * T.t + 4 == d.G;
  const int tc = min(T.t, d.G / 4 - 1);
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a) {
    const int j = T.j0 + a;
    T.six[a] = 4 * T.t < d.G && j >= 1 && j <= d.G - 2 ? GC_SIXTH : 0.0f;
    T.at[a] = min(max(j, 0), d.G - 1) * d.H + 2 * tc;
  }
  return T;
}

// Two slots of row a on plane q (clamped) of a colour half.
__device__ __forceinline__ float2 fl_load(const float *__restrict__ half, int q, const Split0 &d, const FlThread &T,
                                          int a) {
  const float *plane = half + (size_t)min(max(q, 0), d.G - 1) * (size_t)(d.G * d.H);
  return __ldg(reinterpret_cast<const float2 *>(plane + T.at[a]));
}

struct FlDown {
  float2 x1[FL_RJ], z1[FL_RJ], x2[FL_RJ], z2[FL_RJ], x3[FL_RJ], z3[FL_RJ], x4[FL_RJ], z4[FL_RJ];
  float2 n0[FL_RJ], n1[FL_RJ], n2[FL_RJ], n3[FL_RJ], n4[FL_RJ];  // each stage's r, loaded a step ahead
  float2 rb[FL_RJ];                         // residual of the black nodes one plane ahead of the red ones'
  float r0[FL_RJ], r1[FL_RJ], sB[FL_RJ];    // plane p - 4: residuals at k = 4t, 4t + 1; k sum of K = 2t + 1
  float tA[FL_RJ], tB[FL_RJ];               // plane p - 5: k sums of K = 2t and 2t + 1
  float accA[FL_RJ / 2], accB[FL_RJ / 2];   // restricted sums under way

  // PP: parity of plane p. Restriction weights are 1/4, 1/2, 1/4, but 0 for a face
  // (wB, wj: 1/4 or 0): with G a multiple of 4 no node lies beyond the last coarse one.
  template <int PP>
  __device__ __forceinline__ void step(int p, int c, float *fs, const FlThread &T, const float *__restrict__ r,
                                       float *__restrict__ eb, float *__restrict__ bc, const Split0 &d, int m, int Jm,
                                       int I0, int I1, int je, float wB, const float (&wj)[FL_RJ / 2], unsigned own) {
    using L = FL;
    constexpr int W = L::W;
    constexpr int PH = L::PH, par = PP + 1;  // k parity of the active nodes of row 0
    const int G = d.G;
    float *base = fs + PH + FL_RJ * T.g * PH + 2 + 2 * T.t;
    float *wr = base + c * 4 * L::plane, *rd = base + (c ^ 1) * 4 * L::plane;
    float *edge = fs + L::pub + FL_RJ * T.g * 32 * W + T.t, *rows = fs + L::pub + 2 * L::ROWS * 32 * W;
    const float *red = r, *blk = r + d.half;
    // restriction, plane p - 6: row and plane sums
    {
      const float2 next = ld2(rows + 2 * (((c ^ 1) * L::NG + min(T.g + 1, L::NG - 1)) * 32 * W + T.t));
      const int i = p - 6, I = (i - 1) >> 1;  // (i has the parity of p)
#pragma unroll
      for (int h = 0; h < FL_RJ / 2; ++h) {
        const int a = 2 * h + 1;  // the centre row
        const float sA2 = a + 1 < FL_RJ ? tA[a + 1 < FL_RJ ? a + 1 : a] : next.x;
        const float sB2 = a + 1 < FL_RJ ? tB[a + 1 < FL_RJ ? a + 1 : a] : next.y;
        float uA = 0.25f * tA[a - 1], uB = 0.25f * tB[a - 1];
        uA += 0.5f * tA[a]; uB += 0.5f * tB[a];
        uA += wj[h] * sA2; uB += wj[h] * sB2;
        if (PP == 0) {  // even plane: the centre one of I
          accA[h] += 0.5f * uA;
          accB[h] += 0.5f * uB;
        } else {        // odd plane: the last one of I, the first one of I + 1
          const float wi = i <= G - 2 ? 0.25f : 0.0f;
          accA[h] += wi * uA;
          accB[h] += wi * uB;
          if (I >= I0 && I <= I1 && ((own >> (8 + h)) & 1u)) {
            float *o = bc + ((size_t)I * m + ((T.j0 + a) >> 1)) * m + 2 * T.t;
            if (!T.first) o[0] = 4.0f * accA[h];
            o[1] = 4.0f * accB[h];
          }
          accA[h] = 0.25f * uA;
          accB[h] = 0.25f * uB;
        }
      }
    }
    // restriction, plane p - 5: the k sums (K = 2t needs the quad before)
    {
      const float *er = edge + (c ^ 1) * L::ROWS * 32 * W;
#pragma unroll
      for (int a = 0; a < FL_RJ; ++a) {
        float s = 0.5f * r0[a];
        s += 0.25f * er[a * 32 * W - 1];
        s += 0.25f * r1[a];
        tA[a] = s;
        tB[a] = sB[a];
      }
      st2(rows + 2 * ((c * L::NG + T.g) * 32 * W + T.t), tA[0], tB[0]);
    }
    float2 v0[FL_RJ], v1[FL_RJ], v2[FL_RJ], v3[FL_RJ], s[FL_RJ];
    // plane p: red from zero (r is zero on the face planes)
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v0[a] = make_float2(__fmul_rn(0.0f - n0[a].x, T.six[a]), __fmul_rn(0.0f - n0[a].y, T.six[a]));
    }
    fl_publish<PH>(wr, v0);
    // plane p - 1: black
    fl_sums<PH>(v0, x1, z1, rd, T, par, s);
    const bool ok1 = p - 1 >= 1 && p - 1 <= G - 2;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v1[a] = fl_relax(s[a], n1[a], ok1 ? T.six[a] : 0.0f, T, (par + a) & 1);
    }
    fl_shift(x1, z1, v0);
    fl_publish<PH>(wr + L::plane, v1);
    // plane p - 2: red
    fl_sums<PH>(v1, x2, z2, rd + L::plane, T, par, s);
    const bool ok2 = p - 2 >= 1 && p - 2 <= G - 2;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v2[a] = fl_relax(s[a], n2[a], ok2 ? T.six[a] : 0.0f, T, (par + a) & 1);
    }
    fl_shift(x2, z2, v1);
    fl_publish<PH>(wr + 2 * L::plane, v2);
    // plane p - 3: black, and its residual
    fl_sums<PH>(v2, x3, z3, rd + 2 * L::plane, T, par, s);
    const bool ok3 = p - 3 >= 1 && p - 3 <= G - 2;
    const float diag = 6.0f;
    float2 rbn[FL_RJ];
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v3[a] = fl_relax(s[a], n3[a], ok3 ? T.six[a] : 0.0f, T, (par + a) & 1);
      rbn[a] = make_float2(n3[a].x - (s[a].x - diag * v3[a].x), n3[a].y - (s[a].y - diag * v3[a].y));
    }
    if (p - 3 >= 2 * I0 - 1 && p - 3 <= je) {  // the black correction for the way up
      float *o = eb + (size_t)(p - 3) * (size_t)(G * d.H);
#pragma unroll
      for (int a = 0; a < FL_RJ; ++a)
        if ((own >> a) & 1u) st2(o + T.at[a], v3[a].x, v3[a].y);
    }
    fl_publish<PH>(wr + 3 * L::plane, v3);
    // plane p - 4: residual of the red nodes (their values are x3), both colours in order
    fl_sums<PH>(v3, x4, z4, rd + 3 * L::plane, T, par, s);
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      const float2 rr = make_float2(n4[a].x - (s[a].x - diag * x3[a].x), n4[a].y - (s[a].y - diag * x3[a].y));
      const bool even = ((par + a) & 1) == 0;
      const float q2 = even ? rr.y : rb[a].y, q3 = even ? rb[a].y : rr.y;
      r0[a] = even ? rr.x : rb[a].x;
      r1[a] = even ? rb[a].x : rr.x;
      edge[c * L::ROWS * 32 * W + a * 32 * W] = q3;
      float k = 0.5f * q2;  // K = 2t + 1
      k += 0.25f * r1[a];
      k += wB * q3;
      sB[a] = k;
      rb[a] = rbn[a];
    }
    fl_shift(x3, z3, v2);
    fl_shift(x4, z4, v3);
    // the next step's r, all at once (a load issued among the stages would be waited for
    // with the next one's: a warp has few scoreboards)
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      n0[a] = fl_load(red, p + 1, d, T, a);
      n1[a] = fl_load(blk, p, d, T, a);
      n2[a] = fl_load(red, p - 1, d, T, a);
      n3[a] = fl_load(blk, p - 2, d, T, a);
      n4[a] = fl_load(red, p - 3, d, T, a);
    }
    __syncthreads();
  }
};

__global__ void __launch_bounds__(FL_THREADS, 1)
    k_fine_down(const float *__restrict__ r, float *__restrict__ eb, float *__restrict__ bc, Split0 d, int m, int Jm,
                int per) {
  gc_after();
  using L = FL;
  extern __shared__ __align__(16) float fs[];
  for (int i = threadIdx.x; i < (int)(L::smem_down / sizeof(float)); i += FL_THREADS) fs[i] = 0.0f;
  const int J0 = 1 + blockIdx.x * L::NJ, I0 = 1 + blockIdx.y * per, I1 = min(I0 + per - 1, Jm);
  const FlThread T = fl_thread(2 * J0 - 5, d);
  const bool in = 4 * T.t < d.G;
  // rows (bits 0 .. 3) and coarse rows (bits 8, 9) this thread writes
  const int re = J0 + L::NJ > Jm ? d.G - 2 : 2 * (J0 + L::NJ - 1);
  unsigned own = 0;
  float wj[FL_RJ / 2];
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a) {
    const int j = T.j0 + a, lr = FL_RJ * T.g + a;
    if (in && j >= 2 * J0 - 1 && j <= re) own |= 1u << a;
    if (a & 1) {
      wj[a >> 1] = j + 1 <= d.G - 2 ? 0.25f : 0.0f;
      if (in && lr >= 5 && lr < 5 + 2 * L::NJ && j >= 2 && j <= 2 * Jm) own |= 1u << (8 + (a >> 1));
    }
  }
  const float wB = T.last ? 0.0f : 0.25f;
  const int je = I1 == Jm ? d.G - 2 : 2 * I1;
  FlDown S = {};
  {  // the first step's loads
    const int p = 2 * I0 - 5;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      S.n0[a] = fl_load(r, p, d, T, a);
      S.n1[a] = fl_load(r + d.half, p - 1, d, T, a);
    }
  }
  __syncthreads();
  for (int p = 2 * I0 - 5; p <= 2 * I1 + 7; p += 2) {
    S.step<1>(p, 0, fs, T, r, eb, bc, d, m, Jm, I0, I1, je, wB, wj, own);
    S.step<0>(p + 1, 1, fs, T, r, eb, bc, d, m, Jm, I0, I1, je, wB, wj, own);
  }
}

__device__ __forceinline__ void fl_cp4(float *dst, const float *src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 4u : 0u)
               : "memory");
}
__device__ __forceinline__ void fl_cp16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void fl_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <bool PLAIN>
struct FlUp {
  float2 x1[FL_RJ], z1[FL_RJ], x2[FL_RJ], z2[FL_RJ], x3[FL_RJ], z3[FL_RJ], x4[FL_RJ], z4[FL_RJ];
  float2 ne[FL_RJ], n1[FL_RJ], n2[FL_RJ], n3[FL_RJ], n4[FL_RJ];  // the next step's correction and r

  // coarse plane I under the strip (rows from c0) into its slot of the ring of two
  static __device__ __forceinline__ void coarse(float *ring, const float *__restrict__ ec, int I, int c0, int m) {
    using L = FL;
    const int lane = threadIdx.x & 31;
    for (int rr = threadIdx.x >> 5; rr < L::CR; rr += FL_THREADS / 32) {
      const int J = c0 + rr;
      const bool in = I >= 0 && I < m && J >= 0 && J < m;
      const float *src = ec + (in ? ((size_t)I * m + J) * m : 0);
      float *dst = ring + ((I & 1) * L::CR + rr) * L::PH;
#pragma unroll
      for (int K = 0; K < L::PH; K += 32)
        if (K + lane < L::PH) fl_cp4(dst + K + lane, in && K + lane < m ? src + K + lane : ec, in && K + lane < m);
    }
  }
  // hi and lo of plane q (the strip's own rows), into the thread's own slots
  static __device__ __forceinline__ void phi(float *slot, const float *hi, const float *lo, int q, int i1, int i2,
                                             int G, const FlThread &T, unsigned own) {
    if (q < i1 || q > i2) return;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      if (!((own >> a) & 1u)) continue;
      const size_t c0 = ((size_t)q * G + T.j0 + a) * G + 4 * T.t;
      fl_cp16(slot + (2 * a) * 4 * FL_THREADS, hi + c0);
      if (!PLAIN) fl_cp16(slot + (2 * a + 1) * 4 * FL_THREADS, lo + c0);
    }
  }

  template <int PP>
  __device__ __forceinline__ void step(int p, int c, float *fs, const FlThread &T, const float *__restrict__ ec,
                                       const float *__restrict__ eb, const float *__restrict__ r, float *hi, float *lo,
                                       const Split0 &d, int m, int i1, int i2, int cr0, unsigned own) {
    using L = FL;
    constexpr int PH = L::PH, par = PP;  // k parity of the active nodes of row 0
    const int G = d.G;
    float *base = fs + PH + FL_RJ * T.g * PH + 2 + 2 * T.t;
    float *wr = base + c * 4 * L::plane, *rd = base + (c ^ 1) * 4 * L::plane;
    float *ring = fs + L::pub, *slot = ring + 2 * L::CR * PH + 4 * threadIdx.x;
    const float *red = r, *blk = r + d.half;
    // the next step's potential, and the next coarse plane before an odd plane needs it
    phi(slot + (c ^ 1) * 8 * FL_RJ * FL_THREADS, hi, lo, p - 3, i1, i2, G, T, own);
    if (PP == 0) coarse(ring, ec, (p >> 1) + 1, cr0, m);
    float2 v0[FL_RJ], v1[FL_RJ], v2[FL_RJ], v3[FL_RJ], s[FL_RJ];
    // plane p: black, the correction of the way down plus the prolonged coarse one:
    // weight 1 on even coordinates, 1/2 and 1/2 on odd ones (with G a multiple of 4 no
    // interior node lies beyond the last coarse one), in k_prolong0bx2's order
    const float okp = p >= 1 && p <= G - 2 ? 1.0f : 0.0f;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      // row j0 + a is odd for even a; its coarse row and the one after it
      constexpr int ni = PP ? 2 : 1;
      const int pa = (par + a) & 1, nj = a & 1 ? 1 : 2;
      const float *q = ring + (((T.j0 + a) >> 1) - cr0) * PH + 2 * T.t;
      const float w = (ni == 2 ? 0.5f : 1.0f) * (nj == 2 ? 0.5f : 1.0f) * (pa ? 0.5f : 1.0f);
      float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int u = 0; u < ni; ++u)
#pragma unroll
        for (int h = 0; h < nj; ++h) {
          const float *row = q + ((((p >> 1) + u) & 1) * L::CR + h) * PH;
          const float2 e01 = ld2(row);
          v.x += w * e01.x;
          if (pa) v.x += w * e01.y;
          v.y += w * e01.y;
          if (pa) v.y += w * row[2];
        }
      const float on = T.six[a] != 0.0f ? okp : 0.0f;
      v = make_float2(__fmul_rn(__fadd_rn(ne[a].x, v.x), on), __fmul_rn(__fadd_rn(ne[a].y, v.y), on));
      if (pa == 0) v.x = T.first ? 0.0f : v.x;
      else v.y = T.last ? 0.0f : v.y;
      v0[a] = v;
    }
    fl_publish<PH>(wr, v0);
    // planes p - 1 (red), p - 2 (black), p - 3 (red)
    fl_sums<PH>(v0, x1, z1, rd, T, par, s);
    const bool ok1 = p - 1 >= 1 && p - 1 <= G - 2;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v1[a] = fl_relax(s[a], n1[a], ok1 ? T.six[a] : 0.0f, T, (par + a) & 1);
    }
    fl_shift(x1, z1, v0);
    fl_publish<PH>(wr + L::plane, v1);
    fl_sums<PH>(v1, x2, z2, rd + L::plane, T, par, s);
    const bool ok2 = p - 2 >= 1 && p - 2 <= G - 2;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v2[a] = fl_relax(s[a], n2[a], ok2 ? T.six[a] : 0.0f, T, (par + a) & 1);
    }
    fl_shift(x2, z2, v1);
    fl_publish<PH>(wr + 2 * L::plane, v2);
    fl_sums<PH>(v2, x3, z3, rd + 2 * L::plane, T, par, s);
    const bool ok3 = p - 3 >= 1 && p - 3 <= G - 2;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      v3[a] = fl_relax(s[a], n3[a], ok3 ? T.six[a] : 0.0f, T, (par + a) & 1);
    }
    fl_shift(x3, z3, v2);
    fl_publish<PH>(wr + 3 * L::plane, v3);
    // plane p - 4: black, then phi += e for the quad (the red nodes are z4)
    fl_sums<PH>(v3, x4, z4, rd + 3 * L::plane, T, par, s);
    const int q = p - 4;
    const bool mine = q >= i1 && q <= i2;
    const float *pv = slot + c * 8 * FL_RJ * FL_THREADS;
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      const float2 rv = n4[a];
      if (!mine || !((own >> a) & 1u)) continue;
      const float2 e = make_float2(__fmul_rn(s[a].x - rv.x, GC_SIXTH), __fmul_rn(s[a].y - rv.y, GC_SIXTH));
      const bool even = ((par + a) & 1) == 0;  // the black nodes are k = 4t, 4t + 2
      const float ev[4] = {even ? e.x : z4[a].x, even ? z4[a].x : e.x, even ? e.y : z4[a].y, even ? z4[a].y : e.y};
      const size_t c0 = ((size_t)q * G + T.j0 + a) * G + 4 * T.t;
      float4 h = ld4(pv + (2 * a) * 4 * FL_THREADS);
      float4 l = PLAIN ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(pv + (2 * a + 1) * 4 * FL_THREADS);
      const float hx = h.x, lx = l.x, hw = h.w, lw = l.w;
      phi_sum<PLAIN>(h.x, l.x, ev[0]);
      phi_sum<PLAIN>(h.y, l.y, ev[1]);
      phi_sum<PLAIN>(h.z, l.z, ev[2]);
      phi_sum<PLAIN>(h.w, l.w, ev[3]);
      if (T.first) { h.x = hx; l.x = lx; }
      if (T.last) { h.w = hw; l.w = lw; }
      st4(hi + c0, h);
      if (!PLAIN) st4(lo + c0, l);
    }
    fl_shift(x4, z4, v3);
    fl_cp_wait();
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      ne[a] = fl_load(eb, p + 1, d, T, a);
      n1[a] = fl_load(red, p, d, T, a);
      n2[a] = fl_load(blk, p - 1, d, T, a);
      n3[a] = fl_load(red, p - 2, d, T, a);
      n4[a] = fl_load(blk, p - 3, d, T, a);
    }
    __syncthreads();
  }
};

template <bool PLAIN>
__global__ void __launch_bounds__(FL_THREADS, 1)
    k_fine_up(const float *__restrict__ ec, int m, const float *__restrict__ eb, const float *__restrict__ r, float *hi,
              float *lo, Split0 d, int per) {
  gc_after();
  using L = FL;
  extern __shared__ __align__(16) float fs[];
  for (int i = threadIdx.x; i < (int)(L::smem_up / sizeof(float)); i += FL_THREADS) fs[i] = 0.0f;
  const int j1 = 1 + blockIdx.x * L::NR, i1 = 1 + blockIdx.y * per, i2 = min(i1 + per - 1, d.G - 2);
  const FlThread T = fl_thread(j1 - 4, d);
  const int cr0 = (j1 - 4) >> 1;
  unsigned own = 0;  // rows whose potential this thread updates
#pragma unroll
  for (int a = 0; a < FL_RJ; ++a)
    if (T.six[a] != 0.0f && T.j0 + a >= j1 && T.j0 + a < j1 + L::NR) own |= 1u << a;
  FlUp<PLAIN> S = {};
  __syncthreads();
  {  // the first step's coarse planes and loads
    const int p = i1 - 4;
    float *ring = fs + L::pub;
    FlUp<PLAIN>::coarse(ring, ec, p >> 1, cr0, m);
    FlUp<PLAIN>::coarse(ring, ec, (p >> 1) + 1, cr0, m);
#pragma unroll
    for (int a = 0; a < FL_RJ; ++a) {
      S.ne[a] = fl_load(eb, p, d, T, a);
      S.n1[a] = fl_load(r, p - 1, d, T, a);
    }
    fl_cp_wait();
  }
  __syncthreads();
  for (int p = i1 - 4; p <= i2 + 4; p += 2) {
    S.template step<1>(p, 0, fs, T, ec, eb, r, hi, lo, d, m, i1, i2, cr0, own);
    S.template step<0>(p + 1, 1, fs, T, ec, eb, r, hi, lo, d, m, i1, i2, cr0, own);
  }
}

// ------------------------------------------------------------------------------
// a level's way down and way up in one launch each, block by block
// ------------------------------------------------------------------------------
// k_block_down: the pre-smoothing from a zero correction, the residual and its
// restriction. k_block_up: the prolongation and the post-smoothing (on the finest
// level with phi += e). A CTA takes a block of nodes and relaxes a region around it
// in shared memory that shrinks by one node a side with every half-sweep, so that
// its block is exact when it gets there: no grid-wide barrier or launch between
// the phases, at the price of relaxing the halo in several CTAs (about four times
// the nodes; the data comes from L2). The arithmetic of every node is that of
// k_smooth / k_resid / k_restrict / k_prolong, so the results equal theirs bit for bit.
//
// A warp is a row j of the region, its lanes the 32 nodes k of the row, and a thread
// walks its column along i: the nodes of one colour lie on every other plane, odd
// and even lanes on alternating ones, so all lanes work at each step and their
// shared-memory words are in 32 different banks. Bound by shared-memory accesses:
// six a node and half-sweep (the i neighbours are carried along the column, the
// right-hand sides stay in registers: reading them from L1 in every half-sweep
// took twice as long).
//
// Only the black nodes pass from the way down to the way up: the first half-sweep of
// the way up overwrites the red ones without reading them. They go through an
// array of their own (neighbouring blocks still read it while a block writes its
// result).
//
// Measured (us per V-cycle, levels 129^3, 65^3 and 33^3 under a 256^3 grid): 124 now
// (down 30.6 + 7.6 + 7.6, up 37.5 + 10 + 10, one launch each) against 156 for two
// cooperative launches with a grid barrier between the phases; one level of 33^3
// under 64^3: 17 against 26.
template <int NS>
struct BlkD {  // way down, NS sweeps: coarse nodes per block along j and k, region
  static constexpr int H = 2 * NS - 1;            // extra halo of the first half-sweep
  static constexpr int CJ = 8, CK = (32 - 3 - 2 * H) / 2;
  static constexpr int LJ = 2 * CJ + 3 + 2 * H;   // rows (warps)
};
template <int NS>
struct BlkU {  // way up: nodes per block along j and k, region
  static constexpr int H = 2 * NS;
  static constexpr int TJ = 16, TK = 32 - 2 * H;
  static constexpr int LJ = TJ + 2 * H;
};

// A thread's column in shared memory and registers: node (i0 + t, j, k) at col + t SI,
// t < LI; its nodes of one colour are t = 2 m + o, and their right-hand sides bv[m].
template <int LI, int LJ>
struct BlkCol {
  static constexpr int SI = LJ * 32, M = (LI + 1) / 2;
  float *col;
  int i0, J, o[2];   // o[c]: first plane of colour c
  float bv[2][M];
  float a, d0, d1, r0, r1;  // far-face weight; diagonal and its reciprocal below and at i = J
  bool lj, lk, in_jk;

  __device__ __forceinline__ void init(float *c, const float *__restrict__ b, const LevelGeom &g, int i0_, int j, int k) {
    col = c;
    i0 = i0_;
    J = g.J;
    in_jk = j >= 1 && j <= J && k >= 1 && k <= J;
    o[0] = (i0 + j + k) & 1;
    o[1] = o[0] ^ 1;
    lj = j == J;
    lk = k == J;
    a = g.a;
    const float dj = lj ? g.dB : 2.0f, dk = lk ? g.dB : 2.0f;
    d0 = (2.0f + dj) + dk;
    d1 = (g.dB + dj) + dk;
    r0 = d0 == 6.0f ? GC_SIXTH : __frcp_rn(d0);
    r1 = d1 == 6.0f ? GC_SIXTH : __frcp_rn(d1);
    const long long n = g.n, nn = n * n;
    const float *bp = b + (long long)i0 * nn + (long long)j * n + k;
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {  // all in flight together
        const int t = 2 * m + o[c2];
        bv[c2][m] = in_jk && t < LI && i0 + t >= 1 && i0 + t <= J ? __ldg(bp + t * nn) : 0.0f;
      }
  }
  // x / diagonal as gs_value does it: times 1/6 where the diagonal is 6, else the
  // correctly rounded quotient from the reciprocal and the exact remainder
  // (Markstein, IBM J. Res. Dev. 34, 1990; the first quotient can be off by more than his
  // theorem takes, but all 2^23 significands were divided by each of the 1633 diagonals of
  // grids to 1024^3, and every quotient is the rounded one)
  __device__ __forceinline__ float over(float x, bool li) const {
    const float d = li ? d1 : d0, r = li ? r1 : r0, q = __fmul_rn(x, r);
    return d == 6.0f ? q : __fmaf_rn(__fmaf_rn(-q, d, x), r, q);
  }
  __device__ __forceinline__ float sum_at(const float *p, float below, float above, bool li) const {
    const float sx = li ? __fmul_rn(a, below) : __fadd_rn(above, below);
    const float sy = lj ? __fmul_rn(a, p[-32]) : __fadd_rn(p[32], p[-32]);
    const float sz = lk ? __fmul_rn(a, p[-1]) : __fadd_rn(p[1], p[-1]);
    return __fadd_rn(__fadd_rn(sx, sy), sz);
  }
  // One half-sweep of colour C over the planes [s, LI - 1 - s]; `far` (uniform in the
  // warp): the block holds far-face nodes.
  template <int C>
  __device__ __forceinline__ void sweep(int s, bool far) {
    const int tl = s > 1 - i0 ? s : 1 - i0, th = LI - 1 - s < J - i0 ? LI - 1 - s : J - i0;
    float *p = col + o[C] * SI;
    float below = o[C] ? col[0] : 0.0f;
    if (far) {
#pragma unroll
      for (int m = 0; m < M; ++m, p += 2 * SI) {
        const int t = 2 * m + o[C];
        const float above = t + 1 < LI ? p[SI] : 0.0f;
        if (t >= tl && t <= th) {
          const bool li = i0 + t == J;
          *p = over(__fsub_rn(sum_at(p, below, above, li), bv[C][m]), li);
        }
        below = above;
      }
    } else {
#pragma unroll
      for (int m = 0; m < M; ++m, p += 2 * SI) {
        const int t = 2 * m + o[C];
        const float above = t + 1 < LI ? p[SI] : 0.0f;
        if (t >= tl && t <= th) {
          const float sum = __fadd_rn(__fadd_rn(__fadd_rn(above, below), __fadd_rn(p[32], p[-32])),
                                      __fadd_rn(p[1], p[-1]));
          *p = __fmul_rn(__fsub_rn(sum, bv[C][m]), GC_SIXTH);
        }
        below = above;
      }
    }
  }
};

// The separable full weighting of restrict_node on a residual in shared memory (zero
// on the faces); p points at fine node (2 I - 1, 2 J - 1, 2 K - 1).
__device__ __forceinline__ float blk_restrict(const float *p, int SI, const float (&wi)[3], const float (&wj)[3],
                                              const float (&wk)[3]) {
  float acc = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float ta = 0.0f;
#pragma unroll
    for (int bb = 0; bb < 3; ++bb) {
      const float *row = p + a * SI + bb * 32;
      float sab = wk[1] * row[1];
      sab += wk[0] * row[0];
      sab += wk[2] * row[2];
      ta += wj[bb] * sab;
    }
    acc += wi[a] * ta;
  }
  return 4.0f * acc;
}

template <int NS, int CI>
__global__ void __launch_bounds__(32 * BlkD<NS>::LJ, 1)
    k_block_down(float *__restrict__ e, const float *__restrict__ b, LevelGeom g, float *__restrict__ bc, LevelGeom cg) {
  gc_after();
  using B = BlkD<NS>;
  constexpr int H = B::H, LJ = B::LJ, LI = 2 * CI + 3 + 2 * H;
  using Col = BlkCol<LI, LJ>;
  constexpr int SI = Col::SI, M = Col::M;
  extern __shared__ float blk_sm[];
  float *E = blk_sm;
  float *R = E + LI * SI;                 // residual on planes and rows [H + 1, L - 2 - H] of E
  constexpr int RJ = 2 * B::CJ + 1, RSI = RJ * 32;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int I0 = 1 + blockIdx.z * CI, J0 = 1 + blockIdx.y * B::CJ, K0 = 1 + blockIdx.x * B::CK;
  const int i0 = 2 * I0 - 2 - H, j = 2 * J0 - 2 - H + row, k0 = 2 * K0 - 2 - H, k = k0 + lane;
  const bool far = i0 + LI > g.J || j == g.J || k0 + 31 >= g.J;
  Col c;
  c.init(E + row * 32 + lane, b, g, i0, j, k);
  // red half-sweep from zero; black nodes and everything outside the interior are zero
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int tr = 2 * m + c.o[0], tb = 2 * m + c.o[1];
    if (tr < LI) c.col[tr * SI] = c.over(0.0f - c.bv[0][m], i0 + tr == g.J);
    if (tb < LI) c.col[tb * SI] = 0.0f;
  }
  __syncthreads();
#pragma unroll
  for (int s = 1; s < 2 * NS; ++s) {
    if (c.in_jk && row >= s && row < LJ - s && lane >= s && lane < 32 - s) {
      if (s & 1) c.template sweep<1>(s, far);
      else c.template sweep<0>(s, far);
    }
    __syncthreads();
  }
  // residual around the block's coarse nodes, zero off the interior
  if (row >= H + 1 && row < H + 1 + RJ) {
    const bool mine = c.in_jk && lane >= H + 1 && lane < 32 - H - 1;
    float *rp = R + (row - H - 1) * 32 + lane;
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = 2 * m + c.o[q], i = i0 + t;
        if (t < H + 1 || t > LI - 2 - H) continue;
        float v = 0.0f;
        if (mine && i >= 1 && i <= g.J) {
          const float *p = c.col + t * SI;
          const bool li = i == g.J;
          const float sum = c.sum_at(p, p[-SI], p[SI], li), diag = li ? c.d1 : c.d0;
          v = c.bv[q][m] - (sum - diag * p[0]);
        }
        rp[(t - H - 1) * RSI] = v;
      }
  }
  // the block's black nodes (fine nodes 2 I - 1 and 2 I of its coarse nodes I, and the
  // one past the last coarse node) for the way up
  {
    const size_t n = g.n, nn = n * n;
    const int ie = I0 + CI > cg.J ? g.J : 2 * (I0 + CI) - 2, je = J0 + B::CJ > cg.J ? g.J : 2 * (J0 + B::CJ) - 2,
              ke = K0 + B::CK > cg.J ? g.J : 2 * (K0 + B::CK) - 2;
    if (j >= 2 * J0 - 1 && j <= je && k >= 2 * K0 - 1 && k <= ke) {
#pragma unroll 4
      for (int i = 2 * I0 - 1 + ((j + k) & 1); i <= ie; i += 2)
        e[(size_t)i * nn + (size_t)j * n + k] = c.col[(i - i0) * SI];
    }
  }
  __syncthreads();
  constexpr int NC = CI * B::CJ * B::CK;
  for (int q = threadIdx.x; q < NC; q += 32 * LJ) {
    const int dk = q % B::CK, r = q / B::CK, dj = r % B::CJ, di = r / B::CJ;
    const int I = I0 + di, Jc = J0 + dj, K = K0 + dk;
    if (I > cg.J || Jc > cg.J || K > cg.J) continue;
    float wi[3], wj[3], wk[3];
#pragma unroll
    for (int o = -1; o <= 1; ++o) {
      wi[o + 1] = restrict_w(I, o, g, cg);
      wj[o + 1] = restrict_w(Jc, o, g, cg);
      wk[o + 1] = restrict_w(K, o, g, cg);
    }
    bc[((size_t)I * cg.n + Jc) * cg.n + K] =
        blk_restrict(R + 2 * di * RSI + 2 * dj * 32 + (H + 1 + 2 * dk), RSI, wi, wj, wk);
  }
}

// PHI: 0 coarse level (e_out), 1 finest level in double-float, 2 in plain f32 (phi += e).
template <int NS, int TI, int PHI>
__global__ void __launch_bounds__(32 * BlkU<NS>::LJ, 1)
    k_block_up(const float *__restrict__ ec, LevelGeom cg, const float *__restrict__ e, const float *__restrict__ b,
               LevelGeom g, float *__restrict__ e_out, float *__restrict__ hi, float *__restrict__ lo) {
  gc_after();
  using B = BlkU<NS>;
  constexpr int H = B::H, LJ = B::LJ, LI = TI + 2 * H;
  using Col = BlkCol<LI, LJ>;
  constexpr int SI = Col::SI, M = Col::M;
  constexpr int PJ = LJ / 2 + 2, PI = LI / 2 + 2, PK = 18;  // the coarse nodes the region interpolates from
  extern __shared__ float blk_sm[];
  float *E = blk_sm, *C = E + LI * SI;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int i0 = 1 + blockIdx.z * TI - H, j0 = 1 + blockIdx.y * B::TJ - H, k0 = 1 + blockIdx.x * B::TK - H;
  const int j = j0 + row, k = k0 + lane;
  const int ci = i0 >> 1, cj = j0 >> 1, ck = k0 >> 1;  // (floor, also below zero)
  const bool far = i0 + LI > g.J || j == g.J || k0 + 31 >= g.J;
  const long long n = g.n, nn = n * n;
  Col c;
  c.init(E + row * 32 + lane, b, g, i0, j, k);
  // black nodes: the correction of the way down ...
  float ev[M];
  {
    const float *ep = e + (long long)i0 * nn + (long long)j * n + k;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int t = 2 * m + c.o[1];
      ev[m] = c.in_jk && t < LI && i0 + t >= 1 && i0 + t <= g.J ? __ldg(ep + t * nn) : 0.0f;
    }
  }
  for (int q = threadIdx.x; q < PI * PJ * PK; q += 32 * LJ) {
    const int dk = q % PK, r = q / PK, dj = r % PJ, di = r / PJ;
    const int I = ci + di, Jc = cj + dj, K = ck + dk;
    const bool in = I >= 0 && I < cg.n && Jc >= 0 && Jc < cg.n && K >= 0 && K < cg.n;
    C[q] = in ? __ldg(ec + ((size_t)I * cg.n + Jc) * cg.n + K) : 0.0f;
  }
  __syncthreads();
  // ... plus the prolonged coarse one; the rest starts at zero (red nodes are
  // overwritten unread)
  {
    // (prolong_value's terms in its order; the j and k weights are the column's)
    int c0, cj0, ck0;
    float wi0, wi1, wj[2], wk[2];
    const int nj = prolong_w(j, g, cg, cj0, wj[0], wj[1]), nk = prolong_w(k, g, cg, ck0, wk[0], wk[1]);
    const float *cs = C + (cj0 - cj) * PK + (ck0 - ck);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int tb = 2 * m + c.o[1], tr = 2 * m + c.o[0], i = i0 + tb;
      float v = 0.0f;
      if (c.in_jk && i >= 1 && i <= g.J) {
        const int ni = prolong_w(i, g, cg, c0, wi0, wi1);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int bb = 0; bb < 2; ++bb) {
            if (a >= ni || bb >= nj) continue;
            const float *q = cs + (c0 - ci + a) * (PJ * PK) + bb * PK;
            const float wab = (a ? wi1 : wi0) * wj[bb];
            v += wab * wk[0] * q[0];
            if (nk == 2) v += wab * wk[1] * q[1];
          }
        v = ev[m] + v;
      }
      if (tb < LI) c.col[tb * SI] = v;
      if (tr < LI) c.col[tr * SI] = 0.0f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < 2 * NS; ++s) {
    if (c.in_jk && row > s && row < LJ - 1 - s && lane > s && lane < 31 - s) {
      if (s & 1) c.template sweep<1>(s + 1, far);
      else c.template sweep<0>(s + 1, far);
    }
    __syncthreads();
  }
  if (!(c.in_jk && row >= H && row < LJ - H && lane >= H && lane < 32 - H)) return;
  const size_t q0 = (size_t)(i0 + H) * nn + (size_t)j * n + k;
  const int nt = g.J - (i0 + H) + 1;  // planes of the block inside the interior
  if (PHI == 0) {
#pragma unroll
    for (int t = 0; t < TI; ++t)
      if (t < nt) e_out[q0 + t * nn] = c.col[(H + t) * SI];
  } else {
    float h[TI], l[TI];
#pragma unroll
    for (int t = 0; t < TI; ++t) {
      h[t] = t < nt ? hi[q0 + t * nn] : 0.0f;
      l[t] = PHI == 1 && t < nt ? lo[q0 + t * nn] : 0.0f;
    }
#pragma unroll
    for (int t = 0; t < TI; ++t) {
      phi_sum<PHI == 2>(h[t], l[t], c.col[(H + t) * SI]);
      if (t < nt) {
        hi[q0 + t * nn] = h[t];
        if (PHI == 1) lo[q0 + t * nn] = l[t];
      }
    }
  }
}

// ------------------------------------------------------------------------------
// tail: all levels with n <= GC_TAIL_MAX_N relaxed by one CTA in shared memory
// ------------------------------------------------------------------------------
// The far face of the coarsest level is at p in (1, 2], so it has one unknown; the
// levels above it have J <= 3, 7 and 15. Each level is relaxed by as many threads
// as it has work for: 1024, 256 (a named barrier) and one warp, the single unknown
// of the last one by one thread in FP64. Bound by latency: about 40 dependent
// phases. So a thread keeps its nodes' right-hand sides, addresses and divisors in
// registers across the sweeps, the transfers are branch-free (weight-zero terms
// read zeros), and the divisions by the far-face diagonals multiply by a
// reciprocal tabulated once and correct the quotient by its exact remainder
// (Markstein, IBM J. Res. Dev. 34, 1990). Measured, all four levels: 34 us with
// every phase on all 1024 threads and pointer tables in local memory, 28 with the
// levels on their own threads, 17 us now.
struct TailDesc {
  int first;         // first level present, 0 .. 3
  int pre, post;
  LevelGeom g[4];    // J <= 15, 7, 3 and J == 1
};

// Level q of the tail: Q = log2 of its 16, 8, 4 rows, P its row pitch (25 spreads the
// rows of a warp over the banks: 8 slots of stride 2 from 4 rows).
template <int Q>
struct TL {
  static constexpr int P = Q == 4 ? 25 : (1 << Q) + 1;
  static constexpr int S = ((1 << Q) + 1) * P;                  // plane stride
  static constexpr int NT = Q == 4 ? 1024 : Q == 3 ? 256 : 32;  // threads that relax it
  static constexpr int words = ((1 << Q) + 1) * S;              // one array
};
static_assert(GC_TAIL_MAX_N == 17, "the tail's levels have at most 15 interior nodes per axis");

// Tables of a level, filled once per launch: Gauss-Seidel diagonal and its
// reciprocal by far-face bits (i, j, k at J), and the 1-D transfer weights between
// it and the next level: restriction weight rw[3 I + a + 1] = restrict_w(I, a);
// prolongation of fine index i: coarse index pc[i], weights pw[2 i], pw[2 i + 1] (the
// second 0 where there is one node).
#define TAIL_TAB 16  // indices 0 .. GC_TAIL_MAX_N - 2
struct TailTab {
  float dg[8], rc[8];
  float rw[TAIL_TAB * 3];
  float pw[TAIL_TAB * 2];
  int pc[TAIL_TAB];
};

// One entry per thread t < 8 + 3 * TAIL_TAB + TAIL_TAB.
__device__ __forceinline__ void t_tables(TailTab &t, const LevelGeom &f, const LevelGeom &cg, int q) {
  if (q < 8) {
    const float dg = ((q & 4 ? f.dB : 2.0f) + (q & 2 ? f.dB : 2.0f)) + (q & 1 ? f.dB : 2.0f);
    t.dg[q] = dg;
    t.rc[q] = dg == 6.0f ? GC_SIXTH : __frcp_rn(dg);
  } else if (q < 8 + 3 * TAIL_TAB) {
    const int w = q - 8, I = w / 3, a = w - 3 * I - 1;
    t.rw[w] = I >= 1 && I <= cg.J ? restrict_w(I, a, f, cg) : 0.0f;
  } else if (q < 8 + 4 * TAIL_TAB) {
    const int i = q - 8 - 3 * TAIL_TAB;
    int c0 = 0, cnt = 0;
    float w0 = 0.0f, w1 = 0.0f;
    if (i >= 1 && i <= f.J) cnt = prolong_w(i, f, cg, c0, w0, w1);
    t.pc[i] = c0;
    t.pw[2 * i] = w0;
    t.pw[2 * i + 1] = cnt == 2 ? w1 : 0.0f;
  }
}

template <int NT>
__device__ __forceinline__ void t_sync() {
  if (NT == 1024) __syncthreads();
  else if (NT == 32) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

// Weighted neighbour sum at p, the far-face terms as in sw_axis.
__device__ __forceinline__ float t_sum(const float *p, int S, int P, float a, bool li, bool lj, bool lk) {
  const float xm = p[-S], xp = p[S], ym = p[-P], yp = p[P], zm = p[-1], zp = p[1];
  const float sx = li ? __fmul_rn(a, xm) : __fadd_rn(xp, xm);
  const float sy = lj ? __fmul_rn(a, ym) : __fadd_rn(yp, ym);
  const float sz = lk ? __fmul_rn(a, zm) : __fadd_rn(zp, zm);
  return __fadd_rn(__fadd_rn(sx, sy), sz);
}

// Red-black sweeps. Thread (kk, j, i0) takes the nodes k = 2 kk + parity of the rows
// (i, j), i = i0 and (16-row level) i0 + 8, which share their parity.
template <int Q>
__device__ __forceinline__ void t_smooth(float *e, const float *b, const LevelGeom &g, const TailTab &tb, int sweeps) {
  constexpr int P = TL<Q>::P, S = TL<Q>::S, NT = TL<Q>::NT, ST = NT >> (2 * Q - 1), NI = (1 << Q) / ST;
  const int J = g.J;
  const int kk = threadIdx.x & ((1 << (Q - 1)) - 1), j = ((threadIdx.x >> (Q - 1)) & ((1 << Q) - 1)) + 1;
  const int i0 = (threadIdx.x >> (2 * Q - 1)) + 1;
  const float a = g.a;
  const bool lj = j == J;
  float bv[2][NI], rc[2][NI], dg[2][NI];
  bool ok[2][NI], li[NI];
  int at[2];
#pragma unroll
  for (int u = 0; u < NI; ++u) li[u] = i0 + u * ST == J;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int k = 2 * kk + ((c + i0 + j) & 1);
    at[c] = i0 * S + j * P + k;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      ok[c][u] = j <= J && k >= 1 && k <= J && i0 + u * ST <= J;
      const int face = (li[u] ? 4 : 0) + (lj ? 2 : 0) + (k == J ? 1 : 0);
      rc[c][u] = tb.rc[face];
      dg[c][u] = tb.dg[face];
      bv[c][u] = ok[c][u] ? b[at[c] + u * ST * S] : 0.0f;
    }
  }
  for (int s = 0; s < sweeps; ++s) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const bool lk = 2 * kk + ((c + i0 + j) & 1) == J;
      float v[NI];
#pragma unroll
      for (int u = 0; u < NI; ++u) {
        if (!ok[c][u]) continue;
        const float x = __fsub_rn(t_sum(e + at[c] + u * ST * S, S, P, a, li[u], lj, lk), bv[c][u]);
        const float q = __fmul_rn(x, rc[c][u]);
        v[u] = dg[c][u] == 6.0f ? q : __fmaf_rn(__fmaf_rn(-q, dg[c][u], x), rc[c][u], q);
      }
#pragma unroll
      for (int u = 0; u < NI; ++u)
        if (ok[c][u]) e[at[c] + u * ST * S] = v[u];
      t_sync<NT>();
    }
  }
}

// r = b - L e; (k, j, i) of the thread: i = i0, i0 + 4, ... (or 2)
template <int Q>
__device__ __forceinline__ void t_resid(const float *e, const float *b, float *r, const LevelGeom &g,
                                        const TailTab &tb) {
  constexpr int P = TL<Q>::P, S = TL<Q>::S, NT = TL<Q>::NT;
  const int J = g.J;
  const int k = (threadIdx.x & ((1 << Q) - 1)) + 1, j = ((threadIdx.x >> Q) & ((1 << Q) - 1)) + 1;
  if (k <= J && j <= J) {
#pragma unroll
    for (int i = (threadIdx.x >> (2 * Q)) + 1, u = 0; u < (1 << (3 * Q)) / NT; i += NT >> (2 * Q), ++u) {
      if (i > J) continue;
      const int c = i * S + j * P + k;
      const bool li = i == J, lj = j == J, lk = k == J;
      const float diag = tb.dg[(li ? 4 : 0) + (lj ? 2 : 0) + (lk ? 1 : 0)];
      r[c] = b[c] - (t_sum(e + c, S, P, g.a, li, lj, lk) - diag * e[c]);
    }
  }
  t_sync<NT>();
}

// b_c = 4 R(r_f) at the coarse node (I, Jj, K); r is zero on the faces.
template <int Q>
__device__ __forceinline__ float t_restrict_node(const float *rf, int I, int Jj, int K, const TailTab &tb) {
  float wa[3], wb[3], wc[3];
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    wa[o] = tb.rw[3 * I + o];
    wb[o] = tb.rw[3 * Jj + o];
    wc[o] = tb.rw[3 * K + o];
  }
  const float *p = rf + (2 * I - 1) * TL<Q>::S + (2 * Jj - 1) * TL<Q>::P + (2 * K - 1);
  float acc = 0.0f;
#pragma unroll
  for (int o = 0; o < 3; ++o)
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int c = 0; c < 3; ++c) acc += wa[o] * wb[m] * wc[c] * p[o * TL<Q>::S + m * TL<Q>::P + c];
  return 4.0f * acc;
}

// Level Q -> Q - 1, by level Q's threads (the caller synchronises).
template <int Q>
__device__ __forceinline__ void t_restrict(const float *rf, float *bc, const LevelGeom &cg, const TailTab &tb) {
  constexpr int C = Q - 1;
  const int J = cg.J;
  const int K = (threadIdx.x & ((1 << C) - 1)) + 1, Jj = ((threadIdx.x >> C) & ((1 << C) - 1)) + 1;
  const int I = (threadIdx.x >> (2 * C)) + 1;
  if (K <= J && Jj <= J && I <= J)
    bc[I * TL<C>::S + Jj * TL<C>::P + K] = t_restrict_node<Q>(rf, I, Jj, K, tb);
}

// e_f += P(e_c) on level Q by its threads (pitch and plane stride of e_c: PC, SC).
template <int Q, int PC, int SC>
__device__ __forceinline__ void t_prolong(const float *ec, float *ef, const LevelGeom &f, const TailTab &tb) {
  constexpr int P = TL<Q>::P, S = TL<Q>::S, NT = TL<Q>::NT;
  const int J = f.J;
  const int k = (threadIdx.x & ((1 << Q) - 1)) + 1, j = ((threadIdx.x >> Q) & ((1 << Q) - 1)) + 1;
  if (k <= J && j <= J) {
    const int cj = tb.pc[j], ck = tb.pc[k];
    const float wj[2] = {tb.pw[2 * j], tb.pw[2 * j + 1]}, wk[2] = {tb.pw[2 * k], tb.pw[2 * k + 1]};
#pragma unroll
    for (int i = (threadIdx.x >> (2 * Q)) + 1, u = 0; u < (1 << (3 * Q)) / NT; i += NT >> (2 * Q), ++u) {
      if (i > J) continue;
      const float wi[2] = {tb.pw[2 * i], tb.pw[2 * i + 1]};
      const float *p = ec + tb.pc[i] * SC + cj * PC + ck;
      float val = 0.0f;
#pragma unroll
      for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int c = 0; c < 2; ++c) val += wi[o] * wj[m] * wk[c] * p[o * SC + m * PC + c];
      ef[i * S + j * P + k] += val;
    }
  }
  t_sync<NT>();
}

#define TAIL_SMEM ((3 * (TL<4>::words + TL<3>::words + TL<2>::words) + 27) * sizeof(float))

// The first level's nodes (i, j, k) of thread t and round u, as a global index; -1 if none.
template <int Q>
__device__ __forceinline__ int t_node(int u, int n, int &sm) {
  const int k = (threadIdx.x & ((1 << Q) - 1)) + 1, j = ((threadIdx.x >> Q) & ((1 << Q) - 1)) + 1;
  const int i = (threadIdx.x >> (2 * Q)) + 1 + u * (1024 >> (2 * Q));
  sm = i * TL<Q>::S + j * TL<Q>::P + k;
  return i < n - 1 && j < n - 1 && k < n - 1 ? (i * n + j) * n + k : -1;
}

__global__ void __launch_bounds__(1024) k_tail(const float *__restrict__ b_in, float *__restrict__ e_out, TailDesc d) {
  gc_after();
  extern __shared__ float tsm[];
  float *EA = tsm, *BA = EA + TL<4>::words, *RA = BA + TL<4>::words;
  float *EB = RA + TL<4>::words, *BB = EB + TL<3>::words, *RB = BB + TL<3>::words;
  float *EC = RB + TL<3>::words, *BC = EC + TL<2>::words, *RC = BC + TL<2>::words;
  float *ED = RC + TL<2>::words;  // the coarsest level's correction: 3^3, one nonzero
  __shared__ TailTab tabs[3];
  __shared__ double inv_d;        // reciprocal of the coarsest level's diagonal
  const int tid = threadIdx.x, first = d.first;
  const int n0 = d.g[first].n;
  // right-hand side of the first level (its interior), in flight while the rest is set up
  float b0[4];
  int sm;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    int q = -1;
    if (first == 0) q = t_node<4>(u, n0, sm);
    else if (first == 1 && u == 0) q = t_node<3>(u, n0, sm);
    else if (first == 2 && u == 0) q = t_node<2>(u, n0, sm);
    else if (first == 3 && u == 0) q = tid == 0 ? 13 : -1;
    b0[u] = q >= 0 ? b_in[q] : 0.0f;
  }
  // tables, 128 threads per level; zero everything (corrections start at zero, and
  // the faces of corrections and residuals stay zero)
  if (tid < 384 && (tid >> 7) >= first) t_tables(tabs[tid >> 7], d.g[tid >> 7], d.g[(tid >> 7) + 1], tid & 127);
  if (tid == 1023) {
    const double dB = (double)d.g[3].dB;
    inv_d = 1.0 / (dB + dB + dB);
  }
  for (int i = tid; i < (int)(TAIL_SMEM / sizeof(float)); i += 1024) tsm[i] = 0.0f;
  __syncthreads();
  if (first == 0) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (t_node<4>(u, n0, sm) >= 0) BA[sm] = b0[u];
  } else if (first == 1) {
    if (t_node<3>(0, n0, sm) >= 0) BB[sm] = b0[0];
  } else if (first == 2) {
    if (t_node<2>(0, n0, sm) >= 0) BC[sm] = b0[0];
  }
  __syncthreads();
  if (first == 0) {
    t_smooth<4>(EA, BA, d.g[0], tabs[0], d.pre);
    t_resid<4>(EA, BA, RA, d.g[0], tabs[0]);
    t_restrict<4>(RA, BB, d.g[1], tabs[0]);
    __syncthreads();
  }
  if (first <= 1 && tid < TL<3>::NT) {
    t_smooth<3>(EB, BB, d.g[1], tabs[1], d.pre);
    t_resid<3>(EB, BB, RB, d.g[1], tabs[1]);
    t_restrict<3>(RB, BC, d.g[2], tabs[1]);
    t_sync<TL<3>::NT>();
  }
  if (tid < 32) {
    float bd = b0[0];
    if (first <= 2) {
      t_smooth<2>(EC, BC, d.g[2], tabs[2], d.pre);
      t_resid<2>(EC, BC, RC, d.g[2], tabs[2]);
      bd = t_restrict_node<2>(RC, 1, 1, 1, tabs[2]);
    }
    // one unknown, every neighbour on a face: solved in FP64
    if (tid == 0) ED[13] = (float)(-(double)bd * inv_d);
    __syncwarp();
    if (first <= 2) {
      t_prolong<2, 3, 9>(ED, EC, d.g[2], tabs[2]);
      t_smooth<2>(EC, BC, d.g[2], tabs[2], d.post);
    }
  }
  if (first <= 1 && tid < TL<3>::NT) {
    t_sync<TL<3>::NT>();
    t_prolong<3, TL<2>::P, TL<2>::S>(EC, EB, d.g[1], tabs[1]);
    t_smooth<3>(EB, BB, d.g[1], tabs[1], d.post);
  }
  __syncthreads();
  if (first == 0) {
    t_prolong<4, TL<3>::P, TL<3>::S>(EB, EA, d.g[0], tabs[0]);
    t_smooth<4>(EA, BA, d.g[0], tabs[0], d.post);
  }
  // the interior (the faces of e_out are zero and stay so)
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (first == 0) {
      const int q = t_node<4>(u, n0, sm);
      if (q >= 0) e_out[q] = EA[sm];
    } else if (u == 0) {
      const int q = first == 1 ? t_node<3>(0, n0, sm) : first == 2 ? t_node<2>(0, n0, sm) : tid == 0 ? 13 : -1;
      if (q >= 0) e_out[q] = first == 1 ? EB[sm] : first == 2 ? EC[sm] : ED[13];
    }
  }
}

// ------------------------------------------------------------------------------
// boundary faces, moments, scaling
// ------------------------------------------------------------------------------
// Multipole Dirichlet faces (multigrid.py:261-295) evaluated in FP64 from the raw
// moments (multigrid.py:378-389), written as double-float pairs.
__global__ void __launch_bounds__(256)
    k_faces(float *__restrict__ hi, float *__restrict__ lo, int G,
            double dx, double grav, const double *__restrict__ mom) {
  gc_after();
  // centre of mass and second moments about it, once per block (FP64 runs at a
  // small fraction of the f32 rate: each face node keeps only its own terms)
  __shared__ double sm[11];
  if (threadIdx.x == 0) {
    const double M = mom[0];
    const double cx = M > 0.0 ? mom[1] / M : 0.0, cy = M > 0.0 ? mom[2] / M : 0.0, cz = M > 0.0 ? mom[3] / M : 0.0;
    sm[0] = M; sm[1] = cx; sm[2] = cy; sm[3] = cz;
    sm[4] = mom[4] - M * cx * cx; sm[5] = mom[5] - M * cy * cy; sm[6] = mom[6] - M * cz * cz;
    sm[7] = mom[7] - M * cx * cy; sm[8] = mom[8] - M * cx * cz; sm[9] = mom[9] - M * cy * cz;
    sm[10] = sm[4] + sm[5] + sm[6];
  }
  __syncthreads();
  const int GG = G * G;  // 6 G^2 < 2^31 for G <= 1024
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 6 * GG) return;
  const int face = t / GG;
  const int rem = t - face * GG;
  const int u = rem / G, v = rem - u * G;
  int i, j, k;
  switch (face) {
    case 0: i = 0; j = u; k = v; break;
    case 1: i = G - 1; j = u; k = v; break;
    case 2: j = 0; i = u; k = v; break;
    case 3: j = G - 1; i = u; k = v; break;
    case 4: k = 0; i = u; j = v; break;
    default: k = G - 1; i = u; j = v; break;
  }
  const double M = sm[0];
  double phi = 0.0;
  if (M > 0.0) {
    const double rx = i * dx - sm[1], ry = j * dx - sm[2], rz = k * dx - sm[3];
    const double d2 = rx * rx + ry * ry + rz * rz + 1e-12;
    // 1/sqrt(d2): the f32 estimate refined by two Newton steps y <- y (3 - d2 y^2) / 2
    // in FP64 (relative error 2^-23 -> 2^-46 -> below the FP64 rounding), a
    // handful of FP64 operations instead of a square root and a division
    double inv = (double)rsqrtf((float)d2);
    inv = inv * (1.5 - 0.5 * d2 * inv * inv);
    inv = inv * (1.5 - 0.5 * d2 * inv * inv);
    // n.S.n d^2 as the quadratic form of r (no normalised n)
    const double rsr = rx * (rx * sm[4] + 2.0 * (ry * sm[7] + rz * sm[8])) + ry * (ry * sm[5] + 2.0 * rz * sm[9]) +
                       rz * rz * sm[6];
    const double inv2 = inv * inv;
    const double quad = 3.0 * rsr * inv2 - sm[10];
    // Phi = -G (M/d + (3 n.S.n - tr S) / (2 d^3)), multigrid.py:261-295
    phi = -grav * (M * inv + quad * (0.5 * inv2 * inv));
  }
  const size_t c = ((size_t)i * G + j) * G + k;
  const float h = (float)phi;
  const float l = (float)(phi - (double)h);
  hi[c] = h;
  lo[c] = l;
}

// Moments of an f32 density and, with b0, its h^2-scaled right-hand side
// b0 = h^2 * f32(f32(4 pi G) * rho) with ||b0||^2, in one pass. A warp takes
// eight neighbouring columns (i, j .. j+7) at a time, persistent over those
// units: Kahan-compensated FP32 sums of rho, rho k and rho k^2 along k (the
// reference's column scheme, multigrid.py:192-221), finished in FP64. The squares of b0 are
// added eight to a tree and those as pairs: a chain of single sums (220 squares a thread at
// 256^3) was 2.3e-8 off in ||b0||, the 32 squares of a thread before that 2.7e-9, this 1.4e-10.
//
// Bound by HBM (read rho, write b0) once FP64 is kept out of the way: an FP64
// warp instruction, conversions included, takes 16 clocks of the SM on this part.
// So the lanes' column sums, unevaluated pairs s - c as they are, meet as FP32 pairs
// in a reduce-scatter (9 pair additions per sum for eight columns) and only the
// eight column totals become FP64; the block's sums are added by ten lanes, and
// the last block finishes the grid's. Measured at 256^3: 405 us for the moments
// (10 values reduced by FP64 shuffles in each of 8192 blocks) and 29 us for the
// right-hand side before, 50 us for both now (99 us with the reduce-scatter in FP64);
// at 64^3 33 + 3 us before, 12 now.
#define MOM_COLS 8
// (rh, rl) = (ah + al) + (bh + bl) as a pair
__device__ __forceinline__ void pair_add(float ah, float al, float bh, float bl, float &rh, float &rl) {
  float h, e;
  df_two_sum(ah, bh, h, e);
  df_fast_two_sum(h, __fadd_rn(e, __fadd_rn(al, bl)), rh, rl);
}

__global__ void __launch_bounds__(256, 2)
    k_rhs_moments(const float *__restrict__ rho, float *__restrict__ b0, int G, double dx, float fpg, float h2,
                  double *__restrict__ parts, unsigned *__restrict__ ticket, double *__restrict__ mom,
                  double *__restrict__ bnorm2, unsigned *__restrict__ status) {
  gc_after();
  __shared__ double wsum[8 * MOM_COLS][11];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int upr = (G + MOM_COLS - 1) / MOM_COLS;  // units per i
  const long long nunits = (long long)G * upr;
  // a row of sums per (warp, column): kept in shared memory, only its lane touches it
  for (int t = threadIdx.x; t < 8 * MOM_COLS * 11; t += 256) (&wsum[0][0])[t] = 0.0;
  __syncthreads();
  float acc = 0.0f, accl = 0.0f;  // ||b0||^2 of the thread, as a pair
  bool bad = false;
  // the column of the unit whose sums this lane ends up with (bits 4, 3, 2 of the lane)
  const int mine = lane >> 2;
  for (long long u = (long long)blockIdx.x * 8 + wid; u < nunits; u += (long long)gridDim.x * 8) {
    const int i = (int)(u / upr), j0 = (int)(u - (long long)i * upr) * MOM_COLS;
    const int nc = G - j0 < MOM_COLS ? G - j0 : MOM_COLS;
    const size_t at = ((size_t)i * G + j0) * G;
    float s[3][MOM_COLS], c[3][MOM_COLS];
#pragma unroll
    for (int t = 0; t < MOM_COLS; ++t)
#pragma unroll
      for (int q = 0; q < 3; ++q) s[q][t] = c[q][t] = 0.0f;
    // the next 32 nodes of the columns are loaded while these are summed
    float r[MOM_COLS], rn[MOM_COLS];
    const float *src = rho + at + lane;
#pragma unroll
    for (int t = 0; t < MOM_COLS; ++t) rn[t] = t < nc && lane < G ? src[(size_t)t * G] : 0.0f;
    for (int k = lane; k < G; k += 32) {
      const float fk = (float)k;
#pragma unroll
      for (int t = 0; t < MOM_COLS; ++t) r[t] = rn[t];
      src += 32;
#pragma unroll
      for (int t = 0; t < MOM_COLS; ++t) rn[t] = t < nc && k + 32 < G ? src[(size_t)t * G] : 0.0f;
      if (b0) {
        float bv[MOM_COLS];
#pragma unroll
        for (int t = 0; t < MOM_COLS; ++t) {
          bv[t] = __fmul_rn(__fmul_rn(fpg, r[t]), h2);
          if (t < nc) b0[at + (size_t)t * G + k] = bv[t];
        }
        const float q0 = __fmaf_rn(bv[1], bv[1], __fmul_rn(bv[0], bv[0])), q1 = __fmaf_rn(bv[3], bv[3], __fmul_rn(bv[2], bv[2])),
                    q2 = __fmaf_rn(bv[5], bv[5], __fmul_rn(bv[4], bv[4])), q3 = __fmaf_rn(bv[7], bv[7], __fmul_rn(bv[6], bv[6]));
        float e;
        df_two_sum(acc, __fadd_rn(__fadd_rn(q0, q1), __fadd_rn(q2, q3)), acc, e);
        accl = __fadd_rn(accl, e);
      }
#pragma unroll
      for (int t = 0; t < MOM_COLS; ++t) {
        const bool fin = fabsf(r[t]) <= 3.402823466e38f;
        bad |= !fin;
        const float x = fin ? r[t] : 0.0f, x1 = __fmul_rn(x, fk);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float y = q == 2 ? __fmaf_rn(x1, fk, -c[q][t]) : __fsub_rn(q ? x1 : x, c[q][t]), z = __fadd_rn(s[q][t], y);
          c[q][t] = __fsub_rn(__fsub_rn(z, s[q][t]), y);
          s[q][t] = z;
        }
      }
    }
    double S[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      // the lanes' pairs (s, -c) summed as pairs: lane bits 4, 3, 2 pick the column
#pragma unroll
      for (int t = 0; t < MOM_COLS; ++t) c[q][t] = -c[q][t];
#pragma unroll
      for (int w = MOM_COLS / 2, o = 16; w >= 1; w >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;  // keeps the upper half of the columns
#pragma unroll
        for (int t = 0; t < MOM_COLS / 2; ++t) {
          if (t >= w) break;
          const float gh = __shfl_xor_sync(0xffffffffu, up ? s[q][t] : s[q][t + w], o);
          const float gl = __shfl_xor_sync(0xffffffffu, up ? c[q][t] : c[q][t + w], o);
          pair_add(up ? s[q][t + w] : s[q][t], up ? c[q][t + w] : c[q][t], gh, gl, s[q][t], c[q][t]);
        }
      }
#pragma unroll
      for (int o = 2; o >= 1; o >>= 1) {
        const float gh = __shfl_xor_sync(0xffffffffu, s[q][0], o), gl = __shfl_xor_sync(0xffffffffu, c[q][0], o);
        pair_add(s[q][0], c[q][0], gh, gl, s[q][0], c[q][0]);
      }
      S[q] = (double)s[q][0] + (double)c[q][0];
    }
    if ((lane & 3) == 0) {  // raw moments in node units; the spacing is applied at the end
      const double x = (double)i, y = (double)(j0 + mine);
      const double S0x = S[0] * x, S0y = S[0] * y;
      double *v = wsum[wid * MOM_COLS + mine];
      v[0] += S[0]; v[1] += S0x; v[2] += S0y; v[3] += S[1];
      v[4] += S0x * x; v[5] += S0y * y; v[6] += S[2];
      v[7] += S0x * y; v[8] += S[1] * x; v[9] += S[1] * y;
    }
  }
  if (bad) atomicOr(status, GC_FLAG_NONFINITE_RHO);
  // the lanes' pairs of ||b0||^2 (an overflow stays an infinity: its error terms are NaN)
  accl = fabsf(acc) <= 3.402823466e38f ? accl : 0.0f;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const float gh = __shfl_xor_sync(0xffffffffu, acc, o), gl = __shfl_xor_sync(0xffffffffu, accl, o);
    const float h = __fadd_rn(acc, gh);
    if (fabsf(h) <= 3.402823466e38f) {
      pair_add(acc, accl, gh, gl, acc, accl);
    } else {
      acc = h;
      accl = 0.0f;
    }
  }
  if (lane == 0) wsum[wid * MOM_COLS][10] = (double)acc + (double)accl;
  __syncthreads();
  if (threadIdx.x < 11) {
    const int q = threadIdx.x;
    const double vol = dx * dx * dx;
    const double sc = q == 10 ? 1.0 : q == 0 ? vol : q <= 3 ? vol * dx : vol * dx * dx;
    double a = 0.0;
    for (int r = 0; r < 8 * MOM_COLS; ++r) a += wsum[r][q];
    wsum[0][q] = a * sc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // one writer: the last-block reduction fences its stores
    for (int q = 0; q < 11; ++q) parts[(size_t)blockIdx.x * 11 + q] = wsum[0][q];
  }
  if (grid_finish_sum<11>(parts, gridDim.x, ticket, mom) && threadIdx.x == 0 && b0) *bnorm2 = mom[10];
}

// Zero the interior nodes 1 .. G-2 of a G^3 array (node_grid launch shape).
__global__ void __launch_bounds__(256) k_zero_interior(float *__restrict__ a, int G) {
  const int k = blockIdx.x * 32 + threadIdx.x + 1, j = blockIdx.y * 8 + threadIdx.y + 1, i = blockIdx.z + 1;
  if (k <= G - 2 && j <= G - 2) a[((size_t)i * G + j) * G + k] = 0.0f;
}

// ------------------------------------------------------------------------------
// host orchestration
// ------------------------------------------------------------------------------
static dim3 rb_grid(const LevelGeom &g) {
  const int nkk = g.n / 2 + 1;
  return dim3(gc_blocks(nkk, RB_TX), gc_blocks(g.J, RB_TY), (unsigned)g.J);
}
static dim3 node_grid(const LevelGeom &g) { return dim3(gc_blocks(g.J, 32), gc_blocks(g.J, 8), (unsigned)g.J); }
// Sweeps each way on the levels below the finest.
static int coarse_pre(const gc_mg_params *p) { return (p->flags & GC_MG_COARSE_ONE_SWEEP) ? 1 : p->pre_sweeps; }
static int coarse_post(const gc_mg_params *p) { return (p->flags & GC_MG_COARSE_ONE_SWEEP) ? 1 : p->post_sweeps; }

static int launch_smooth(gc_ctx *ctx, int l, int sweeps) {
  const LevelGeom &g = ctx->lev[l];
  for (int s = 0; s < sweeps; ++s)
    for (int color = 0; color < 2; ++color)
      gc_launch(ctx, GK_SMOOTH, k_smooth, dim3(rb_grid(g)), dim3(dim3(RB_TX, RB_TY)), 0, ctx->e[l], ctx->b[l], g, color);
  GC_LAUNCH_CHECK(ctx, "smooth");
  return GC_OK;
}

static int launch_tail(gc_ctx *ctx, const gc_mg_params *p) {
  TailDesc d;
  memset(&d, 0, sizeof(d));
  const int nl = ctx->nlev - ctx->tail;
  // the coarsest level has one unknown (its far face is at most two nodes away),
  // and every level above it at most twice as many per axis and one
  GC_REQUIRE(ctx, nl >= 1 && nl <= 4 && ctx->lev[ctx->nlev - 1].J == 1, "tail: unexpected level sizes");
  d.first = 4 - nl;
  d.pre = coarse_pre(p);
  d.post = coarse_post(p);
  for (int l = 0; l < nl; ++l) d.g[d.first + l] = ctx->lev[ctx->tail + l];
  if (!ctx->tail_smem_set) {  // opt in to more than 48 KB (once per context)
    GC_CUDA(ctx, cudaFuncSetAttribute(k_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM));
    ctx->tail_smem_set = 1;
  }
  gc_launch_after(ctx, GK_TAIL, k_tail, dim3(1), dim3(1024), TAIL_SMEM, ctx->b[ctx->tail], ctx->e[ctx->tail], d);
  GC_LAUNCH_CHECK(ctx, "tail");
  return GC_OK;
}

static int finalize_to(gc_ctx *ctx, int nparts, int slot, const MgDecide *dec = nullptr);

static Split0 split0(const gc_ctx *ctx) {
  Split0 d;
  d.G = ctx->G;
  d.H = ctx->H0;
  d.half = ctx->half0;
  return d;
}
// (kk, j, i) over the interior rows of the colour-split finest level
static dim3 split_grid(const gc_ctx *ctx) {
  return dim3(gc_blocks(ctx->H0, 64), gc_blocks(ctx->G - 2, 4), (unsigned)(ctx->G - 2));
}
#define SPLIT_BLOCK dim3(64, 4)
// slot pairs (vectorised kernels, G % 4 == 0)
static dim3 split_grid2(const gc_ctx *ctx) {
  return dim3(gc_blocks(ctx->H0 / 2, 64), gc_blocks(ctx->G - 2, 4), (unsigned)(ctx->G - 2));
}
// node quads of the interior rows (vectorised kernels, G % 4 == 0)
static dim3 quad_grid(const gc_ctx *ctx) {
  return dim3(gc_blocks(ctx->G / 4, 32), gc_blocks(ctx->G - 2, 8), (unsigned)(ctx->G - 2));
}
static bool vec4(const gc_ctx *ctx) { return ctx->G % 4 == 0; }

template <int NS, int CI>
static size_t blk_down_smem() {
  using B = BlkD<NS>;
  return sizeof(float) * 32 * ((size_t)(2 * CI + 3 + 2 * B::H) * B::LJ + (size_t)(2 * CI + 1) * (2 * B::CJ + 1));
}
template <int NS, int TI>
static size_t blk_up_smem() {
  using B = BlkU<NS>;
  const size_t LI = TI + 2 * B::H;
  return sizeof(float) * (32 * LI * B::LJ + (LI / 2 + 2) * (B::LJ / 2 + 2) * 18);
}

// Blocks are 8 coarse planes (way down) or 16 planes (way up) long; half as long
// where that leaves SMs without a block (63^3 nodes: 48 long blocks, 96 short ones).
template <int NS, int CI>
static int blk_down(gc_ctx *ctx, int kid, float *e, const float *b, const LevelGeom &g, float *bc,
                    const LevelGeom &cg) {
  using B = BlkD<NS>;
  const dim3 grid(gc_blocks(cg.J, B::CK), gc_blocks(cg.J, B::CJ), gc_blocks(cg.J, CI));
  if (CI > 4 && (unsigned long long)grid.x * grid.y * grid.z < gc_sms())
    return blk_down<NS, 4>(ctx, kid, e, b, g, bc, cg);
  const size_t smem = blk_down_smem<NS, CI>();
  if (smem > 48 * 1024)
    GC_CUDA(ctx, cudaFuncSetAttribute(k_block_down<NS, CI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gc_launch_after(ctx, kid, k_block_down<NS, CI>, grid, dim3(32 * B::LJ), smem, e, b, g, bc, cg);
  GC_LAUNCH_CHECK(ctx, "block down");
  return GC_OK;
}
static int block_down(gc_ctx *ctx, int kid, int sweeps, float *e, const float *b, const LevelGeom &g, float *bc,
                      const LevelGeom &cg) {
  return sweeps == 1 ? blk_down<1, 8>(ctx, kid, e, b, g, bc, cg) : blk_down<2, 8>(ctx, kid, e, b, g, bc, cg);
}

template <int NS, int PHI, int TI>
static int blk_up(gc_ctx *ctx, int kid, const float *ec, const LevelGeom &cg, const float *e, const float *b,
                  const LevelGeom &g, float *e_out) {
  using B = BlkU<NS>;
  const dim3 grid(gc_blocks(g.J, B::TK), gc_blocks(g.J, B::TJ), gc_blocks(g.J, TI));
  if (TI > 8 && (unsigned long long)grid.x * grid.y * grid.z < gc_sms())
    return blk_up<NS, PHI, 8>(ctx, kid, ec, cg, e, b, g, e_out);
  const size_t smem = blk_up_smem<NS, TI>();
  if (smem > 48 * 1024)
    GC_CUDA(ctx,
            cudaFuncSetAttribute(k_block_up<NS, TI, PHI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gc_launch_after(ctx, kid, k_block_up<NS, TI, PHI>, grid, dim3(32 * B::LJ), smem, ec, cg, e, b, g, e_out, ctx->hi, ctx->lo);
  GC_LAUNCH_CHECK(ctx, "block up");
  return GC_OK;
}
template <int PHI>
static int block_up(gc_ctx *ctx, int kid, int sweeps, const float *ec, const LevelGeom &cg, const float *e,
                    const float *b, const LevelGeom &g, float *e_out) {
  return sweeps == 1 ? blk_up<1, PHI, 16>(ctx, kid, ec, cg, e, b, g, e_out)
                     : blk_up<2, PHI, 16>(ctx, kid, ec, cg, e, b, g, e_out);
}

// Sweep counts the block kernels are built for.
static bool block_sweeps(int pre, int post) { return pre >= 1 && pre <= 2 && post >= 1 && post <= 2; }

// The finest level block by block on a natural-layout correction: for grids whose
// eleven colour-split passes are too short to fill the GPU. Measured, kernel us per
// V-cycle in blocks and in passes: 64^3 66 and 73, 80^3 93 and 91, 100^3 120 and 105;
// without the vectorised passes (G not a multiple of 4) 97^3 111 and 116, 129^3 157
// and 162. Nine launches fewer decide where the two are even.
static bool finest_blocks(const gc_ctx *ctx, const gc_mg_params *p) {
  return ctx->nlev > 1 && ctx->G <= (ctx->G % 4 == 0 ? 80 : 129) && !(p->flags & GC_MG_NATURAL_LAYOUT) &&
         block_sweeps(p->pre_sweeps, p->post_sweeps);
}

// The finest level as two passes over its planes (two sweeps each way): rows of at most
// 64 quads, and grids large enough that the passes' halos weigh less than the traffic
// they save. Measured, kernel us per V-cycle in plane passes and in half-sweeps: 128^3
// 140 and 126, 144^3 177 and 181, 192^3 254 and 277, 256^3 405 and 488.
static bool finest_planes(const gc_ctx *ctx, const gc_mg_params *p) {
  return ctx->nlev > 1 && ctx->G % 4 == 0 && ctx->G >= 144 && ctx->G <= 256 && !(p->flags & GC_MG_NATURAL_LAYOUT) &&
         p->pre_sweeps == 2 && p->post_sweeps == 2 && !finest_blocks(ctx, p);
}

// Strips of rows along x; along y as many stretches of planes as the remaining SMs
// allow (one CTA per SM).
static int fine_down(gc_ctx *ctx) {
  using L = FL;
  const LevelGeom &cg = ctx->lev[1];
  const unsigned strips = gc_blocks(cg.J, L::NJ);
  const unsigned parts = gc_sms() > strips ? gc_sms() / strips : 1;
  const int per = (int)gc_blocks(cg.J, (int)parts);
  GC_CUDA(ctx, cudaFuncSetAttribute(k_fine_down, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem_down));
  gc_launch_after(ctx, GK_SMOOTH0, k_fine_down, dim3(strips, gc_blocks(cg.J, per)), dim3(FL_THREADS), L::smem_down,
            ctx->r0s, ctx->e0s + ctx->half0, ctx->b[1], split0(ctx), cg.n, cg.J, per);
  GC_LAUNCH_CHECK(ctx, "fine down");
  return GC_OK;
}
template <bool PLAIN>
static int fine_up(gc_ctx *ctx) {
  using L = FL;
  const LevelGeom &g0 = ctx->lev[0], &cg = ctx->lev[1];
  const unsigned strips = gc_blocks(g0.J, L::NR);
  const unsigned parts = gc_sms() > strips ? gc_sms() / strips : 1;
  const int per = ((int)gc_blocks(g0.J, (int)parts) + 1) & ~1;  // even: a stretch starts on an odd plane
  GC_CUDA(ctx, cudaFuncSetAttribute(k_fine_up<PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem_up));
  gc_launch_after(ctx, GK_UPDATE0, k_fine_up<PLAIN>, dim3(strips, gc_blocks(g0.J, per)), dim3(FL_THREADS), L::smem_up,
            ctx->e[1], cg.n, ctx->e0s + ctx->half0, ctx->r0s, ctx->hi, ctx->lo, split0(ctx), per);
  GC_LAUNCH_CHECK(ctx, "fine up");
  return GC_OK;
}

// Levels 1 .. nlev-1 of a V-cycle: b[1] in, e[1] out: one launch per level each way
// around the single-CTA tail. Sweep counts the block kernels do not have, and the
// validation path (natural layout), take one launch per phase.
static int coarse_levels(gc_ctx *ctx, const gc_mg_params *p) {
  const int L = ctx->nlev, pre = coarse_pre(p), post = coarse_post(p);
  int st;
  if (!(p->flags & GC_MG_NATURAL_LAYOUT) && block_sweeps(pre, post)) {
    for (int l = 1; l < ctx->tail; ++l)
      if ((st = block_down(ctx, GK_COARSE, pre, ctx->ed[l], ctx->b[l], ctx->lev[l], ctx->b[l + 1], ctx->lev[l + 1])))
        return st;
    if (ctx->tail < L && (st = launch_tail(ctx, p))) return st;
    for (int l = ctx->tail - 1; l >= 1; --l)
      if ((st = block_up<0>(ctx, GK_COARSE, post, ctx->e[l + 1], ctx->lev[l + 1], ctx->ed[l], ctx->b[l], ctx->lev[l],
                            ctx->e[l])))
        return st;
    return GC_OK;
  }
  for (int l = 1; l < ctx->tail; ++l) {
    const LevelGeom &g = ctx->lev[l];
    const size_t n3 = (size_t)g.n * g.n * g.n;
    GC_CUDA(ctx, cudaMemsetAsync(ctx->e[l], 0, n3 * sizeof(float), ctx->stream));
    if ((st = launch_smooth(ctx, l, pre))) return st;
    gc_launch(ctx, GK_RESID, k_resid, dim3(node_grid(g)), dim3(dim3(32, 8)), 0, ctx->e[l], ctx->b[l], ctx->rc, g);
    gc_launch_after(ctx, GK_RESTRICT, k_restrict, dim3(node_grid(ctx->lev[l + 1])), dim3(dim3(32, 8)), 0, ctx->rc, g,
              ctx->b[l + 1], ctx->lev[l + 1]);
    GC_LAUNCH_CHECK(ctx, "resid/restrict");
  }
  if (ctx->tail < L) {
    if ((st = launch_tail(ctx, p))) return st;
  }
  for (int l = ctx->tail - 1; l >= 1; --l) {
    gc_launch(ctx, GK_PROLONG, k_prolong, dim3(node_grid(ctx->lev[l])), dim3(dim3(32, 8)), 0, ctx->e[l + 1],
              ctx->lev[l + 1], ctx->e[l], ctx->lev[l]);
    GC_LAUNCH_CHECK(ctx, "prolong");
    if ((st = launch_smooth(ctx, l, post))) return st;
  }
  return GC_OK;
}

// r = b0 - L phi on the finest interior (colour-split, or natural for the
// validation path), with ||r||^2 into dsmall[GC_S_RNORM2] (async). The split
// path also writes the first red half-sweep of the next pre-smoothing.
static int residual0(gc_ctx *ctx, const gc_mg_params *p, const MgDecide *dec) {
  const LevelGeom &g0 = ctx->lev[0];
  const dim3 grid = node_grid(g0);
  const size_t nb = (size_t)grid.x * grid.y * grid.z;
  int st = gc_ensure_red(ctx, nb);
  if (st) return st;
  const bool plain = (p->flags & GC_MG_PLAIN_F32) != 0;
  const Split0 d = split0(ctx);
  const bool natural = (p->flags & GC_MG_NATURAL_LAYOUT) != 0 || finest_blocks(ctx, p);
  if ((st = mg_alloc_finest(ctx, p))) return st;
  const int pre = ctx->nlev == 1 ? p->coarse_sweeps : p->pre_sweeps;
  float *ef = pre >= 1 && !natural && !finest_planes(ctx, p) ? ctx->e0s : nullptr, *r = natural ? ctx->r0n : ctx->r0s;
  if (vec4(ctx) && !(p->flags & GC_MG_NATURAL_LAYOUT)) {
    const dim3 qg = quad_grid(ctx);
    const size_t nq = (size_t)qg.x * qg.y * qg.z;
    if ((st = gc_ensure_red(ctx, nq))) return st;
    auto k = natural ? (plain ? k_resid0x4<true, false> : k_resid0x4<false, false>)
                     : (plain ? k_resid0x4<true, true> : k_resid0x4<false, true>);
    gc_launch_after(ctx, GK_RESID0, k, qg, dim3(32, 8), 0, ctx->hi, ctx->lo, ctx->b0, r, ef, ctx->red, d);
    GC_LAUNCH_CHECK(ctx, "resid0");
    // (a last-block sum of the 16k block partials in this kernel was slower: the
    // blocks' tickets serialise on one counter)
    return finalize_to(ctx, (int)nq, GC_S_RNORM2, dec);
  }
  auto k = natural ? (plain ? k_resid0<true, false> : k_resid0<false, false>)
                   : (plain ? k_resid0<true, true> : k_resid0<false, true>);
  gc_launch_after(ctx, GK_RESID0, k, grid, dim3(32, 8), 0, ctx->hi, ctx->lo, ctx->b0, r, ef, ctx->red, d);
  GC_LAUNCH_CHECK(ctx, "resid0");
  return finalize_to(ctx, (int)nb, GC_S_RNORM2, dec);
}

// One V-cycle of the defect correction: relax L e = r from e = 0 (FP32,
// colour-split), restrict its residual, coarse correction, prolong, relax, then
// phi += e and the new residual r = b0 - L phi with its norm. Expects r (and,
// when pre-smoothing, the first red half-sweep) from the previous residual0.
static int vcycle(gc_ctx *ctx, const gc_mg_params *p, const MgDecide *dec) {
  const int L = ctx->nlev;
  if (L == 0) return GC_OK;
  const bool plain = (p->flags & GC_MG_PLAIN_F32) != 0;
  const int pre = L == 1 ? p->coarse_sweeps : p->pre_sweeps;  // one level: relaxation alone
  const int post = L == 1 ? 0 : p->post_sweeps;
  const LevelGeom &g0 = ctx->lev[0];
  const Split0 d = split0(ctx);
  int st;
  if (p->flags & GC_MG_NATURAL_LAYOUT) {
    // the same cycle with the generic kernels on a natural-layout correction
    const size_t g3 = (size_t)ctx->G * ctx->G * ctx->G;
    GC_CUDA(ctx, cudaMemsetAsync(ctx->e0n, 0, g3 * sizeof(float), ctx->stream));
    for (int h = 0; h < 2 * pre; ++h)
      gc_launch(ctx, GK_SMOOTH0, k_smooth, rb_grid(g0), dim3(RB_TX, RB_TY), 0, ctx->e0n, ctx->r0n, g0, h & 1);
    if (L > 1) {
      gc_launch(ctx, GK_RESIDE, k_resid, node_grid(g0), dim3(32, 8), 0, ctx->e0n, ctx->r0n, ctx->r0, g0);
      gc_launch_after(ctx, GK_RESTRICT, k_restrict, node_grid(ctx->lev[1]), dim3(32, 8), 0, ctx->r0, g0, ctx->b[1],
                ctx->lev[1]);
      GC_LAUNCH_CHECK(ctx, "natural resid/restrict");
      if ((st = coarse_levels(ctx, p))) return st;
      gc_launch(ctx, GK_PROLONG0, k_prolong, node_grid(g0), dim3(32, 8), 0, ctx->e[1], ctx->lev[1], ctx->e0n, g0);
      for (int h = 0; h < 2 * post; ++h)
        gc_launch(ctx, GK_SMOOTH0, k_smooth, rb_grid(g0), dim3(RB_TX, RB_TY), 0, ctx->e0n, ctx->r0n, g0, h & 1);
    }
    if (plain)
      gc_launch(ctx, GK_UPDATE0, k_update0<true, false>, node_grid(g0), dim3(32, 8), 0, (const float *)ctx->e0n,
                ctx->hi, ctx->lo, d);
    else
      gc_launch(ctx, GK_UPDATE0, k_update0<false, false>, node_grid(g0), dim3(32, 8), 0, (const float *)ctx->e0n,
                ctx->hi, ctx->lo, d);
    GC_LAUNCH_CHECK(ctx, "natural cycle");
    return residual0(ctx, p, dec);
  }
  if (finest_blocks(ctx, p)) {
    if ((st = block_down(ctx, GK_SMOOTH0, pre, ctx->e0n, ctx->r0n, g0, ctx->b[1], ctx->lev[1]))) return st;
    if ((st = coarse_levels(ctx, p))) return st;
    st = plain ? block_up<2>(ctx, GK_UPDATE0, post, ctx->e[1], ctx->lev[1], ctx->e0n, ctx->r0n, g0, nullptr)
               : block_up<1>(ctx, GK_UPDATE0, post, ctx->e[1], ctx->lev[1], ctx->e0n, ctx->r0n, g0, nullptr);
    return st ? st : residual0(ctx, p, dec);
  }
  if (finest_planes(ctx, p)) {
    if ((st = fine_down(ctx))) return st;
    if ((st = coarse_levels(ctx, p))) return st;
    st = plain ? fine_up<true>(ctx) : fine_up<false>(ctx);
    return st ? st : residual0(ctx, p, dec);
  }
  const dim3 sg = split_grid(ctx), sg2 = split_grid2(ctx), qg = quad_grid(ctx);
  const bool v4 = vec4(ctx);
  auto half_sweep = [&](int color) {
    if (v4)
      gc_launch_after(ctx, GK_SMOOTH0, k_rb0x2<false>, sg2, SPLIT_BLOCK, 0, ctx->e0s, (const float *)ctx->r0s, d, color);
    else
      gc_launch(ctx, GK_SMOOTH0, k_rb0<false>, sg, SPLIT_BLOCK, 0, ctx->e0s, (const float *)ctx->r0s, d, color);
  };
  if (pre == 0) GC_CUDA(ctx, cudaMemsetAsync(ctx->e0s, 0, 2 * ctx->half0 * sizeof(float), ctx->stream));
  // half-sweep 0 (red, from zero) came with the residual
  for (int h = 1; h < 2 * pre; ++h) half_sweep(h & 1);
  if (L > 1) {
    if (v4)
      gc_launch_after(ctx, GK_RESIDE, k_resid0ex4, qg, dim3(32, 8), 0, (const float *)ctx->e0s, (const float *)ctx->r0s,
                ctx->r0, d);
    else
      gc_launch(ctx, GK_RESIDE, k_resid0e, node_grid(g0), dim3(32, 8), 0, (const float *)ctx->e0s,
                (const float *)ctx->r0s, ctx->r0, d);
    gc_launch_after(ctx, GK_RESTRICT, k_restrict, node_grid(ctx->lev[1]), dim3(32, 8), 0, ctx->r0, g0, ctx->b[1],
              ctx->lev[1]);
    GC_LAUNCH_CHECK(ctx, "resid0e/restrict");
    if ((st = coarse_levels(ctx, p))) return st;
    if (v4 && post >= 1)
      gc_launch_after(ctx, GK_PROLONG0, k_prolong0bx2, sg2, SPLIT_BLOCK, 0, (const float *)ctx->e[1], ctx->lev[1], ctx->e0s,
                g0, d);
    else
      gc_launch(ctx, GK_PROLONG0, k_prolong0s, sg, SPLIT_BLOCK, 0, (const float *)ctx->e[1], ctx->lev[1], ctx->e0s,
                g0, d, post == 0 ? 1 : 0);
    for (int h = 0; h < 2 * post - 1; ++h) half_sweep(h & 1);
  }
  if (post >= 1 && v4) {  // last half-sweep (black) and phi += e in one pass
    if (plain)
      gc_launch_after(ctx, GK_UPDATE0, k_rb0_lastx4<true>, sg2, SPLIT_BLOCK, 0, (const float *)ctx->e0s,
                (const float *)ctx->r0s, ctx->hi, ctx->lo, d);
    else
      gc_launch_after(ctx, GK_UPDATE0, k_rb0_lastx4<false>, sg2, SPLIT_BLOCK, 0, (const float *)ctx->e0s,
                (const float *)ctx->r0s, ctx->hi, ctx->lo, d);
  } else if (post >= 1) {  // last half-sweep (black) and phi += e in one pass
    if (plain)
      gc_launch(ctx, GK_UPDATE0, k_rb0_last<true>, sg, SPLIT_BLOCK, 0, (const float *)ctx->e0s,
                (const float *)ctx->r0s, ctx->hi, ctx->lo, d);
    else
      gc_launch(ctx, GK_UPDATE0, k_rb0_last<false>, sg, SPLIT_BLOCK, 0, (const float *)ctx->e0s,
                (const float *)ctx->r0s, ctx->hi, ctx->lo, d);
  } else {
    if (plain)
      gc_launch(ctx, GK_UPDATE0, k_update0<true, true>, node_grid(g0), dim3(32, 8), 0, (const float *)ctx->e0s,
                ctx->hi, ctx->lo, d);
    else
      gc_launch(ctx, GK_UPDATE0, k_update0<false, true>, node_grid(g0), dim3(32, 8), 0, (const float *)ctx->e0s,
                ctx->hi, ctx->lo, d);
  }
  GC_LAUNCH_CHECK(ctx, "finest cycle");
  return residual0(ctx, p, dec);
}

// One value, with the stopping rule where `dec` asks for it.
static int finalize_one(gc_ctx *ctx, const double *parts, int nparts, double *dst, const MgDecide *dec) {
  MgDecide d = {};
  if (dec) d = *dec;
  if (nparts > 32 * GC_FIN_CHUNKS) {
    double *tmp = ctx->dsmall + GC_S_FIN_TMP;
    gc_launch_after(ctx, GK_REDUCE, k_fin_chunks, dim3(GC_FIN_CHUNKS), dim3(256), 0, parts, nparts, tmp);
    parts = tmp;
    nparts = GC_FIN_CHUNKS;
  }
  gc_launch_after(ctx, GK_REDUCE, k_fin_one, dim3(1), dim3(256), 0, parts, nparts, dst, ctx->dsmall, d);
  GC_LAUNCH_CHECK(ctx, "finalize");
  return GC_OK;
}

int gc_finalize(gc_ctx *ctx, const double *parts, int nparts, int nv, double *dst) {
  GC_REQUIRE(ctx, nv >= 1 && nv <= GC_FIN_NV, "gc_finalize: %d values per row (at most %d)", nv, GC_FIN_NV);
  if (nv == 1) return finalize_one(ctx, parts, nparts, dst, nullptr);
  gc_launch(ctx, GK_REDUCE, k_fin_warps, dim3(1), dim3(32 * nv), 0, parts, nparts, nv, dst);
  GC_LAUNCH_CHECK(ctx, "finalize");
  return GC_OK;
}

static int finalize_to(gc_ctx *ctx, int nparts, int slot, const MgDecide *dec) {
  return finalize_one(ctx, ctx->red, nparts, ctx->dsmall + slot, dec);
}

static int read_small(gc_ctx *ctx, int slot, int count) {
  GC_CUDA(ctx, cudaMemcpyAsync(ctx->hsmall + slot, ctx->dsmall + slot, count * sizeof(double), cudaMemcpyDeviceToHost,
                               ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GC_OK;
}

int gc_faces_from_moments(gc_ctx *ctx) {
  const long long tot = 6LL * ctx->G * ctx->G;
  gc_launch_after(ctx, GK_FACES, k_faces, dim3(gc_blocks(tot, 256)), dim3(256), 0, ctx->hi, ctx->lo, ctx->G, ctx->dx, ctx->grav, ctx->dmom);
  GC_LAUNCH_CHECK(ctx, "faces");
  return GC_OK;
}

// The adaptive loop inside a stream capture: the residual of the initial guess
// with the first decision, then a conditional while node whose body (captured on
// the context's side stream) is one V-cycle and its residual with the next decision.
// Same kernels in the same order as the host loop, so the same potential. The
// cycle count, the converged flag and both norms are left in dsmall and copied
// to the pinned host mirror at the end.
static int mg_run_captured(gc_ctx *ctx, const gc_mg_params *p, int count) {
  int s;
  if (ctx->nlev == 0) return GC_OK;
  cudaStreamCaptureStatus cs;
  cudaGraph_t graph = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  size_t nd = 0;
  GC_CUDA(ctx, cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &graph, &deps, nullptr, &nd));
  GC_REQUIRE(ctx, cs == cudaStreamCaptureStatusActive, "captured solve outside a stream capture");
  cudaGraphConditionalHandle h;
  GC_CUDA(ctx, cudaGraphConditionalHandleCreate(&h, graph, 0, 0));
  MgDecide dec = {h, p->tol, 1, p->min_cycles, p->max_cycles, 1, count};
  if ((s = residual0(ctx, p, &dec))) return s;
  dec.first = 0;
  GC_CUDA(ctx, cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &graph, &deps, nullptr, &nd));
  cudaGraphNodeParams np = {};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = h;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t cond;
  GC_CUDA(ctx, cudaGraphAddNode(&cond, graph, deps, nullptr, nd, &np));
  cudaGraph_t body = np.conditional.phGraph_out[0];
  cudaStream_t main = ctx->stream;
  GC_CUDA(ctx, cudaStreamBeginCaptureToGraph(ctx->side, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  ctx->stream = ctx->side;
  const long long before = gc_launch_total(ctx);
  long long at[GK_COUNT];
  memcpy(at, ctx->prof.launches, sizeof(at));
  s = vcycle(ctx, p, &dec);
  ctx->cap_body_launches = gc_launch_total(ctx) - before;
  for (int k = 0; k < GK_COUNT; ++k) ctx->cap_body[k] = (int)(ctx->prof.launches[k] - at[k]);
  cudaGraph_t got = nullptr;
  const cudaError_t e = cudaStreamEndCapture(ctx->side, &got);
  ctx->stream = main;
  if (s) return s;
  GC_CUDA(ctx, e);
  GC_CUDA(ctx, cudaStreamUpdateCaptureDependencies(main, &cond, nullptr, 1, cudaStreamSetCaptureDependencies));
  GC_CUDA(ctx, cudaMemcpyAsync(ctx->hsmall, ctx->dsmall, GC_S_MIRROR * sizeof(double), cudaMemcpyDeviceToHost, main));
  return GC_OK;
}

// The adaptive loop of an eager solve as a graph of its own: the residual of the guess,
// then the conditional V-cycle loop, then the counts and norms to the pinned mirror: one
// launch and one host wait per solve instead of ten launches and a host read per cycle
// (about 40 us of an idle GPU per cycle: a 64^3 step of 2.2 cycles 356 -> 240 us, a 97^3
// cold solve of 6 cycles 951 -> 776 us). Everything it touches belongs to the context (faces,
// guess and right-hand side are in place before it), so it stays valid while the
// parameters and the reduction scratch stay the same. It is built when the same
// parameters come a second time: a single solve does not pay for it.
static void mg_loop_drop(gc_ctx *ctx) {
  if (ctx->loop_exec) cudaGraphExecDestroy(ctx->loop_exec);
  ctx->loop_exec = nullptr;
}

static bool same_params(const gc_mg_params &a, const gc_mg_params &b) {
  return a.pre_sweeps == b.pre_sweeps && a.post_sweeps == b.post_sweeps && a.coarse_sweeps == b.coarse_sweeps &&
         a.max_cycles == b.max_cycles && a.min_cycles == b.min_cycles && a.flags == b.flags && a.tol == b.tol;
}

static int mg_loop_build(gc_ctx *ctx, const gc_mg_params *p) {
  mg_loop_drop(ctx);
  if (!ctx->side) GC_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking));
  GC_CUDA(ctx, cudaStreamBeginCapture(ctx->cap, cudaStreamCaptureModeRelaxed));
  cudaStream_t main = ctx->stream;  // (it may be the default stream, which cannot be captured)
  long long at[GK_COUNT];
  memcpy(at, ctx->prof.launches, sizeof(at));
  ctx->stream = ctx->cap;
  ctx->capturing = 1;
  const int s = mg_run_captured(ctx, p, 0);
  ctx->capturing = 0;
  ctx->stream = main;
  for (int k = 0; k < GK_COUNT; ++k) {
    ctx->loop_body[k] = ctx->cap_body[k];
    ctx->loop_fixed[k] = (int)(ctx->prof.launches[k] - at[k]) - ctx->cap_body[k];
  }
  memcpy(ctx->prof.launches, at, sizeof(at));  // nothing ran
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(ctx->cap, &g);
  cudaError_t ei = cudaErrorUnknown;
  if (!s && e == cudaSuccess) ei = cudaGraphInstantiate(&ctx->loop_exec, g, 0);
  if (g) cudaGraphDestroy(g);
  if (s || e != cudaSuccess || ei != cudaSuccess) {
    ctx->loop_exec = nullptr;
    cudaGetLastError();
    return s ? s : GC_ERR_CUDA;
  }
  ctx->loop_params = *p;
  ctx->loop_red = ctx->red;
  return GC_OK;
}

// Whether this solve's loop runs as the context's graph (built here when due).
static bool mg_loop_ready(gc_ctx *ctx, const gc_mg_params *p) {
  if (ctx->nlev == 0 || ctx->prof.enabled || ctx->loop_off) return false;
  const bool repeated = ctx->loop_seen && same_params(ctx->loop_last, *p);
  ctx->loop_seen = 1;
  ctx->loop_last = *p;
  if (ctx->loop_exec && ctx->loop_red == ctx->red && same_params(ctx->loop_params, *p)) return true;
  if (!repeated) return false;
  if (mg_loop_build(ctx, p) == GC_OK) return true;
  ctx->loop_off = 1;  // keep the host loop
  return false;
}

void gc_mg_loop_free(gc_ctx *ctx) {
  mg_loop_drop(ctx);
  if (ctx->cap) cudaStreamDestroy(ctx->cap);
  ctx->cap = nullptr;
}

// Adaptive V-cycling (multigrid.py:473-485): at least one cycle, then stop once
// ||r|| < tol ||b|| (never before min_cycles; no test when ||b|| = 0), at most
// max_cycles. Expects b0, faces and the initial interior guess in place and
// ||b0||^2 in dsmall. The residual of the initial guess is formed first; every
// cycle ends with the residual of its result and its norm.
int gc_mg_run(gc_ctx *ctx, const gc_mg_params *p, gc_mg_stats *stats) {
  gc_mg_stats st;
  memset(&st, 0, sizeof(st));
  int s;
  if (ctx->capturing && !(p->flags & GC_MG_FIXED_CYCLES)) {
    if ((s = mg_run_captured(ctx, p, 1))) return s;
    st.cycles = -1;  // decided on the device: read them with gc_pm_graph_stats
    st.converged = -1;
    st.rhs_norm = st.res_norm = NAN;
    ctx->last_stats = st;
    ctx->solved_once = 1;
    if (stats) *stats = st;
    return GC_OK;
  }
  if (!(p->flags & GC_MG_FIXED_CYCLES) && mg_loop_ready(ctx, p)) {
    GC_CUDA(ctx, cudaGraphLaunch(ctx->loop_exec, ctx->stream));
    GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    st.cycles = (int)ctx->hsmall[GC_S_CYCLES];
    st.converged = ctx->hsmall[GC_S_CONVERGED] != 0.0;
    st.rhs_norm = sqrt(ctx->hsmall[GC_S_BNORM2]) / (ctx->dx * ctx->dx);
    st.res_norm = sqrt(ctx->hsmall[GC_S_RNORM2]) / (ctx->dx * ctx->dx);
    for (int k = 0; k < GK_COUNT; ++k)
      ctx->prof.launches[k] += ctx->loop_fixed[k] + (long long)st.cycles * ctx->loop_body[k];
    ctx->last_stats = st;
    ctx->solved_once = 1;
    if (stats) *stats = st;
    return GC_OK;
  }
  if (ctx->nlev > 0 && (s = residual0(ctx, p, nullptr))) return s;
  if (p->flags & GC_MG_FIXED_CYCLES) {
    // exactly max_cycles V-cycles and no host read: the residual norm is left on
    // the device (gc_pm_last_residual reads it), so the solve can be captured in
    // a CUDA graph
    for (int c = 0; c < p->max_cycles && ctx->nlev > 0; ++c)
      if ((s = vcycle(ctx, p, nullptr))) return s;
    // ||b0||^2 and ||r0||^2 (slots 0 and 1) to the pinned host mirror, stream
    // ordered: after a synchronisation the caller reads them without a copy
    GC_CUDA(ctx, cudaMemcpyAsync(ctx->hsmall, ctx->dsmall, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    st.cycles = ctx->nlev > 0 ? p->max_cycles : 0;
    st.converged = -1;
    st.rhs_norm = st.res_norm = NAN;
    ctx->last_stats = st;
    ctx->solved_once = 1;
    if (stats) *stats = st;
    return GC_OK;
  }
  if ((s = read_small(ctx, GC_S_BNORM2, 2))) return s;
  const double bnorm = sqrt(ctx->hsmall[GC_S_BNORM2]);
  const double h2 = ctx->dx * ctx->dx;
  st.rhs_norm = bnorm / h2;
  if (ctx->nlev == 0) {
    st.cycles = 0;
    st.converged = 1;
    st.res_norm = 0.0;
  } else {
    double rnorm = sqrt(ctx->hsmall[GC_S_RNORM2]);
    const int min_c = p->min_cycles > 1 ? p->min_cycles : 1;
    int c = 0;
    for (;;) {
      if (c >= min_c && bnorm > 0.0 && rnorm < p->tol * bnorm) {
        st.converged = 1;
        break;
      }
      if (c >= p->max_cycles) break;
      if ((s = vcycle(ctx, p, nullptr))) return s;
      ++c;
      if ((s = read_small(ctx, GC_S_RNORM2, 1))) return s;
      rnorm = sqrt(ctx->hsmall[GC_S_RNORM2]);
    }
    st.cycles = c;
    st.res_norm = rnorm / h2;
  }
  ctx->last_stats = st;
  ctx->solved_once = 1;
  if (stats) *stats = st;
  return GC_OK;
}

int gc_mg_check_params(gc_ctx *ctx, const gc_mg_params *p) {
  GC_REQUIRE(ctx, p->pre_sweeps >= 0 && p->post_sweeps >= 0 && p->pre_sweeps + p->post_sweeps >= 1,
             "sweep counts must be >= 0 with at least one smoothing sweep");
  GC_REQUIRE(ctx, p->coarse_sweeps >= 1, "coarse_sweeps must be >= 1");
  GC_REQUIRE(ctx, p->max_cycles >= 0 && p->max_cycles <= 100000, "max_cycles out of range");
  GC_REQUIRE(ctx, p->tol >= 0.0, "tol must be >= 0");
  return GC_OK;
}

// Moments of an f32 density into ctx->dmom and, when b0 is given, the right-hand
// side and dsmall[GC_S_BNORM2] (async). Raises GC_FLAG_NONFINITE_RHO.
static int rhs_moments_async(gc_ctx *ctx, const float *rho, float *b0) {
  const long long units = (long long)ctx->G * ((ctx->G + MOM_COLS - 1) / MOM_COLS);
  unsigned nb = gc_blocks(units, 8);
  if (nb > gc_sms() * 2u) nb = gc_sms() * 2u;  // persistent: two CTAs per SM (registers)
  int s = gc_ensure_red(ctx, (size_t)nb * 11);
  if (s) return s;
  // b0 = h^2 * 4 pi G rho (multigrid.py:463)
  gc_launch_after(ctx, b0 ? GK_RHS : GK_MOMENTS, k_rhs_moments, dim3(nb), dim3(256), 0, rho, b0, ctx->G, ctx->dx,
            (float)(4.0 * M_PI * ctx->grav), (float)(ctx->dx * ctx->dx), ctx->red,
            reinterpret_cast<unsigned *>(ctx->dsmall + GC_S_TICKET), ctx->dmom, ctx->dsmall + GC_S_BNORM2,
            ctx->dstatus);
  GC_LAUNCH_CHECK(ctx, "moments");
  return GC_OK;
}

extern "C" int gc_moments(gc_ctx *ctx, const float *rho, double out[10]) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, rho && out, "gc_moments: NULL pointer");
  int s = rhs_moments_async(ctx, rho, nullptr);
  if (s) return s;
  GC_CUDA(ctx, cudaMemcpyAsync(out, ctx->dmom, 10 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  GC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GC_OK;
}

extern "C" int gc_mg_solve(gc_ctx *ctx, const float *rho, float *phi, int warm_start, const gc_mg_params *params,
                           gc_mg_stats *stats) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, rho && phi, "gc_mg_solve: NULL rho or phi");
  gc_mg_params p;
  if (params)
    p = *params;
  else
    gc_mg_default_params(&p);
  int s = gc_mg_check_params(ctx, &p);
  if (s) return s;
  const size_t g3 = (size_t)ctx->G * ctx->G * ctx->G;
  // moments (multigrid.py:364-389), b0 and ||b0||^2 (multigrid.py:477), on the device
  if ((s = rhs_moments_async(ctx, rho, ctx->b0))) return s;
  // initial guess (multigrid.py:464-467): previous phi or zero; the lo part starts at zero
  if (p.flags & GC_MG_FACES_GIVEN) {  // faces (and the guess) from phi
    GC_CUDA(ctx, cudaMemcpyAsync(ctx->hi, phi, g3 * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    if (!warm_start && ctx->nlev > 0) {
      gc_launch(ctx, GK_COPY, k_zero_interior, dim3(node_grid(ctx->lev[0])), dim3(32, 8), 0, ctx->hi, ctx->G);
      GC_LAUNCH_CHECK(ctx, "zero interior");
    }
  } else if (warm_start) {
    GC_CUDA(ctx, cudaMemcpyAsync(ctx->hi, phi, g3 * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
  } else {
    GC_CUDA(ctx, cudaMemsetAsync(ctx->hi, 0, g3 * sizeof(float), ctx->stream));
  }
  GC_CUDA(ctx, cudaMemsetAsync(ctx->lo, 0, g3 * sizeof(float), ctx->stream));
  if (!(p.flags & GC_MG_FACES_GIVEN) && (s = gc_faces_from_moments(ctx))) return s;
  if ((s = gc_mg_run(ctx, &p, stats))) return s;
  // phi = f32(hi + lo) == hi (the pair is normalised)
  GC_CUDA(ctx, cudaMemcpyAsync(phi, ctx->hi, g3 * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
  uint32_t flags = 0;
  if ((s = gc_status(ctx, &flags, 0))) return s;
  if (flags & GC_FLAG_NONFINITE_RHO) {
    gc_set_error(ctx, "rho contains non-finite values");
    return GC_ERR_NONFINITE;
  }
  if (flags & GC_FLAG_TIMEOUT) {
    gc_set_error(ctx, "a bounded device wait of the solve timed out (the potential is incomplete)");
    return GC_ERR_TIMEOUT;
  }
  return GC_OK;
}

extern "C" int gc_mg_residual_norm(gc_ctx *ctx, const float *phi_f32, double *out) {
  if (!ctx) return GC_ERR_ARG;
  GC_REQUIRE(ctx, out, "gc_mg_residual_norm: NULL out");
  if (ctx->nlev == 0) {
    *out = 0.0;
    return GC_OK;
  }
  const LevelGeom &g0 = ctx->lev[0];
  const dim3 grid = node_grid(g0);
  const size_t nb = (size_t)grid.x * grid.y * grid.z;
  int s = gc_ensure_red(ctx, nb);
  if (s) return s;
  if (phi_f32)
    gc_launch(ctx, GK_RESID64, k_resid64, dim3(grid), dim3(dim3(32, 8)), 0, phi_f32, nullptr, ctx->b0, ctx->red, ctx->G);
  else
    gc_launch(ctx, GK_RESID64, k_resid64, dim3(grid), dim3(dim3(32, 8)), 0, ctx->hi, ctx->lo, ctx->b0, ctx->red, ctx->G);
  GC_LAUNCH_CHECK(ctx, "resid64");
  if ((s = finalize_to(ctx, (int)nb, GC_S_RNORM64))) return s;
  if ((s = read_small(ctx, GC_S_RNORM64, 1))) return s;
  *out = sqrt(ctx->hsmall[GC_S_RNORM64]) / (ctx->dx * ctx->dx);
  return GC_OK;
}

extern "C" const float *gc_pm_potential(const gc_ctx *ctx) { return ctx ? ctx->hi : nullptr; }
