// CCD operator for sm_100a: batched 2x2 block-tridiagonal line solves.
//
// Each line (all lines perpendicular to the axis) solves the CCD system of the
// reference (src/twophase/ccd/ccd_solver.py:11-22, coefficients :70-76):
//   Eq-I : a1 (f'_{i-1}+f'_{i+1}) + f'_i - b1 h (f''_{i+1}-f''_{i-1}) = a1/h (f_{i+1}-f_{i-1})
//   Eq-II: b2 (f''_{i-1}+f''_{i+1}) + f''_i - b2/h (f'_{i+1}-f'_{i-1}) = a2/h^2 (f_{i-1}-2f_i+f_{i+1})
// Wall axes fold the one-sided closure into the first/last block rows
// (ccd_solver_helpers.py:227-245); periodic axes are block-circulant
// (ccd_solver_helpers.py:406-423).
//
// Algorithm (this file's own design, not the reference's dense LU):
// the block matrix is the same for every line, so its 2x2 block-LU factors
// (block_tridiag.py:67-104) are computed once on the host.  Lines of up to
// 4 096 rows are solved by the chunk kernels of ccd_chunk.cuh; the kernel below
// takes longer ones.  Every line is cut
// into P chunks of C rows; each chunk runs the forward/backward block-Thomas
// sweeps locally, and the exact coupling between chunks is restored by a short
// scan over the chunk carries (the sweeps are affine first-order recurrences
// whose chunk transfer matrices Phi/Psi are precomputed).  Away from the wall
// rows the factors equal the fixed point of the block Riccati recurrence, so
// only chunk 0 needs per-row tables.  A periodic axis uses the Wiener-Hopf
// factorization A = (I + Lf S^-1) LU (I + H S) of the circulant matrix and
// closes the two recurrences on the ring with (I - T_ring)^-1.
//
// Threads of a CTA: TL consecutive lines x P chunks (lines fastest), so for a
// strided axis the lanes of a warp read consecutive addresses; for the
// contiguous axis the TL lines are staged through shared memory first.
#include "tpf_common.cuh"

#include <cmath>
#include <vector>
#include <array>
#include <algorithm>
#include <type_traits>

namespace {

constexpr double kAlpha1 = 7.0 / 16.0, kA1 = 15.0 / 16.0, kB1 = 1.0 / 16.0;
constexpr double kBeta2 = -1.0 / 8.0, kA2 = 3.0, kB2 = -9.0 / 8.0;

using M2 = std::array<double, 4>;  // row-major 2x2
inline M2 mul(const M2& a, const M2& b) {
  return {a[0] * b[0] + a[1] * b[2], a[0] * b[1] + a[1] * b[3],
          a[2] * b[0] + a[3] * b[2], a[2] * b[1] + a[3] * b[3]};
}
inline M2 sub(const M2& a, const M2& b) { return {a[0] - b[0], a[1] - b[1], a[2] - b[2], a[3] - b[3]}; }
inline M2 add(const M2& a, const M2& b) { return {a[0] + b[0], a[1] + b[1], a[2] + b[2], a[3] + b[3]}; }
inline M2 neg(const M2& a) { return {-a[0], -a[1], -a[2], -a[3]}; }
inline double det(const M2& a) { return a[0] * a[3] - a[1] * a[2]; }
inline M2 inv(const M2& a) {
  double d = det(a), id = 1.0 / d;
  return {a[3] * id, -a[1] * id, -a[2] * id, a[0] * id};
}
inline M2 eye() { return {1.0, 0.0, 0.0, 1.0}; }
inline double maxabs(const M2& a) {
  return std::max(std::max(std::fabs(a[0]), std::fabs(a[1])), std::max(std::fabs(a[2]), std::fabs(a[3])));
}

// ---- chunk kernels (ccd_chunk.cuh) ----
constexpr int kChunkWindow = 4;
constexpr int kChunkHead = 48;   // 0.455^48 = 4e-17
constexpr int kChunkR = 16;

// constants of a plan for chunks of R rows, in the compute type
template <typename T, int R>
struct ChunkConst {
  T A[4], AR[4], B[4], BR[4];     // A (scaled) and B, and their R-th powers
  T P[4], Z[4];                   // P (scaled), P_last P^-1
  T Gf[4], Gb[4], AL[4], BL[4];   // periodic: ring closures, A and B to the power of the last chunk's rows
  // walls, in FP64 for FP32 too: the closures are evaluated in it
  double cl[4], cr[4];            // closure -> first right-hand side (scaled) / last solution
  double Ml[4], Mr[4], cIl[4], cIr[4], cII[6];
};

// Table layout (doubles).  C = chunk length, H0 = rows [0, H0) of the wall
// "head" that carry per-row factors (the block-LU factors only reach the
// fixed point ~30 rows away from the wall closure).
struct TabLayout {
  int C, H0;
  __host__ __device__ int head() const { return 0; }                // H0 x 20: Lf P H PhiH PsiH
  __host__ __device__ int phi() const { return 20 * H0; }           // C x 4
  __host__ __device__ int psi() const { return 20 * H0 + 4 * C; }   // (C+1) x 4
  __host__ __device__ int cst() const { return 20 * H0 + 8 * C + 4; }  // Lfi Pi Hi Plast Gf Gb
  __host__ __device__ int bc() const { return cst() + 24; }         // L0 UN Ml Mr cIl cIr cII(6) c1 c2
  __host__ __device__ int total() const { return bc() + 32; }
};

}  // namespace

struct tpf_ccd_plan {
  int64_t n_pts = 0;
  double h = 0.0;
  int bc = TPF_BC_WALL;
  int dtype = TPF_F64;
  int n_rows = 0, C = 32, P = 1, H0 = 0;
  double* d_tab = nullptr;   // double table
  float* d_tabf = nullptr;   // float copy (interior factors for F32)
  double* d_J = nullptr;     // metric J, dJ (n_pts each)
  bool has_metric = false;
  // constants of the chunk kernels, and their wall tables G [kChunkHead + kChunkR][4]
  ChunkConst<double, kChunkR> c64;
  ChunkConst<float, kChunkR> c32;
  double* d_g64 = nullptr;
  float* d_g32 = nullptr;
  // FP32 per-row block-LU factors of the folded wall system (Lf, P, H per
  // row) for the iterative-refinement correction solves, built on first use
  mutable float* d_rfac = nullptr;
};

namespace {

struct CcdArgs {
  const void* f;
  void* d1;
  void* d2;
  int64_t outer, inner, n_lines;
  int n, n_rows, C, P, H0, TL, tl_shift;
  int tl_inv;             // floor(2^16 / TL) + 1: x tl_inv >> 16 is x / TL for x <= 1024, TL <= 32
  int LS, FS;             // ybuf line stride / staged-f line stride (elements)
  int nbuf;               // f tile buffers (1 or 2)
  int n_tiles;
  int tab_total;
  const double* tab;      // double table (closures)
  const void* tabT;       // table in compute type
  const double* J;        // metric (J[0..n), dJ[n..2n)) or nullptr
  int ovl, ovr;           // wall closure overrides (left / right)
  double bcl0, bcl1, bcr0, bcr1;
  // variable-density epilogue: out (+)= d2/rho - (drho/rho^2) d1 instead of d1, d2
  const void* vd_rho;
  const void* vd_drho;
  void* vd_out;
  int vd_accumulate;
  // velocity-corrector epilogue: out = u* - (dt / rho) d1 instead of d1, d2;
  // on wall planes (first / last node of a line) d1 counts as 0, so out = u*
  const void* cr_u;
  const void* cr_rho;
  void* cr_out;
  double cr_dt;
  int cr_wall;
};

template <typename T>
struct V2 { T a, b; };

// Write one node's result: either (d1, d2) or the variable-density term.
template <typename T>
__device__ __forceinline__ void store_out(const CcdArgs& a, int64_t gi, double o1, double o2, int k) {
  if (a.cr_out) {
    // u_new = u* - (dt / rho) dp/dx, with the reference's operation order
    // (quotient, product, difference; no fused multiply-add).  The loads are
    // read-only-path loads so that they need not wait for earlier nodes'
    // stores: every address is read once, by the lane that later writes it
    // (u_out may be u_star), so no stale value can be read.
    const double u = (double)__ldg(static_cast<const T*>(a.cr_u) + gi);
    double v = u;
    if (!(a.cr_wall && (k == 0 || k == a.n - 1))) {   // k: node along the line
      const double q = a.cr_dt / (double)__ldg(static_cast<const T*>(a.cr_rho) + gi);
      v = __dsub_rn(u, __dmul_rn(q, o1));
    }
    static_cast<T*>(a.cr_out)[gi] = (T)v;
    return;
  }
  if (a.vd_out) {
    const double r = (double)static_cast<const T*>(a.vd_rho)[gi];
    const double dr = (double)static_cast<const T*>(a.vd_drho)[gi];
    double t = o2 / r - (dr / (r * r)) * o1;
    T* out = static_cast<T*>(a.vd_out);
    if (a.vd_accumulate) t = (double)out[gi] + t;
    out[gi] = (T)t;
    return;
  }
  if (a.d1) static_cast<T*>(a.d1)[gi] = (T)o1;
  if (a.d2) static_cast<T*>(a.d2)[gi] = (T)o2;
}

template <typename T>
__device__ __forceinline__ V2<T> mv(const T* m, V2<T> v) {
  return {m[0] * v.a + m[1] * v.b, m[2] * v.a + m[3] * v.b};
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool valid) {
  unsigned int sa = (unsigned int)__cvta_generic_to_shared(smem);
  int src = valid ? BYTES : 0;   // src-size 0 -> zero fill
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(sa), "l"(gmem), "n"(BYTES), "r"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Stage a read-only table into shared memory with asynchronous copies: every
// thread issues its share and waits once, so the copy costs one global round
// trip rather than one per element a thread copies (a block of one warp and a
// 700-entry table otherwise spends ~10 us here, longer than a small field's
// whole solve).  Called before any other asynchronous copy of the block.
template <typename T>
__device__ __forceinline__ void stage_table(T* dst, const T* src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) cp_async<sizeof(T)>(dst + i, src + i, true);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
}

// Issue the asynchronous copy of tile `t` (TL lines x n points) into fb.
// Strided axis: fb[k*TL + l]; contiguous axis: fb[l*FS + k].  lb receives the
// global base offset of each line (strided) for the output pass.
template <typename T, bool CONTIG>
__device__ __forceinline__ void issue_tile(const CcdArgs& a, const T* __restrict__ f, T* fb, long long* lb, int t) {
  const int TL = a.TL, n = a.n;
  const int64_t line0 = (int64_t)t * TL;
  if (CONTIG) {
    const int64_t nl = min((int64_t)TL, a.n_lines - line0);
    const T* src = f + line0 * n;
    const int total = TL * n;
    int l = threadIdx.x / n, k = threadIdx.x - (threadIdx.x / n) * n;
    const int step_l = blockDim.x / n, step_k = blockDim.x - step_l * n;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const bool v = l < nl;
      cp_async<sizeof(T)>(fb + l * a.FS + k, v ? src + e : f, v);
      l += step_l;
      k += step_k;
      if (k >= n) { k -= n; ++l; }
    }
  } else {
    if (threadIdx.x < TL) {
      const int64_t line = line0 + threadIdx.x;
      long long b = -1;
      if (line < a.n_lines) {
        const int64_t o = line / a.inner, i = line - o * a.inner;
        b = o * (int64_t)n * a.inner + i;
      }
      lb[threadIdx.x] = b;
    }
    __syncthreads();
    const int total = TL * n;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int k = e >> a.tl_shift, l = e & (TL - 1);
      const long long b = lb[l];
      cp_async<sizeof(T)>(fb + e, b >= 0 ? f + b + (int64_t)k * a.inner : f, b >= 0);
    }
  }
  cp_async_commit();
}

template <typename T, bool PERIODIC, bool CONTIG>
__global__ void __launch_bounds__(512, 1) ccd_line_kernel(CcdArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int TL = a.TL, C = a.C, P = a.P, n = a.n, n_rows = a.n_rows, H0 = a.H0;
  const TabLayout lay{C, H0};
  const int fsz = CONTIG ? TL * a.FS : TL * n;
  // shared layout: bcs(double) | lbase(2 x TL) | tab(T) | ybuf | fbuf[nbuf] | cin | cinb
  double* bcs = reinterpret_cast<double*>(smem_raw);
  long long* lbase = reinterpret_cast<long long*>(bcs + 4 * TL);
  T* tab = reinterpret_cast<T*>(lbase + 2 * TL);
  T* ybuf = tab + ((a.tab_total + 1) & ~1);
  T* fbuf = ybuf + (((size_t)TL * a.LS + 1) & ~(size_t)1);
  T* cin = fbuf + (size_t)a.nbuf * fsz;
  T* cinb = cin + (size_t)P * TL * 2;

  const T* __restrict__ f = static_cast<const T*>(a.f);
  const T* tabT = static_cast<const T*>(a.tabT);
  stage_table<T>(tab, tabT, a.tab_total);   // the table is read below (c1, c2) and in every phase

  const int tid = threadIdx.x;
  const int l = tid & (TL - 1), c = tid >> a.tl_shift;
  const int j0 = c * C;
  const int j1 = min(j0 + C, n_rows);
  const T c1 = tab[lay.bc() + 30], c2 = tab[lay.bc() + 31];
  const T* Lfi = tab + lay.cst();
  const T* Pi = Lfi + 4;
  const T* Hi = Lfi + 8;
  const T* Plast = Lfi + 12;
  const T* Phi = tab + lay.phi();
  const T* Psi = tab + lay.psi();
  const T* head = tab + lay.head();
  const double* tb = a.tab + lay.bc();
  const double* J = a.J;
  T* yl = ybuf + (size_t)l * a.LS;
  T* cinl = cin + (size_t)l * P * 2;
  T* cinbl = cinb + (size_t)l * P * 2;

  int t = blockIdx.x;
  int buf = 0;
  if (t < a.n_tiles) issue_tile<T, CONTIG>(a, f, fbuf, lbase, t);
  for (; t < a.n_tiles; t += gridDim.x) {
    const int tn = t + gridDim.x;
    if (a.nbuf == 2 && tn < a.n_tiles) {
      issue_tile<T, CONTIG>(a, f, fbuf + (size_t)(buf ^ 1) * fsz, lbase + (buf ^ 1) * TL, tn);
      cp_async_wait<1>();
    } else {
      // single buffer: this tile's copy is issued here (the first one in the prologue)
      if (a.nbuf == 1 && t != (int)blockIdx.x) issue_tile<T, CONTIG>(a, f, fbuf, lbase, t);
      cp_async_wait<0>();
    }
    __syncthreads();
    const T* fb = fbuf + (size_t)buf * fsz;
    const long long* lb = lbase + buf * TL;
    const int64_t line0 = (int64_t)t * TL;
    const bool valid = CONTIG ? (line0 + l < a.n_lines) : (lb[l] >= 0);
    auto F = [&](int k) -> T { return CONTIG ? fb[l * a.FS + k] : fb[k * TL + l]; };

    // ---- wall closures (FP64) ---------------------------------------------
    if (!PERIODIC) {
      if (c == 0) {
        double r0, r1;
        if (a.ovl) { r0 = a.bcl0; r1 = a.bcl1; }
        else {
          double fv[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) fv[k] = (double)F(k);
          r0 = tb[16] * fv[0] + tb[17] * fv[1] + tb[18] * fv[2] + tb[19] * fv[3];
          r1 = tb[24] * fv[0] + tb[25] * fv[1] + tb[26] * fv[2] + tb[27] * fv[3] + tb[28] * fv[4] + tb[29] * fv[5];
        }
        bcs[l * 4 + 0] = r0;
        bcs[l * 4 + 1] = r1;
      }
      if (c == P - 1) {
        double r0, r1;
        if (a.ovr) { r0 = a.bcr0; r1 = a.bcr1; }
        else {
          double fv[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) fv[k] = (double)F(n - 1 - k);
          r0 = tb[20] * fv[0] + tb[21] * fv[1] + tb[22] * fv[2] + tb[23] * fv[3];
          r1 = tb[24] * fv[0] + tb[25] * fv[1] + tb[26] * fv[2] + tb[27] * fv[3] + tb[28] * fv[4] + tb[29] * fv[5];
        }
        bcs[l * 4 + 2] = r0;
        bcs[l * 4 + 3] = r1;
      }
      __syncthreads();
    }

    // ---- forward local sweep: y_j = b_j - Lf_j y_{j-1}, zero carry-in --------
    {
      const int Nn = n - 1;
      const int off = PERIODIC ? 0 : 1;
      auto node = [&](int k) -> int {
        if (PERIODIC) { if (k < 0) return k + Nn; if (k >= Nn) return k - Nn; }
        return k;
      };
      T fm = T(0), f0 = T(0);
      if (j0 < j1) {
        fm = F(node(j0 + off - 1));
        f0 = F(node(j0 + off));
      }
      V2<T> y{T(0), T(0)};
      for (int j = j0; j < j1; ++j) {
        const T fp = F(node(j + off + 1));
        V2<T> b{c1 * (fp - fm), c2 * ((fm - T(2) * f0) + fp)};
        if (!PERIODIC) {
          if (j == 0) {
            const double l0 = bcs[l * 4 + 0], l1 = bcs[l * 4 + 1];
            b.a = (T)((double)b.a - (tb[0] * l0 + tb[1] * l1));
            b.b = (T)((double)b.b - (tb[2] * l0 + tb[3] * l1));
          }
          if (j == n_rows - 1) {
            const double r0 = bcs[l * 4 + 2], r1 = bcs[l * 4 + 3];
            b.a = (T)((double)b.a - (tb[4] * r0 + tb[5] * r1));
            b.b = (T)((double)b.b - (tb[6] * r0 + tb[7] * r1));
          }
        }
        if (j == j0) {
          y = b;
        } else {
          const T* Lf = (!PERIODIC && j < H0) ? head + 20 * j : Lfi;
          const V2<T> q = mv(Lf, y);
          y = {b.a - q.a, b.b - q.b};
        }
        yl[2 * j] = y.a;
        yl[2 * j + 1] = y.b;
        fm = f0;
        f0 = fp;
      }
    }
    __syncthreads();

    // ---- forward carry scan (one thread per line) ---------------------------
    if (c == 0) {
      auto Tc = [&](int s, int e) -> const T* {
        return (!PERIODIC && e - 1 < H0) ? head + 20 * (e - 1) + 12 : Phi + 4 * (e - s - 1);
      };
      if (!PERIODIC) {
        const int e0 = min(C, n_rows) - 1;
        V2<T> Y{yl[2 * e0], yl[2 * e0 + 1]};
        for (int cc = 1; cc < P; ++cc) {
          cinl[2 * cc] = Y.a;
          cinl[2 * cc + 1] = Y.b;
          const int s = cc * C, e = min(s + C, n_rows);
          const V2<T> q = mv(Tc(s, e), Y);
          Y = {yl[2 * (e - 1)] + q.a, yl[2 * (e - 1) + 1] + q.b};
        }
      } else {
        V2<T> Y{T(0), T(0)};
        for (int cc = 0; cc < P; ++cc) {
          const int s = cc * C, e = min(s + C, n_rows);
          const V2<T> q = mv(Tc(s, e), Y);
          Y = {yl[2 * (e - 1)] + q.a, yl[2 * (e - 1) + 1] + q.b};
        }
        Y = mv(Lfi + 16, Y);  // Gf = (I - T_ring)^-1
        for (int cc = 0; cc < P; ++cc) {
          cinl[2 * cc] = Y.a;
          cinl[2 * cc + 1] = Y.b;
          const int s = cc * C, e = min(s + C, n_rows);
          const V2<T> q = mv(Tc(s, e), Y);
          Y = {yl[2 * (e - 1)] + q.a, yl[2 * (e - 1) + 1] + q.b};
        }
      }
    }
    __syncthreads();

    // ---- forward fix-up + backward local sweep -------------------------------
    {
      if (PERIODIC || c > 0) {
        const V2<T> Yin{cinl[2 * c], cinl[2 * c + 1]};
        for (int j = j0; j < j1; ++j) {
          const T* m = (!PERIODIC && j < H0) ? head + 20 * j + 12 : Phi + 4 * (j - j0);
          const V2<T> q = mv(m, Yin);
          yl[2 * j] += q.a;
          yl[2 * j + 1] += q.b;
        }
      }
      V2<T> xn{T(0), T(0)};
      for (int j = j1 - 1; j >= j0; --j) {
        const V2<T> y{yl[2 * j], yl[2 * j + 1]};
        V2<T> x;
        if (!PERIODIC && j < H0) {
          const V2<T> p = mv(head + 20 * j + 4, y);
          const V2<T> q = mv(head + 20 * j + 8, xn);
          x = {p.a - q.a, p.b - q.b};
        } else if (!PERIODIC && j == n_rows - 1) {
          x = mv(Plast, y);
        } else {
          const V2<T> p = mv(Pi, y);
          const V2<T> q = mv(Hi, xn);
          x = {p.a - q.a, p.b - q.b};
        }
        yl[2 * j] = x.a;
        yl[2 * j + 1] = x.b;
        xn = x;
      }
    }
    __syncthreads();

    // ---- backward carry scan -------------------------------------------------
    if (c == 0) {
      auto Rc = [&](int s, int e) -> const T* {
        return (!PERIODIC && s < H0) ? head + 20 * s + 16 : Psi + 4 * (e - s);
      };
      if (!PERIODIC) {
        const int s = (P - 1) * C;
        V2<T> X{yl[2 * s], yl[2 * s + 1]};
        for (int cc = P - 2; cc >= 0; --cc) {
          cinbl[2 * cc] = X.a;
          cinbl[2 * cc + 1] = X.b;
          if (cc >= 1) {
            const int s2 = cc * C, e2 = min(s2 + C, n_rows);
            const V2<T> q = mv(Rc(s2, e2), X);
            X = {yl[2 * s2] + q.a, yl[2 * s2 + 1] + q.b};
          }
        }
      } else {
        V2<T> X{T(0), T(0)};
        for (int cc = P - 1; cc >= 0; --cc) {
          const int s = cc * C, e = min(s + C, n_rows);
          const V2<T> q = mv(Rc(s, e), X);
          X = {yl[2 * s] + q.a, yl[2 * s + 1] + q.b};
        }
        X = mv(Lfi + 20, X);  // Gb = (I - R_ring)^-1
        for (int cc = P - 1; cc >= 0; --cc) {
          cinbl[2 * cc] = X.a;
          cinbl[2 * cc + 1] = X.b;
          const int s = cc * C, e = min(s + C, n_rows);
          const V2<T> q = mv(Rc(s, e), X);
          X = {yl[2 * s] + q.a, yl[2 * s + 1] + q.b};
        }
      }
    }
    __syncthreads();

    // ---- backward fix-up (+ direct output for strided axes) ----------------
    {
      const bool has_cin = PERIODIC || c < P - 1;
      V2<T> Xin{T(0), T(0)};
      if (has_cin) { Xin.a = cinbl[2 * c]; Xin.b = cinbl[2 * c + 1]; }
      const long long base = CONTIG ? 0 : lb[l];
      for (int j = j0; j < j1; ++j) {
        V2<T> x{yl[2 * j], yl[2 * j + 1]};
        if (has_cin) {
          const T* m = (!PERIODIC && j < H0) ? head + 20 * j + 16 : Psi + 4 * (j1 - j);
          const V2<T> q = mv(m, Xin);
          x.a += q.a;
          x.b += q.b;
          yl[2 * j] = x.a;
          yl[2 * j + 1] = x.b;
        }
        if (!CONTIG && valid) {
          const int k = PERIODIC ? j : j + 1;
          double o1 = (double)x.a, o2 = (double)x.b;
          if (J) {
            const double Jk = J[k], dJk = J[n + k];
            o2 = Jk * Jk * o2 + Jk * dJk * o1;
            o1 = Jk * o1;
          }
          store_out<T>(a, base + (int64_t)k * a.inner, o1, o2, k);
        }
      }
    }
    __syncthreads();

    // ---- boundary nodes / contiguous-axis output ------------------------------
    auto boundary_pair = [&](int ll, bool left, double& o1, double& o2) {
      const T* yy = ybuf + (size_t)ll * a.LS;
      if (left) {
        const double x0 = (double)yy[0], x1 = (double)yy[1];
        o1 = (tb[8] * x0 + tb[9] * x1) + bcs[ll * 4 + 0];
        o2 = (tb[10] * x0 + tb[11] * x1) + bcs[ll * 4 + 1];
      } else {
        const int jl = n_rows - 1;
        const double x0 = (double)yy[2 * jl], x1 = (double)yy[2 * jl + 1];
        o1 = (tb[12] * x0 + tb[13] * x1) + bcs[ll * 4 + 2];
        o2 = (tb[14] * x0 + tb[15] * x1) + bcs[ll * 4 + 3];
      }
    };
    auto metric = [&](int k, double& o1, double& o2) {
      if (J) {
        const double Jk = J[k], dJk = J[n + k];
        const double t1 = Jk * o1;
        o2 = Jk * Jk * o2 + Jk * dJk * o1;
        o1 = t1;
      }
    };
    if (!CONTIG) {
      if (valid) {
        const long long base = lb[l];
        if (!PERIODIC) {
          if (c == 0) {
            double o1, o2;
            boundary_pair(l, true, o1, o2);
            metric(0, o1, o2);
            store_out<T>(a, base, o1, o2, 0);
          }
          if (c == P - 1) {
            double o1, o2;
            boundary_pair(l, false, o1, o2);
            metric(n - 1, o1, o2);
            store_out<T>(a, base + (int64_t)(n - 1) * a.inner, o1, o2, n - 1);
          }
        } else if (c == 0) {
          double o1 = (double)yl[0], o2 = (double)yl[1];
          metric(n - 1, o1, o2);
          store_out<T>(a, base + (int64_t)(n - 1) * a.inner, o1, o2, n - 1);
        }
      }
    } else {
      const int64_t nl = min((int64_t)TL, a.n_lines - line0);
      const int cnt = (int)nl * n;
      int ll = tid / n, k = tid - (tid / n) * n;
      const int step_l = blockDim.x / n, step_k = blockDim.x - step_l * n;
      for (int e = tid; e < cnt; e += blockDim.x) {
        const T* yy = ybuf + (size_t)ll * a.LS;
        double o1, o2;
        if (!PERIODIC) {
          if (k == 0) boundary_pair(ll, true, o1, o2);
          else if (k == n - 1) boundary_pair(ll, false, o1, o2);
          else { o1 = (double)yy[2 * (k - 1)]; o2 = (double)yy[2 * (k - 1) + 1]; }
        } else {
          const int kk = (k == n - 1) ? 0 : k;
          o1 = (double)yy[2 * kk];
          o2 = (double)yy[2 * kk + 1];
        }
        if (J) metric(k, o1, o2);
        store_out<T>(a, line0 * n + e, o1, o2, k);
        ll += step_l;
        k += step_k;
        if (k >= n) { k -= n; ++ll; }
      }
    }
    __syncthreads();
    buf ^= (a.nbuf == 2) ? 1 : 0;
  }
  cp_async_wait<0>();
}

template <typename T>
__global__ void wall_zero_kernel(T* g, int64_t outer, int64_t n, int64_t inner) {
  int64_t tot = outer * inner * 2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t side = e / (outer * inner), r = e % (outer * inner);
    int64_t o = r / inner, i = r % inner;
    int64_t k = side ? n - 1 : 0;
    g[o * n * inner + k * inner + i] = T(0);
  }
}

}  // namespace

#include "ccd_chunk.cuh"

namespace {

// ---- host: factor tables ---------------------------------------------------

template <typename T, int R>
ChunkConst<T, R> cast_chunk(const ChunkConst<double, R>& d) {
  ChunkConst<T, R> o;
  auto cp = [](const double* a, T* b, int n) { for (int k = 0; k < n; ++k) b[k] = (T)a[k]; };
  cp(d.A, o.A, 4); cp(d.AR, o.AR, 4); cp(d.B, o.B, 4); cp(d.BR, o.BR, 4);
  cp(d.P, o.P, 4); cp(d.Z, o.Z, 4); cp(d.Gf, o.Gf, 4); cp(d.Gb, o.Gb, 4); cp(d.AL, o.AL, 4); cp(d.BL, o.BL, 4);
  std::copy(d.cl, d.cl + 4, o.cl); std::copy(d.cr, d.cr + 4, o.cr);
  std::copy(d.Ml, d.Ml + 4, o.Ml); std::copy(d.Mr, d.Mr + 4, o.Mr);
  std::copy(d.cIl, d.cIl + 4, o.cIl); std::copy(d.cIr, d.cIr + 4, o.cIr); std::copy(d.cII, d.cII + 6, o.cII);
  return o;
}

// constants of the chunk kernels (see ccd_chunk.cuh); G: the wall table, rows
// beyond kChunkHead or beyond the line are 0
template <int R>
ChunkConst<double, R> chunk_tables(const tpf_ccd_plan* p, std::vector<double>& G) {
  const double h = p->h;
  const int n_rows = p->n_rows;
  const M2 L = {kAlpha1, kB1 * h, kB2 / h, kBeta2};
  const M2 U = {kAlpha1, -kB1 * h, -kB2 / h, kBeta2};
  const M2 Ml = {-1.5, 1.5 * h, 0.0, 0.0};
  const M2 Mr = {-1.5, -1.5 * h, 0.0, 0.0};
  M2 S = eye();   // fixed point of S = I - L S^-1 U
  for (int it = 0; it < 400; ++it) S = sub(eye(), mul(mul(L, inv(S)), U));
  const M2 P = inv(S), A = neg(mul(L, P)), B = neg(mul(P, U));
  const double d[2] = {kA1 / h, kA2 / (h * h)};
  auto sim = [&](const M2& m) { return M2{m[0], m[1] * d[1] / d[0], m[2] * d[0] / d[1], m[3]}; };   // D^-1 m D
  auto rmul = [&](const M2& m) { return M2{m[0] * d[0], m[1] * d[1], m[2] * d[0], m[3] * d[1]}; };  // m D
  ChunkConst<double, R> K{};
  G.assign(4 * (kChunkHead + R), 0.0);
  auto set = [](double* o, const M2& m) { for (int k = 0; k < 4; ++k) o[k] = m[k]; };
  M2 pa = eye(), pb = eye();
  for (int r = 0; r < R; ++r) {
    pa = mul(A, pa);
    pb = mul(B, pb);
  }
  set(K.A, sim(A));
  set(K.AR, sim(pa));
  set(K.B, B);
  set(K.BR, pb);
  set(K.P, rmul(P));
  set(K.Ml, Ml);
  set(K.Mr, Mr);
  const double cIl[4] = {-23.0 / 6.0, 21.0 / 4.0, -1.5, 1.0 / 12.0};
  const double cII[6] = {45.0, -154.0, 214.0, -156.0, 61.0, -10.0};
  for (int q = 0; q < 4; ++q) {
    K.cIl[q] = cIl[q] / h;
    K.cIr[q] = -cIl[q] / h;
  }
  for (int q = 0; q < 6; ++q) K.cII[q] = cII[q] / (12.0 * h * h);
  set(K.cl, {L[0] / d[0], L[1] / d[0], L[2] / d[1], L[3] / d[1]});
  if (p->bc == TPF_BC_WALL) {
    // the last pivot, and M^-1 e_0 by the two sweeps
    const M2 Sl = add(sub(eye(), mul(neg(A), U)), mul(U, Mr)), Pl = inv(Sl);
    set(K.Z, mul(Pl, S));
    set(K.cr, mul(Pl, U));
    std::vector<M2> V(n_rows);
    M2 y = eye();
    for (int j = 0; j < n_rows; ++j) {
      V[j] = y;
      y = mul(A, y);
    }
    V[n_rows - 1] = mul(Pl, V[n_rows - 1]);
    for (int j = n_rows - 2; j >= 0; --j) V[j] = add(mul(P, V[j]), mul(B, V[j + 1]));
    const M2 B0 = sub(add(eye(), mul(L, Ml)), S);
    const M2 Kg = mul(B0, inv(add(eye(), mul(V[0], B0))));
    for (int j = 0; j < std::min(n_rows, kChunkHead); ++j) set(G.data() + 4 * j, mul(V[j], Kg));
  } else {
    const int Q = (n_rows + R - 1) / R, len = n_rows - (Q - 1) * R;
    M2 an = eye(), bn = eye(), al = eye(), bl = eye();
    for (int k = 0; k < n_rows; ++k) {
      an = mul(A, an);
      bn = mul(B, bn);
      if (k == len - 1) {
        al = an;
        bl = bn;
      }
    }
    set(K.Gf, sim(inv(sub(eye(), an))));
    set(K.Gb, inv(sub(eye(), bn)));
    set(K.AL, sim(al));
    set(K.BL, bl);
  }
  return K;
}

int build_tables(tpf_ccd_plan* p, std::vector<double>& tab) {
  const double h = p->h;
  const int n_rows = p->n_rows;
  const int C = p->C;
  const M2 L = {kAlpha1, kB1 * h, kB2 / h, kBeta2};
  const M2 U = {kAlpha1, -kB1 * h, -kB2 / h, kBeta2};
  const M2 Ml = {-1.5, 1.5 * h, 0.0, 0.0};
  const M2 Mr = {-1.5, -1.5 * h, 0.0, 0.0};
  // fixed point of LU = I - L LU^-1 U (interior block-LU factor)
  M2 LUi = eye();
  for (int it = 0; it < 400; ++it) LUi = sub(eye(), mul(mul(L, inv(LUi)), U));
  const M2 Pinf = inv(LUi), Lfinf = mul(L, Pinf), Hinf = mul(Pinf, U);
  const int P = (n_rows + C - 1) / C;
  int H0 = 0;
  std::vector<M2> Lf, Pm, Hm;
  if (p->bc == TPF_BC_WALL) {
    // per-row factors of the folded system (ccd_solver_helpers.py:238-245)
    std::vector<M2> LU(n_rows);
    Lf.resize(n_rows); Pm.resize(n_rows); Hm.resize(n_rows);
    for (int j = 0; j < n_rows; ++j) {
      M2 D = eye();
      if (j == 0) D = add(D, mul(L, Ml));
      if (j == n_rows - 1) D = add(D, mul(U, Mr));
      if (j == 0) {
        LU[j] = D;
        Lf[j] = {0, 0, 0, 0};
      } else {
        Lf[j] = mul(L, inv(LU[j - 1]));
        LU[j] = sub(D, mul(Lf[j], U));
      }
      const double dt = det(LU[j]);
      if (!std::isfinite(dt) || std::fabs(dt) < 1e-300) {
        tpf::set_error("CCD block-tridiagonal factorization encountered a singular pivot at block %d", j);
        return TPF_ESINGULAR;
      }
      Pm[j] = inv(LU[j]);
      Hm[j] = (j < n_rows - 1) ? mul(Pm[j], U) : M2{0, 0, 0, 0};
    }
    // smallest head (a multiple of C) beyond which the factors sit at the fixed point
    H0 = n_rows;
    for (int hh = C; hh < n_rows; hh += C) {
      // rows >= hh use the fixed-point Lf (all rows, the last included) and
      // the fixed-point P, H (all but the last, which carries the closure)
      bool conv = true;
      for (int j = hh; j < n_rows && conv; ++j) {
        double e = maxabs(sub(Lf[j], Lfinf)) / maxabs(Lfinf);
        if (j < n_rows - 1)
          e = std::max(e, std::max(maxabs(sub(Pm[j], Pinf)) / maxabs(Pinf), maxabs(sub(Hm[j], Hinf)) / maxabs(Hinf)));
        conv = e < 1e-15;
      }
      if (conv) { H0 = hh; break; }
    }
  }
  TabLayout lay{C, H0};
  tab.assign(lay.total(), 0.0);
  // Phi_k = (-Lf)^(k+1), Psi_k = (-H)^k in the fixed-point region
  M2 acc = eye();
  for (int k = 0; k < C; ++k) {
    acc = mul(neg(Lfinf), acc);
    for (int q = 0; q < 4; ++q) tab[lay.phi() + 4 * k + q] = acc[q];
  }
  acc = eye();
  for (int k = 0; k <= C; ++k) {
    for (int q = 0; q < 4; ++q) tab[lay.psi() + 4 * k + q] = acc[q];
    acc = mul(neg(Hinf), acc);
  }
  for (int q = 0; q < 4; ++q) {
    tab[lay.cst() + q] = Lfinf[q];
    tab[lay.cst() + 4 + q] = Pinf[q];
    tab[lay.cst() + 8 + q] = Hinf[q];
  }
  if (p->bc == TPF_BC_WALL) {
    for (int q = 0; q < 4; ++q) tab[lay.cst() + 12 + q] = Pm[n_rows - 1][q];
    // head rows: Lf, P, H and the chunk-relative transfer products
    //   PhiH_j = prod_{m=s..j} (-Lf_m),  PsiH_j = prod_{m=j..e-1} (-H_m)
    for (int cc = 0; cc * C < H0; ++cc) {
      const int s = cc * C, e = std::min(s + C, n_rows);
      M2 ph = eye();
      for (int j = s; j < e; ++j) {
        ph = mul(neg(Lf[j]), ph);
        for (int q = 0; q < 4; ++q) tab[lay.head() + 20 * j + 12 + q] = ph[q];
      }
      M2 ps = eye();
      for (int j = e - 1; j >= s; --j) {
        ps = mul(neg(Hm[j]), ps);
        for (int q = 0; q < 4; ++q) tab[lay.head() + 20 * j + 16 + q] = ps[q];
      }
      for (int j = s; j < e; ++j)
        for (int q = 0; q < 4; ++q) {
          tab[lay.head() + 20 * j + q] = Lf[j][q];
          tab[lay.head() + 20 * j + 4 + q] = Pm[j][q];
          tab[lay.head() + 20 * j + 8 + q] = Hm[j][q];
        }
    }
  } else {
    // ring transfers of the two cyclic recurrences
    M2 Tr = eye(), Rr = eye();
    for (int cc = 0; cc < P; ++cc) {
      const int s = cc * C, e = std::min(s + C, n_rows);
      M2 Tc, Rc;
      for (int q = 0; q < 4; ++q) {
        Tc[q] = tab[lay.phi() + 4 * (e - s - 1) + q];
        Rc[q] = tab[lay.psi() + 4 * (e - s) + q];
      }
      Tr = mul(Tc, Tr);   // T_{P-1} ... T_0
      Rr = mul(Rr, Rc);   // R_0 R_1 ... R_{P-1}
    }
    const M2 Gf = inv(sub(eye(), Tr)), Gb = inv(sub(eye(), Rr));
    for (int q = 0; q < 4; ++q) {
      tab[lay.cst() + 16 + q] = Gf[q];
      tab[lay.cst() + 20 + q] = Gb[q];
    }
  }
  // closure constants (ccd_solver.py:408-456)
  const int b = lay.bc();
  for (int q = 0; q < 4; ++q) {
    tab[b + q] = L[q];
    tab[b + 4 + q] = U[q];
    tab[b + 8 + q] = Ml[q];
    tab[b + 12 + q] = Mr[q];
  }
  const double cIl[4] = {-23.0 / 6.0, 21.0 / 4.0, -1.5, 1.0 / 12.0};
  const double cII[6] = {45.0, -154.0, 214.0, -156.0, 61.0, -10.0};
  for (int q = 0; q < 4; ++q) {
    tab[b + 16 + q] = cIl[q] / h;
    tab[b + 20 + q] = -cIl[q] / h;
  }
  for (int q = 0; q < 6; ++q) tab[b + 24 + q] = cII[q] / (12.0 * h * h);
  tab[b + 30] = kA1 / h;
  tab[b + 31] = kA2 / (h * h);
  p->P = P;
  p->H0 = H0;
  return TPF_OK;
}

struct LaunchShape {
  int TL, LS, FS, nbuf, grid;
  size_t smem;
};

template <typename T>
size_t smem_bytes(const tpf_ccd_plan* p, bool contig, int TL, int nbuf, int LS, int FS) {
  TabLayout lay{p->C, p->H0};
  const size_t fsz = contig ? (size_t)TL * FS : (size_t)TL * p->n_pts;
  return sizeof(double) * 4 * TL + sizeof(long long) * 2 * TL +
         sizeof(T) * (((size_t)lay.total() + 1) & ~(size_t)1) + sizeof(T) * (((size_t)TL * LS + 1) & ~(size_t)1) +
         sizeof(T) * nbuf * fsz + sizeof(T) * (size_t)p->P * TL * 4 + 64;
}

template <typename T>
LaunchShape pick_shape(const tpf_ccd_plan* p, bool contig, int64_t n_lines) {
  const int n = (int)p->n_pts;
  const int LS = 2 * p->n_rows + 1;
  const int FS = (n % 2) ? n : n + 1;
  const int nsm = tpf::sm_count();
  LaunchShape best{};
  best.TL = 0;
  double best_score = -1e30;
  const int tl_opts[6] = {32, 16, 8, 4, 2, 1};
  for (int t = 0; t < 6; ++t) {
    const int TL = tl_opts[t];
    if (TL * p->P > 512) continue;
    const int64_t tiles = (n_lines + TL - 1) / TL;
    for (int nbuf = 2; nbuf >= 1; --nbuf) {
      const size_t sm = smem_bytes<T>(p, contig, TL, nbuf, LS, FS);
      if (sm > 225 * 1024) continue;
      const int per_sm = std::max(1, (int)std::min<size_t>(8, (228 * 1024) / (sm + 1024)));
      const int64_t slots = (int64_t)nsm * per_sm;
      const int64_t grid = std::min<int64_t>(tiles, slots);
      // score: enough resident threads, full waves, prefetch when CTAs own >1 tile
      const double waves = (double)tiles / (double)grid;
      const double threads_per_sm = (double)std::min<int64_t>(per_sm, (grid + nsm - 1) / nsm) * TL * p->P;
      double score = std::min(threads_per_sm, 512.0) + (nbuf == 2 && waves > 1.5 ? 200.0 : 0.0) +
                     (grid >= nsm ? 100.0 : 100.0 * grid / nsm);
      if (nbuf == 2 && waves <= 1.0) score -= 300.0;   // a second buffer without a second tile is waste
      if (score > best_score) {
        best_score = score;
        best = {TL, LS, FS, nbuf, (int)grid, sm};
      }
    }
  }
  return best;
}

// ---- chunk kernels: launch -------------------------------------------------------
// How a call's lines are cut up: TL adjacent lines per block (0: a line is too
// long for a block), `staged`, `steal` and `wide` (up to 1024 threads) for the
// strided axes, `pitch` of the contiguous axis' lines in shared memory.  The results do
// not depend on any of them (each line is solved by its own threads).
struct ChunkShape {
  int TL, threads, pitch;
  bool staged, steal, wide;
  size_t smem;
  unsigned blocks;
};

// The rule (one B200, FP64 unless said; us per call; plain: d1 and d2 stored as
// they are, heavy: the corrector and variable-density epilogues).  What counts is how many
// threads are resident on an SM, and then how long a run of adjacent lines a
// block reads of each row:
// * Strided axes: 16 lines, i.e. 128-byte rows; 32 where that keeps as many
//   threads resident and the rows do not start on 32-byte sectors (257^3: 98.8
//   against 108.9 on axis 0; 256^3 nodes, whose rows do: 89.0 against 81.7;
//   129 x 97 x 162 axis 1, 480 resident threads against 384: 13.1 against 16.3);
//   not for FP64 lines of 11 to 14 chunks, where two blocks of 16 lines hold as
//   many threads as one of 32 (209^3 53.4 against 60.2, 225^3 65.5 against 68.2,
//   193^3 45 and 47; 241^3, 15 chunks, the other way, 93.5 against 81, and so the
//   epilogues on walls, whose 128 registers spill, 193^3 108 against 103).
//   Longer lines (more than 32 chunks) take fewer: half as many each time.
// * Where such a block has more than half of the threads an SM holds in FP64, a
//   second one does not fit beside it and half as many lines again keep more
//   threads resident: 24, 12, 6 or 3, where there are several tiles per SM (axis
//   0, wall: 273^3 134 against 160 with 16 lines, 300^3 153 against 182, 520 x
//   200 x 200 149 against 180, 600 x 160 x 160 104 against 125; 2051^2 57 against
//   62).  At 20 chunks and more of 16 lines, where rows do not start on a sector,
//   20 are the better number on walls (321^3 221 with 20, 228 with 24, 242 with
//   16; 385^3 the other way, 406 against 372) and 16 on periodic lines (321^3 198
//   with 16, 209 with 20, 218 with 24; 320^3, aligned, 198 with 16, 178 with 24).
// * FP32, plain, where there are several tiles per SM: up to 1024 threads of 64
//   registers instead of 512 of 74; 32 to 24 lines where two blocks fit, else the
//   most that one holds (wall, axis 0: 145^3 11.4 against 14.2, 209^3 34 against
//   43, 257^3 66 against 79, 273^3 93 against 108, 300^3 87 against 103, 417^3 305
//   against 403, 513^3 540 against 653, 1100 x 140 x 140 127 against 192, 2049 x
//   140 x 140 243 against 387).  Not where rows start on 16 bytes and one block of
//   32 lines leaves no room for a second (340^3 148 against 139).  Periodic lines,
//   which take 64 registers anyway, only from 64 chunks on, where 512 threads hold
//   but 16 to 28 bytes of a row, or where misaligned rows lie far apart (513^3 axis
//   0, rows 1 MB apart: 536 against 570; axis 1 506 against 465, 256^3 50 against 44).
// * Contiguous axis: 8 or 16 lines, whichever keeps more threads resident (193
//   nodes: 45.3 with 8, 54.5 with 16; 162 nodes: 18.6 and 15.3).
// * Fewer lines per block while that leaves half of the SMs without one, down
//   to 128 threads (401 x 301: 6.2 with 8 lines, 7.6 with 16).
// * Staging (the next tile's f copied while this one is solved) in FP64 once
//   every resident block has more than two tiles: 257^3 98.8 against 112.5,
//   193^3 45.3 against 57.9; 129 x 97 x 162 the other way, 14.1 against 13.1;
//   FP32 191 x 160 x 225 29.5 against 19.6.
// * Its tiles dealt out instead of taken by a fixed stride for fields of more than
//   2 GB in and out and for up to 8 lines a block, from 22 chunks on (periodic
//   449^3 491 against 678, 577^3 axis 0 1338 against 1760; wall 449^3 550 against
//   577, 1025 x 140 x 140 154 against 170; 300^3 154 and 156; 600 x 161 x 161 the
//   other way, 128 against 122).  Not walls of 29 to 32 chunks (481^3 805 against
//   769), nor the heavy epilogues on walls, which it makes spill more (193^3 115
//   against 105).
template <typename T>
ChunkShape chunk_shape(const tpf_ccd_plan* p, bool contig, bool plain, bool heavy, int64_t n_lines, int64_t inner) {
  constexpr bool F64 = std::is_same<T, double>::value;
  const int Q = (p->n_rows + kChunkR - 1) / kChunkR, n = (int)p->n_pts, nsm = tpf::sm_count();
  ChunkShape s{};
  // a pitch of n has bank conflicts of degree gcd(n, 16) (FP64; FP32 gcd(n, 32))
  s.pitch = (n & 3) == 0 ? n + 1 : n;
  const size_t fixed = 4 * (size_t)(kChunkHead + kChunkR);
  auto threads = [&](int tl) { return (tl * Q + 31) / 32 * 32; };
  auto smem = [&](int tl, bool staged) {
    const size_t tiles = contig ? 2 * (((size_t)tl * s.pitch + 3) & ~(size_t)3) : staged ? (size_t)tl * n : 0;
    return sizeof(T) * (fixed + 4 * (size_t)threads(tl) + tl + tiles);
  };
  const size_t limit = 200 * 1024;
  auto fits = [&](int tl) { return tl * Q <= 512 && smem(tl, false) <= limit; };
  auto per_sm = [&](int tl) { return std::max(1, 65536 / ((F64 ? 128 : 96) * threads(tl))); };
  auto resident = [&](int tl) { return fits(tl) ? per_sm(tl) * tl * Q : 0; };
  auto tiles = [&](int tl) { return (n_lines + tl - 1) / tl; };
  auto many = [&](int tl) { return tiles(tl) >= 4 * (int64_t)nsm; };
  auto done = [&](int tl) {
    s.TL = tl;
    s.threads = threads(tl);
    s.smem = smem(tl, s.staged);
    s.blocks = (unsigned)(s.staged && !s.steal ? (int64_t)nsm * per_sm(tl) : tiles(tl));
    return s;
  };
  const bool wall = p->bc == TPF_BC_WALL, ragged = (inner * sizeof(T)) % 16 != 0;
  if (!F64 && !contig && plain &&
      (wall ? ragged || Q < 22 || Q > 32 : Q > 64 || (ragged && Q > 16 && inner * sizeof(T) >= 128 * 1024))) {
    int tl = 0;
    for (int k : {24, 28, 32})   // two blocks of an SM's 1024 threads
      if (k * Q <= 512) tl = k;
    if (!tl)
      for (int k : {4, 6, 8, 12, 16, 24, 28, 32})
        if (k * Q <= 1024) tl = k;
    if (tl && many(tl)) {
      s.wide = true;
      return done(tl);
    }
  }
  int TL = 16;
  if (contig) TL = resident(16) > resident(8) ? 16 : 8;
  else if (resident(32) >= resident(16) && (inner * sizeof(T)) % 32 != 0 && tiles(32) >= nsm &&
           !(F64 && Q > 10 && Q < 15 && (plain || !wall)))
    TL = 32;
  while (TL > 2 && !fits(TL)) TL >>= 1;
  if (!fits(TL)) return s;
  if (F64 && !contig && TL <= 16 && TL * Q > 256) {
    int more = TL + TL / 2;
    if (TL == 16 && Q > 19 && (inner * sizeof(T)) % 32 != 0) more = wall && Q < 23 ? 20 : TL;
    if (more * Q <= 512 && many(more)) TL = more;
  }
  while (TL > 2 && 2 * tiles(TL) <= nsm && TL / 2 * Q >= 128) TL >>= 1;
  s.staged = !contig && F64 && tiles(TL) > 2 * (int64_t)nsm * per_sm(TL) && smem(TL, true) <= limit;
  const bool far = 3 * sizeof(T) * (double)n_lines * n > 2e9;   // in and out
  s.steal = s.staged && Q > 21 && (far || TL <= 8) && !(wall && (heavy || (Q > 28 && Q < 33)));
  return done(TL);
}

template <typename T>
int launch_chunk(const tpf_ccd_plan* p, CcdArgs a, bool per, bool contig, const ChunkShape& sh, cudaStream_t s) {
  const int Q = (p->n_rows + kChunkR - 1) / kChunkR;
  a.TL = sh.TL;
  a.tl_shift = 0;
  while ((1 << a.tl_shift) < sh.TL) ++a.tl_shift;
  a.tl_inv = 65536 / sh.TL + 1;
  a.n_tiles = (int)((a.n_lines + sh.TL - 1) / sh.TL);
  const T* g;
  const ChunkConst<T, kChunkR>* K;
  if constexpr (std::is_same<T, double>::value) {
    g = p->d_g64;
    K = &p->c64;
  } else {
    g = p->d_g32;
    K = &p->c32;
  }
  const bool plain = !a.J && !a.vd_out && !a.cr_out;
  if (contig) {
    // 16-byte pieces where the pitch is n and every block's run of every array starts on 16 bytes
    const bool vec = sh.pitch == p->n_pts && ((size_t)sh.TL * p->n_pts * sizeof(T)) % 16 == 0 &&
                     (((uintptr_t)a.f | (uintptr_t)a.d1 | (uintptr_t)a.d2) & 15) == 0;
    auto pick = [&](auto pl) {
      constexpr bool PL = decltype(pl)::value;
      return per ? ccd_chunk_contig_kernel<T, kChunkR, true, PL> : ccd_chunk_contig_kernel<T, kChunkR, false, PL>;
    };
    auto kern = plain ? pick(std::true_type{}) : pick(std::false_type{});
    if (sh.smem > 48 * 1024)   // more than a launch may use unasked
      TPF_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    kern<<<sh.blocks, sh.threads, sh.smem, s>>>(a, *K, g, Q, sh.pitch, vec ? 1 : 0);
  } else {
    auto pick = [&](auto epi, auto stage, auto pow2, auto threads) {
      constexpr int E = decltype(epi)::value, S = decltype(stage)::value, TH = decltype(threads)::value;
      constexpr bool P2 = decltype(pow2)::value;
      return per ? ccd_chunk_strided_kernel<T, kChunkR, true, E, S, P2, TH>
                 : ccd_chunk_strided_kernel<T, kChunkR, false, E, S, P2, TH>;
    };
    const bool pow2 = (sh.TL & (sh.TL - 1)) == 0;
    using Direct = std::integral_constant<int, kChunkDirect>;
    using Few = std::integral_constant<int, 512>;
    auto pick2 = [&](auto epi) {
      constexpr int E = decltype(epi)::value;
      if constexpr (std::is_same<T, double>::value) {
        auto lines = [&](auto stage) {
          return pow2 ? pick(epi, stage, std::true_type{}, Few{}) : pick(epi, stage, std::false_type{}, Few{});
        };
        if (sh.steal) return lines(std::integral_constant<int, kChunkSteal>{});
        if (sh.staged) return lines(std::integral_constant<int, kChunkStride>{});
        return lines(Direct{});
      } else {
        if constexpr (E == kChunkPlain)
          if (sh.wide) return pick(epi, Direct{}, std::false_type{}, std::integral_constant<int, 1024>{});
        return pick(epi, Direct{}, std::true_type{}, Few{});
      }
    };
    auto kern = a.cr_out   ? pick2(std::integral_constant<int, kChunkCorrector>{})
                : a.vd_out ? pick2(std::integral_constant<int, kChunkVd>{})
                : a.J      ? pick2(std::integral_constant<int, kChunkMetric>{})
                           : pick2(std::integral_constant<int, kChunkPlain>{});
    if (sh.smem > 48 * 1024) TPF_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    kern<<<sh.blocks, sh.threads, sh.smem, s>>>(a, *K, g, Q);
  }
  TPF_CUDA_TRY(cudaGetLastError());
  return TPF_OK;
}

template <typename T>
int launch_ccd(const tpf_ccd_plan* p, int64_t outer, int64_t inner, const void* f, void* d1, void* d2,
               const double* bcl, const double* bcr, int flags, cudaStream_t stream,
               const void* vd_rho = nullptr, const void* vd_drho = nullptr, void* vd_out = nullptr,
               int vd_accumulate = 0, const CcdArgs* corrector = nullptr) {
  const bool contig = (inner == 1);
  const int64_t n_lines = outer * inner;
  if (n_lines == 0) return TPF_OK;
  TPF_CHECK_ARG(f != d1 && f != d2 && f != vd_out, "the CCD input must not alias an output array");
  TPF_CHECK_ARG(!corrector || (f != corrector->cr_out && f != corrector->cr_u && f != corrector->cr_rho),
                "the pressure must not alias the velocity or density arrays");
  TPF_CHECK_ARG(n_lines < ((int64_t)1 << 31), "too many lines");
  CcdArgs a{};
  a.f = f; a.d1 = d1; a.d2 = d2;
  a.outer = outer; a.inner = inner; a.n_lines = n_lines;
  a.n = (int)p->n_pts; a.n_rows = p->n_rows; a.C = p->C; a.P = p->P; a.H0 = p->H0;
  a.tab_total = TabLayout{p->C, p->H0}.total();
  a.tab = p->d_tab;
  a.tabT = std::is_same<T, double>::value ? (const void*)p->d_tab : (const void*)p->d_tabf;
  a.J = ((flags & TPF_CCD_APPLY_METRIC) && p->has_metric) ? p->d_J : nullptr;
  a.ovl = bcl ? 1 : 0;
  a.ovr = bcr ? 1 : 0;
  if (bcl) { a.bcl0 = bcl[0]; a.bcl1 = bcl[1]; }
  if (bcr) { a.bcr0 = bcr[0]; a.bcr1 = bcr[1]; }
  a.vd_rho = vd_rho;
  a.vd_drho = vd_drho;
  a.vd_out = vd_out;
  a.vd_accumulate = vd_accumulate;
  if (corrector) {
    a.cr_u = corrector->cr_u;
    a.cr_rho = corrector->cr_rho;
    a.cr_out = corrector->cr_out;
    a.cr_dt = corrector->cr_dt;
    a.cr_wall = corrector->cr_wall;
  }
  const bool per = (p->bc == TPF_BC_PERIODIC) && !a.ovl && !a.ovr;
  if (per == (p->bc == TPF_BC_PERIODIC)) {
    const bool heavy = a.vd_out || a.cr_out;
    const ChunkShape sh = chunk_shape<T>(p, contig, !a.J && !heavy, heavy, n_lines, inner);
    if (sh.TL > 0) return launch_chunk<T>(p, a, per, contig, sh, stream);
  }
  // longer lines, and closure overrides on a periodic plan
  const LaunchShape s = pick_shape<T>(p, contig, n_lines);
  TPF_CHECK_ARG(s.TL > 0, "CCD axis of %lld points does not fit the line kernel's shared memory",
                (long long)p->n_pts);
  a.TL = s.TL;
  a.tl_shift = 0;
  while ((1 << a.tl_shift) < s.TL) ++a.tl_shift;
  a.LS = s.LS; a.FS = contig ? s.FS : 0; a.nbuf = s.nbuf;
  a.n_tiles = (int)((n_lines + s.TL - 1) / s.TL);
  void (*kern)(CcdArgs);
  if (per) kern = contig ? ccd_line_kernel<T, true, true> : ccd_line_kernel<T, true, false>;
  else kern = contig ? ccd_line_kernel<T, false, true> : ccd_line_kernel<T, false, false>;
  TPF_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem));
  kern<<<s.grid, s.TL * p->P, s.smem, stream>>>(a);
  TPF_CUDA_TRY(cudaGetLastError());
  return TPF_OK;
}

// ---- FP32 line solves under FP64 iterative refinement (wall axes) ----------------
//
// d = K32(f) in FP32, then per refinement the residual of the full
// (N+1)-node CCD system, R = B f - A d, in FP64 (interior Eq-I / Eq-II rows,
// the one-sided closure rows at both walls, ccd_solver.py:11-22,408-465),
// and d += A^-1 R with the correction solved in FP32: the boundary rows are
// folded into the first / last interior rows (delta_0 = M_l delta_1 + R_0,
// ccd_solver_helpers.py:242-245), one thread runs the block-Thomas sweeps of
// a line with per-row factors, and the boundary corrections are recovered.

__device__ __forceinline__ float2 mv2f(const float* m, float a, float b) {
  return make_float2(m[0] * a + m[1] * b, m[2] * a + m[3] * b);
}

__global__ void ccd_cast_kernel(int64_t n, const double* __restrict__ in, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}

__global__ void ccd_widen_kernel(int64_t n, const float* __restrict__ in, double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}

// R = B f - A d at every node, FP64 arithmetic, FP32 storage
__global__ void ccd_resid_kernel(int64_t total, int64_t inner, int n, double h, const double* __restrict__ f,
                                 const double* __restrict__ d1, const double* __restrict__ d2,
                                 float* __restrict__ R1, float* __restrict__ R2) {
  const double a1h = kA1 / h, a2h2 = kA2 / (h * h), b1h = kB1 * h, b2h = kB2 / h;
  const double inv12h2 = 1.0 / (12.0 * h * h);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ln = e / inner;
    const int k = (int)(ln % n);
    const int64_t s = inner;
    double r1, r2;
    if (k == 0) {
      const double cI = (-23.0 / 6.0 * f[e] + 21.0 / 4.0 * f[e + s] - 1.5 * f[e + 2 * s] + 1.0 / 12.0 * f[e + 3 * s]) / h;
      const double cII = (45.0 * f[e] - 154.0 * f[e + s] + 214.0 * f[e + 2 * s] - 156.0 * f[e + 3 * s] +
                          61.0 * f[e + 4 * s] - 10.0 * f[e + 5 * s]) * inv12h2;
      r1 = cI - (d1[e] - (-1.5 * d1[e + s] + 1.5 * h * d2[e + s]));
      r2 = cII - d2[e];
    } else if (k == n - 1) {
      const double cI = (23.0 / 6.0 * f[e] - 21.0 / 4.0 * f[e - s] + 1.5 * f[e - 2 * s] - 1.0 / 12.0 * f[e - 3 * s]) / h;
      const double cII = (45.0 * f[e] - 154.0 * f[e - s] + 214.0 * f[e - 2 * s] - 156.0 * f[e - 3 * s] +
                          61.0 * f[e - 4 * s] - 10.0 * f[e - 5 * s]) * inv12h2;
      r1 = cI - (d1[e] - (-1.5 * d1[e - s] - 1.5 * h * d2[e - s]));
      r2 = cII - d2[e];
    } else {
      const double fm = f[e - s], f0 = f[e], fp = f[e + s];
      const double pm = d1[e - s], p0 = d1[e], pp = d1[e + s];
      const double qm = d2[e - s], q0 = d2[e], qp = d2[e + s];
      r1 = a1h * (fp - fm) - (kAlpha1 * (pm + pp) + p0 - b1h * (qp - qm));
      r2 = a2h2 * ((fm - 2.0 * f0) + fp) - (kBeta2 * (qm + qp) + q0 - b2h * (pp - pm));
    }
    R1[e] = (float)r1;
    R2[e] = (float)r2;
  }
}

// d += A^-1 R on every line (FP32 sweeps; R is overwritten by the forward sweep)
__global__ void ccd_corr_kernel(int64_t n_lines, int64_t inner, int n, float h, const float* __restrict__ fac,
                                float* R1, float* R2, double* d1, double* d2) {
  const int64_t L = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (L >= n_lines) return;
  const int64_t o = L / inner, i = L - o * inner;
  const int64_t base = o * (int64_t)n * inner + i;
  const int64_t s = inner;
  const int nr = n - 2;
  const float La[4] = {(float)kAlpha1, (float)kB1 * h, (float)kB2 / h, (float)kBeta2};
  const float Ua[4] = {(float)kAlpha1, -(float)kB1 * h, -(float)kB2 / h, (float)kBeta2};
  const float Ml[4] = {-1.5f, 1.5f * h, 0.0f, 0.0f};
  const float Mr[4] = {-1.5f, -1.5f * h, 0.0f, 0.0f};
  const float r0a = R1[base], r0b = R2[base];
  const float rNa = R1[base + (int64_t)(n - 1) * s], rNb = R2[base + (int64_t)(n - 1) * s];
  float ya = 0.0f, yb = 0.0f;
  for (int j = 0; j < nr; ++j) {
    const int64_t e = base + (int64_t)(j + 1) * s;
    float ra = R1[e], rb = R2[e];
    if (j == 0) {
      const float2 q = mv2f(La, r0a, r0b);
      ra -= q.x;
      rb -= q.y;
    }
    if (j == nr - 1) {
      const float2 q = mv2f(Ua, rNa, rNb);
      ra -= q.x;
      rb -= q.y;
    }
    const float* lf = fac + 12 * j;
    const float2 q = mv2f(lf, ya, yb);
    ya = ra - q.x;
    yb = rb - q.y;
    R1[e] = ya;
    R2[e] = yb;
  }
  float xa = 0.0f, xb = 0.0f, x1a = 0.0f, x1b = 0.0f, xla = 0.0f, xlb = 0.0f;
  for (int j = nr - 1; j >= 0; --j) {
    const int64_t e = base + (int64_t)(j + 1) * s;
    const float* pm = fac + 12 * j + 4;
    const float* hm = pm + 4;
    const float2 py = mv2f(pm, R1[e], R2[e]);
    const float2 hx = mv2f(hm, xa, xb);
    xa = py.x - hx.x;
    xb = py.y - hx.y;
    d1[e] += (double)xa;
    d2[e] += (double)xb;
    if (j == nr - 1) { xla = xa; xlb = xb; }
    if (j == 0) { x1a = xa; x1b = xb; }
  }
  const float2 b0 = mv2f(Ml, x1a, x1b);
  const float2 bN = mv2f(Mr, xla, xlb);
  d1[base] += (double)(b0.x + r0a);
  d2[base] += (double)(b0.y + r0b);
  d1[base + (int64_t)(n - 1) * s] += (double)(bN.x + rNa);
  d2[base + (int64_t)(n - 1) * s] += (double)(bN.y + rNb);
}

// per-row factors of the folded wall system (the recurrence of build_tables)
int refine_factors(const tpf_ccd_plan* p) {
  if (p->d_rfac) return TPF_OK;
  const double h = p->h;
  const int nr = p->n_rows;
  const M2 L = {kAlpha1, kB1 * h, kB2 / h, kBeta2};
  const M2 U = {kAlpha1, -kB1 * h, -kB2 / h, kBeta2};
  const M2 Ml = {-1.5, 1.5 * h, 0.0, 0.0};
  const M2 Mr = {-1.5, -1.5 * h, 0.0, 0.0};
  std::vector<float> fac((size_t)12 * nr);
  M2 LUp = eye();
  for (int j = 0; j < nr; ++j) {
    M2 D = eye();
    if (j == 0) D = add(D, mul(L, Ml));
    if (j == nr - 1) D = add(D, mul(U, Mr));
    M2 Lf = {0, 0, 0, 0}, LU;
    if (j == 0) LU = D;
    else {
      Lf = mul(L, inv(LUp));
      LU = sub(D, mul(Lf, U));
    }
    const double dt = det(LU);
    if (!std::isfinite(dt) || std::fabs(dt) < 1e-300) {
      tpf::set_error("CCD block-tridiagonal factorization encountered a singular pivot at block %d", j);
      return TPF_ESINGULAR;
    }
    const M2 Pm = inv(LU);
    const M2 Hm = (j < nr - 1) ? mul(Pm, U) : M2{0, 0, 0, 0};
    for (int q = 0; q < 4; ++q) {
      fac[12 * j + q] = (float)Lf[q];
      fac[12 * j + 4 + q] = (float)Pm[q];
      fac[12 * j + 8 + q] = (float)Hm[q];
    }
    LUp = LU;
  }
  float* d = nullptr;
  if (cudaMalloc(&d, fac.size() * sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    tpf::set_error("cudaMalloc of the refinement factors failed");
    return TPF_ECUDA;
  }
  if (cudaMemcpy(d, fac.data(), fac.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(d);
    tpf::set_error("cudaMemcpy of the refinement factors failed");
    return TPF_ECUDA;
  }
  p->d_rfac = d;
  return TPF_OK;
}

}  // namespace

extern "C" {

int tpf_ccd_plan_create(tpf_ccd_plan** out, int64_t n_pts, double h, int bc, int dtype) {
  TPF_CHECK_ARG(out != nullptr, "plan pointer is NULL");
  *out = nullptr;
  TPF_CHECK_ARG(bc == TPF_BC_WALL || bc == TPF_BC_PERIODIC, "unsupported boundary type %d", bc);
  TPF_CHECK_ARG(dtype == TPF_F64 || dtype == TPF_F32, "unsupported dtype %d", dtype);
  TPF_CHECK_ARG(std::isfinite(h) && h > 0.0, "grid spacing must be positive and finite");
  if (bc == TPF_BC_WALL) {
    TPF_CHECK_ARG(n_pts >= 6,
                  "CCD wall Eq-II boundary closure requires n_pts >= 6 for the six-point O(h^4) formula");
  } else {
    TPF_CHECK_ARG(n_pts >= 4, "Need >= 3 unique nodes for periodic CCD; got %lld", (long long)(n_pts - 1));
  }
  TPF_CHECK_ARG(n_pts <= 8193, "CCD axis longer than 8193 points is not supported");
  auto* p = new tpf_ccd_plan();
  p->n_pts = n_pts;
  p->h = h;
  p->bc = bc;
  p->dtype = dtype;
  p->n_rows = (bc == TPF_BC_WALL) ? (int)(n_pts - 2) : (int)(n_pts - 1);
  // chunk length of ccd_line_kernel's tables: 8 rows up to 1024, else a 32nd of
  // the line
  p->C = p->n_rows <= 1024 ? 8 : (p->n_rows + 31) / 32;
  std::vector<double> tab;
  int st = build_tables(p, tab);
  if (st != TPF_OK) { delete p; return st; }
  if (cudaMalloc(&p->d_tab, tab.size() * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&p->d_tabf, tab.size() * sizeof(float)) != cudaSuccess) {
    tpf::set_error("cudaMalloc of CCD tables failed");
    cudaFree(p->d_tab);
    delete p;
    return TPF_ECUDA;
  }
  std::vector<float> tf(tab.begin(), tab.end());
  if (cudaMemcpy(p->d_tab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(p->d_tabf, tf.data(), tf.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
    tpf::set_error("copy of CCD tables failed");
    cudaFree(p->d_tab);
    cudaFree(p->d_tabf);
    delete p;
    return TPF_ECUDA;
  }
  {
    std::vector<double> G;
    p->c64 = chunk_tables<kChunkR>(p, G);
    p->c32 = cast_chunk<float>(p->c64);
    const std::vector<float> Gf(G.begin(), G.end());
    if (cudaMalloc(&p->d_g64, G.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&p->d_g32, G.size() * sizeof(float)) != cudaSuccess ||
        cudaMemcpy(p->d_g64, G.data(), G.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(p->d_g32, Gf.data(), Gf.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
      tpf::set_error("allocation / copy of the CCD wall table failed");
      cudaFree(p->d_tab);
      cudaFree(p->d_tabf);
      cudaFree(p->d_g64);
      cudaFree(p->d_g32);
      delete p;
      return TPF_ECUDA;
    }
  }
  *out = p;
  return TPF_OK;
}

int tpf_ccd_plan_set_autotune(tpf_ccd_plan* p, int enable) {
  TPF_CHECK_ARG(p != nullptr, "plan is NULL");
  (void)enable;   // launch shapes follow from the sizes
  return TPF_OK;
}

int tpf_ccd_plan_destroy(tpf_ccd_plan* p) {
  if (!p) return TPF_OK;
  cudaFree(p->d_tab);
  cudaFree(p->d_tabf);
  cudaFree(p->d_g64);
  cudaFree(p->d_g32);
  cudaFree(p->d_J);
  cudaFree(p->d_rfac);
  delete p;
  return TPF_OK;
}

int tpf_ccd_plan_set_metric(tpf_ccd_plan* p, const double* J, const double* dJ) {
  TPF_CHECK_ARG(p && J && dJ, "NULL argument");
  if (!p->d_J) TPF_CUDA_TRY(cudaMalloc(&p->d_J, 2 * p->n_pts * sizeof(double)));
  TPF_CUDA_TRY(cudaMemcpy(p->d_J, J, p->n_pts * sizeof(double), cudaMemcpyHostToDevice));
  TPF_CUDA_TRY(cudaMemcpy(p->d_J + p->n_pts, dJ, p->n_pts * sizeof(double), cudaMemcpyHostToDevice));
  p->has_metric = true;
  return TPF_OK;
}

int tpf_ccd_apply(const tpf_ccd_plan* p, int64_t outer, int64_t inner, const void* f, void* d1, void* d2,
                  const double* bc_left, const double* bc_right, int flags, void* stream) {
  TPF_CHECK_ARG(p != nullptr, "plan is NULL");
  TPF_CHECK_ARG(outer >= 0 && inner >= 1, "invalid line decomposition outer=%lld inner=%lld",
                (long long)outer, (long long)inner);
  TPF_CHECK_ARG(f != nullptr, "input is NULL");
  TPF_CHECK_ARG(d1 != nullptr || d2 != nullptr, "no output requested");
  TPF_CHECK_ARG(!(flags & TPF_CCD_APPLY_METRIC) || p->has_metric, "metric requested but not set");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->dtype == TPF_F64) return launch_ccd<double>(p, outer, inner, f, d1, d2, bc_left, bc_right, flags, s);
  return launch_ccd<float>(p, outer, inner, f, d1, d2, bc_left, bc_right, flags, s);
}

int tpf_ccd_apply_refined(const tpf_ccd_plan* p64, const tpf_ccd_plan* p32, int64_t outer, int64_t inner,
                          const double* f, double* d1, double* d2, int refinements, float* work, void* stream) {
  TPF_CHECK_ARG(p64 && p32 && f && d1 && d2 && work, "NULL argument");
  TPF_CHECK_ARG(p64->dtype == TPF_F64 && p32->dtype == TPF_F32, "plans must be FP64 and FP32");
  TPF_CHECK_ARG(p64->bc == TPF_BC_WALL && p32->bc == TPF_BC_WALL,
                "iterative refinement of the CCD line solves covers wall axes");
  TPF_CHECK_ARG(p64->n_pts == p32->n_pts && p64->h == p32->h, "the FP64 and FP32 plans differ");
  TPF_CHECK_ARG(outer >= 0 && inner >= 1, "invalid line decomposition");
  TPF_CHECK_ARG(refinements >= 0 && refinements <= 8, "refinements must be in [0, 8]");
  TPF_CHECK_ARG(f != d1 && f != d2 && d1 != d2, "f, d1 and d2 must be distinct");
  const int64_t n_lines = outer * inner;
  if (n_lines == 0) return TPF_OK;
  int st = refine_factors(p64);
  if (st) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = (int)p64->n_pts;
  const int64_t total = n_lines * n;
  float* f32 = work;
  float* a32 = work + total;
  float* b32 = work + 2 * total;
  float* R1 = work + 3 * total;
  float* R2 = work + 4 * total;
  const int eb = (int)std::min<int64_t>((total + 255) / 256, 8 * 148 * 4);
  ccd_cast_kernel<<<eb, 256, 0, s>>>(total, f, f32);
  TPF_CUDA_TRY(cudaGetLastError());
  if ((st = launch_ccd<float>(p32, outer, inner, f32, a32, b32, nullptr, nullptr, 0, s))) return st;
  ccd_widen_kernel<<<eb, 256, 0, s>>>(total, a32, d1);
  ccd_widen_kernel<<<eb, 256, 0, s>>>(total, b32, d2);
  for (int r = 0; r < refinements; ++r) {
    ccd_resid_kernel<<<eb, 256, 0, s>>>(total, inner, n, p64->h, f, d1, d2, R1, R2);
    ccd_corr_kernel<<<(int)((n_lines + 127) / 128), 128, 0, s>>>(n_lines, inner, n, (float)p64->h, p64->d_rfac, R1,
                                                                 R2, d1, d2);
  }
  TPF_CUDA_TRY(cudaGetLastError());
  return TPF_OK;
}

int tpf_ccd_apply_vd(const tpf_ccd_plan* p, int64_t outer, int64_t inner, const void* f, const void* rho,
                     const void* drho, void* out, int accumulate, int flags, void* stream) {
  TPF_CHECK_ARG(p != nullptr, "plan is NULL");
  TPF_CHECK_ARG(outer >= 0 && inner >= 1, "invalid line decomposition");
  TPF_CHECK_ARG(f && rho && drho && out, "NULL argument");
  TPF_CHECK_ARG(!(flags & TPF_CCD_APPLY_METRIC) || p->has_metric, "metric requested but not set");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->dtype == TPF_F64)
    return launch_ccd<double>(p, outer, inner, f, nullptr, nullptr, nullptr, nullptr, flags, s, rho, drho, out,
                              accumulate);
  return launch_ccd<float>(p, outer, inner, f, nullptr, nullptr, nullptr, nullptr, flags, s, rho, drho, out,
                           accumulate);
}

int tpf_ccd_apply_corrector(const tpf_ccd_plan* p, int64_t outer, int64_t inner, const void* pres,
                            const void* u_star, const void* rho, double dt, void* u_out, int flags, void* stream) {
  TPF_CHECK_ARG(p != nullptr, "plan is NULL");
  TPF_CHECK_ARG(outer >= 0 && inner >= 1, "invalid line decomposition");
  TPF_CHECK_ARG(pres && u_star && rho && u_out, "NULL argument");
  TPF_CHECK_ARG(!(flags & TPF_CCD_APPLY_METRIC) || p->has_metric, "metric requested but not set");
  CcdArgs cr{};
  cr.cr_u = u_star;
  cr.cr_rho = rho;
  cr.cr_out = u_out;
  cr.cr_dt = dt;
  cr.cr_wall = (p->bc == TPF_BC_WALL) ? 1 : 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->dtype == TPF_F64)
    return launch_ccd<double>(p, outer, inner, pres, nullptr, nullptr, nullptr, nullptr, flags, s, nullptr, nullptr,
                              nullptr, 0, &cr);
  return launch_ccd<float>(p, outer, inner, pres, nullptr, nullptr, nullptr, nullptr, flags, s, nullptr, nullptr,
                           nullptr, 0, &cr);
}

int tpf_ccd_enforce_wall_neumann(const tpf_ccd_plan* p, int64_t outer, int64_t inner, void* grad,
                                 void* stream) {
  TPF_CHECK_ARG(p != nullptr && grad != nullptr, "NULL argument");
  if (p->bc != TPF_BC_WALL || outer * inner == 0) return TPF_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t tot = outer * inner * 2;
  int blocks = (int)std::min<int64_t>((tot + 255) / 256, 4096);
  if (p->dtype == TPF_F64)
    wall_zero_kernel<double><<<blocks, 256, 0, s>>>(static_cast<double*>(grad), outer, p->n_pts, inner);
  else
    wall_zero_kernel<float><<<blocks, 256, 0, s>>>(static_cast<float*>(grad), outer, p->n_pts, inner);
  TPF_CUDA_TRY(cudaGetLastError());
  return TPF_OK;
}

}  // extern "C"
