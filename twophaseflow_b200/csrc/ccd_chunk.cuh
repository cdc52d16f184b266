// Chunk-per-thread CCD line solve (included by ccd.cu).
//
// A line's rows are cut into chunks of R; one thread owns one chunk and holds
// its rows in registers, so a line of n rows is solved by Q = ceil(n / R)
// threads in two block barriers and f is read, d1 and d2 are written exactly
// once.
//
// Every row uses the fixed-point block-LU factors (the limit of the block
// Riccati recurrence), so the two sweeps are constant-coefficient recurrences
//     y_j = b_j + A y_{j-1},   x_j = P y_j + B x_{j+1},   A = -Lf, B = -H,
// whose powers decay like 0.455^k.  Hence a chunk needs only the end values of
// the kChunkWindow chunks next to it: what is left out is 0.455^64 = 1e-22 of the
// carry, on a ring whose last chunk is short at most 0.455^49 = 2e-17 (that chunk
// counts as one of the window's).  A thread sweeps its chunk from a zero carry, publishes the end value,
// reads its neighbours', and sweeps again from the carry they add up to.  No
// scan over the line, no per-row tables.  (Adding A^(r+1) times the carry to
// row r instead of the second sweep takes as many multiplications, but each
// with a constant of its own: the loads of those made 1 500 instructions per
// warp and tile of ~430 FP64 ones, 104 us on the 257^3 strided axes.)
//
// Walls: the factors above belong to a matrix M that differs from the folded
// wall system in its first diagonal block only (the last row's pivot is set
// exactly).  With V = M^-1 e_0 and the difference B0 of the two blocks,
// x = x' - V B0 (I + V_0 B0)^-1 x'_0, and the table G_j = V_j B0 (I + V_0 B0)^-1
// vanishes beyond kChunkHead rows: the first chunks subtract G_j x'_0.
// Periodic axes: the window wraps, and the ring sums are closed with
// (I - A^N)^-1 and (I - B^N)^-1, which makes short rings exact too.
//
// What bounds it: HBM's floor is 24 bytes a node (63 us at 257^3 FP64, 16 us
// per axis in FP32 at 192 x 161 x 226); at 128 registers a thread 16 warps are
// resident per SM, and between the two barriers they issue in 44 % of the
// cycles, 430 FP64 instructions a warp and tile.  8 rows a thread and twice the
// warps (64 registers) is slower, 160-180 us.  The FP64 wall kernels of the
// corrector and the variable-density term spill 16 to 48 bytes of a thread's
// stack at their 128 registers; the others spill nothing.  Against the kernels
// this replaces, a thread per line that read f twice and a scan of 2 x 2 maps over
// the warps of a line (us per call): 257^3 FP64 wall 99 / 99 / 97 on axes 0 / 1 / 2, before
// 116 / 118 / 209; periodic 96 / 95 / 91, before 105 / 108 / 193; FP32 192 x 161
// x 226 19 / 17 / 24, before 31 / 32 / 80; 129 x 97 x 162 13 / 13 / 15, before
// 64 / 80 / 51; 1025^2 8.7 / 9.2, before 25 / 22.
//
// The recurrences run on y scaled by diag(a1/h, a2/h^2)^-1, so that a row's
// right-hand side is the plain differences (f+ - f-, f+ - 2 f + f-).  Both come
// from the first differences, which are exact where f varies by less than a
// factor of two from node to node: f+ + f- - 2 f would round at the size of
// 2 f, which in FP32 doubled the error of f''.
#pragma once

namespace {

template <typename T>
__device__ __forceinline__ V2<T> cmv(const T* m, V2<T> v, V2<T> add) {   // add + m v
  return {fma(m[0], v.a, fma(m[1], v.b, add.a)), fma(m[2], v.a, fma(m[3], v.b, add.b))};
}

// Closure pieces of one wall from the six nodes next to it (FP64).
template <typename T>
__device__ __forceinline__ void chunk_closure(const double* cI, const double* cII, const T* v, int64_t step,
                                              double& r0, double& r1) {
  double fv[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) fv[k] = (double)v[(int64_t)k * step];
  r0 = cI[0] * fv[0] + cI[1] * fv[1] + cI[2] * fv[2] + cI[3] * fv[3];
  r1 = cII[0] * fv[0] + cII[1] * fv[1] + cII[2] * fv[2] + cII[3] * fv[3] + cII[4] * fv[4] + cII[5] * fv[5];
}

// Solve one chunk.  q: chunk of the line (q >= Q: an idle thread, which only
// takes part in the barriers), cnt: its rows, fv: f at the nodes before, of and
// after its rows; bl / br: wall closure pieces (chunks 0 / Q - 1).  e: shared
// [4][threads]; at, st: this thread's index and the distance of a neighbouring
// chunk in it.  G: shared [kChunkHead + R][4].  On return w: (f', f'') of the
// rows.
// A line with a value that is not finite becomes NaN from end to end, as the
// full recurrences would make it: its chunks find that in `poison`, a shared
// word of the line.
template <typename T, int R, bool PERIODIC>
__device__ __forceinline__ void chunk_solve(const ChunkConst<T, R>& K, const T (&fv)[R + 2], int q, int Q, int cnt,
                                            double bl0, double bl1, double br0, double br1, T* e, int nthr, int at,
                                            int st, T* poison, const T* G, V2<T> (&w)[R]) {
  const bool act = q < Q, last = q == Q - 1;
  const V2<T> zero{T(0), T(0)};
  T* ea = e;
  T* eb = e + nthr;
  T* xa = e + 2 * nthr;
  T* xb = e + 3 * nthr;
  // forward sweep from a zero carry; w: right-hand sides, later P y, then x
  V2<T> y = zero;
  T d0 = fv[1] - fv[0];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const T d1 = fv[r + 2] - fv[r + 1];
    w[r] = {d1 + d0, d1 - d0};
    d0 = d1;
    if (!PERIODIC && r == 0 && q == 0) {
      w[0].a -= (T)(K.cl[0] * bl0 + K.cl[1] * bl1);
      w[0].b -= (T)(K.cl[2] * bl0 + K.cl[3] * bl1);
    }
    y = r == 0 ? w[0] : cmv(K.A, y, w[r]);
  }
  if (PERIODIC && cnt < R) {   // the ring continues from the line's last row
    y = w[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
      if (r < cnt) y = cmv(K.A, y, w[r]);
  }
  ea[at] = y.a;
  eb[at] = y.b;
  if (q == 0) *poison = T(0);
  __syncthreads();
  const T bad = (y.a - y.a) + (y.b - y.b);   // 0 or NaN
  if (act && bad != T(0)) *poison = bad;
  // carry into this chunk
  V2<T> c = zero;
  auto ey = [&](int chunk) { const int i = at + (chunk - q) * st; return V2<T>{ea[i], eb[i]}; };
  if (act) {
    if (!PERIODIC || q >= kChunkWindow) {
#pragma unroll
      for (int m = kChunkWindow; m >= 1; --m)
        if (q >= m) c = cmv(K.AR, c, ey(q - m));
    } else {
      // into chunk 0 across the ring, then up to this one
      for (int m = min(kChunkWindow, Q); m >= 2; --m) c = cmv(K.AR, c, ey(Q - m));
      c = cmv(K.AL, c, ey(Q - 1));
      c = cmv(K.Gf, c, zero);
      for (int m = 0; m < q; ++m) c = cmv(K.AR, c, ey(m));
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    c = cmv(K.A, c, w[r]);
    w[r] = cmv(K.P, c, zero);
  }
  if (last) {   // the last row's closure and pivot; rows beyond the line count as 0
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!PERIODIC && r == cnt - 1) {
        w[r] = cmv(K.Z, w[r], V2<T>{-(T)(K.cr[0] * br0 + K.cr[1] * br1),
                                    -(T)(K.cr[2] * br0 + K.cr[3] * br1)});
      }
      if (r >= cnt) w[r] = zero;
    }
  }
  // backward sweep from a zero carry
  c = w[R - 1];
#pragma unroll
  for (int r = R - 2; r >= 0; --r) c = cmv(K.B, c, w[r]);
  xa[at] = c.a;
  xb[at] = c.b;
  __syncthreads();
  if (!act) return;
  auto ex = [&](int chunk) { const int i = at + (chunk - q) * st; return V2<T>{xa[i], xb[i]}; };
  const T bad_line = *poison;
  c = {bad_line, bad_line};
  if (!PERIODIC || q + kChunkWindow < Q) {
#pragma unroll
    for (int m = kChunkWindow; m >= 1; --m)
      if (q + m < Q) c = cmv(K.BR, c, ex(q + m));
  } else {
    // x_0, the carry into the last chunk, then down to this one
    auto down = [&](int m) { c = m == Q - 1 ? cmv(K.BL, c, ex(m)) : cmv(K.BR, c, ex(m)); };
    for (int m = min(kChunkWindow, Q) - 1; m >= 0; --m) down(m);
    c = cmv(K.Gb, c, zero);
    for (int m = Q - 1; m > q; --m) down(m);
  }
  if (!PERIODIC && q * R < kChunkHead) {   // the wall's first block
    V2<T> v = zero;
#pragma unroll
    for (int m = kChunkWindow; m >= 1; --m)
      if (m < Q) v = cmv(K.BR, v, ex(m));
    v = cmv(K.BR, v, ex(0));
    const V2<T>* g = reinterpret_cast<const V2<T>*>(G) + (size_t)q * R * 2;
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      c = cmv(K.B, c, w[r]);
      const V2<T> g0 = g[2 * r], g1 = g[2 * r + 1];
      w[r] = {c.a - (g0.a * v.a + g0.b * v.b), c.b - (g1.a * v.a + g1.b * v.b)};
    }
  } else {
    if (!PERIODIC || cnt == R) {
#pragma unroll
      for (int r = R - 1; r >= 0; --r) {
        c = cmv(K.B, c, w[r]);
        w[r] = c;
      }
    } else {   // the ring's carry enters at the line's last row
#pragma unroll
      for (int r = R - 1; r >= 0; --r)
        if (r < cnt) {
          c = cmv(K.B, c, w[r]);
          w[r] = c;
        }
    }
  }
}

// (f', f'') of a boundary node from its neighbouring row's solution
template <typename T>
__device__ __forceinline__ V2<double> chunk_edge(const double* M, V2<T> x, double b0, double b1) {
  const double x0 = (double)x.a, x1 = (double)x.b;
  return {(M[0] * x0 + M[1] * x1) + b0, (M[2] * x0 + M[3] * x1) + b1};
}

// EPI: what is written.  A kernel each, so that the operands of one do not
// cost the others registers.
enum { kChunkPlain = 0, kChunkMetric = 1, kChunkCorrector = 2, kChunkVd = 3 };

// Write a chunk's rows (element `base` + node * inner of the arrays).
template <typename T, int R, bool PERIODIC, int EPI>
__device__ __forceinline__ void chunk_store(const CcdArgs& a, const ChunkConst<T, R>& K, const V2<T> (&x)[R],
                                            int64_t base, int64_t inner, int q, bool last, int cnt, double bl0,
                                            double bl1, double br0, double br1) {
  const int n = a.n, off = PERIODIC ? 0 : 1;   // node of row 0
  const int k0 = q * R + off;
  const double* J = a.J;
  auto put = [&](int k, double o1, double o2) {
    if (EPI != kChunkPlain && J) {
      const double Jk = J[k], dJk = J[n + k];
      o2 = Jk * Jk * o2 + Jk * dJk * o1;
      o1 = Jk * o1;
    }
    const int64_t gi = base + (int64_t)k * inner;
    if constexpr (EPI == kChunkPlain || EPI == kChunkMetric) {   // without the others' registers
      if (a.d1) static_cast<T*>(a.d1)[gi] = (T)o1;
      if (a.d2) static_cast<T*>(a.d2)[gi] = (T)o2;
    } else {
      store_out<T>(a, gi, o1, o2, k);
    }
  };
  const int64_t o0 = base + (int64_t)k0 * inner;
  if constexpr (EPI == kChunkPlain) {
    T* p1 = a.d1 ? static_cast<T*>(a.d1) + o0 : nullptr;
    T* p2 = a.d2 ? static_cast<T*>(a.d2) + o0 : nullptr;
    if (cnt == R && p1 && p2) {
#pragma unroll
      for (int r = 0; r < R; ++r, p1 += inner, p2 += inner) {
        *p1 = x[r].a;
        *p2 = x[r].b;
      }
    } else {
      if (p1) {
#pragma unroll
        for (int r = 0; r < R; ++r, p1 += inner)
          if (r < cnt) *p1 = x[r].a;
      }
      if (p2) {
#pragma unroll
        for (int r = 0; r < R; ++r, p2 += inner)
          if (r < cnt) *p2 = x[r].b;
      }
    }
  } else if constexpr (EPI == kChunkCorrector) {
    // the operands of half a chunk first, then its stores (the output may be
    // u*, so a load cannot pass an earlier node's store)
    const T* pu = static_cast<const T*>(a.cr_u) + o0;
    const T* pr = static_cast<const T*>(a.cr_rho) + o0;
    T* p = static_cast<T*>(a.cr_out) + o0;
    constexpr int H = R / 2;
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += H) {
      T u[H], rho[H];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int r = r0 + i;
        u[i] = r < cnt ? pu[(int64_t)r * inner] : T(0);
        rho[i] = r < cnt ? pr[(int64_t)r * inner] : T(1);
      }
#pragma unroll
      for (int i = 0; i < H; ++i, p += inner) {
        const int r = r0 + i, k = k0 + r;
        if (r < cnt) {
          double o1 = (double)x[r].a, v = (double)u[i];
          if (J) o1 = J[k] * o1;
          if (!(a.cr_wall && (k == 0 || k == n - 1))) v = __dsub_rn(v, __dmul_rn(a.cr_dt / (double)rho[i], o1));
          *p = (T)v;
        }
      }
    }
  } else if constexpr (EPI == kChunkVd) {
    const T* pr = static_cast<const T*>(a.vd_rho) + o0;
    const T* pd = static_cast<const T*>(a.vd_drho) + o0;
    T* po = static_cast<T*>(a.vd_out) + o0;
    constexpr int H = R / 4;   // operands of a quarter first
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += H) {
      T rho[H], dr[H], acc[H];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int r = r0 + i;
        rho[i] = r < cnt ? pr[(int64_t)r * inner] : T(1);
        dr[i] = r < cnt ? pd[(int64_t)r * inner] : T(0);
        acc[i] = r < cnt && a.vd_accumulate ? po[(int64_t)i * inner] : T(0);
      }
#pragma unroll
      for (int i = 0; i < H; ++i, po += inner) {
        const int r = r0 + i, k = k0 + r;
        if (r < cnt) {
          double o1 = (double)x[r].a, o2 = (double)x[r].b;
          if (J) {
            const double Jk = J[k], dJk = J[n + k];
            o2 = Jk * Jk * o2 + Jk * dJk * o1;
            o1 = Jk * o1;
          }
          const double rr = (double)rho[i];
          double v = o2 / rr - ((double)dr[i] / (rr * rr)) * o1;
          if (a.vd_accumulate) v = (double)acc[i] + v;
          *po = (T)v;
        }
      }
    }
  } else {
    T* p1 = a.d1 ? static_cast<T*>(a.d1) + o0 : nullptr;
    T* p2 = a.d2 ? static_cast<T*>(a.d2) + o0 : nullptr;
    constexpr int H = R / 4;   // J of a quarter first: 193^3 67 -> 51 us, 65^2 10.4 -> 7.1
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += H) {
      double Jr[H], dJr[H];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int k = r0 + i < cnt ? k0 + r0 + i : 0;
        Jr[i] = J[k];
        dJr[i] = J[n + k];
      }
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const int r = r0 + i;
        if (r < cnt) {
          const double o1 = (double)x[r].a, o2 = (double)x[r].b;
          if (p1) p1[(int64_t)r * inner] = (T)(Jr[i] * o1);
          if (p2) p2[(int64_t)r * inner] = (T)(Jr[i] * Jr[i] * o2 + Jr[i] * dJr[i] * o1);
        }
      }
    }
  }
  if (q == 0) {   // the wall node, or the image node N = node 0
    const V2<double> v = PERIODIC ? V2<double>{(double)x[0].a, (double)x[0].b} : chunk_edge(K.Ml, x[0], bl0, bl1);
    put(PERIODIC ? n - 1 : 0, v.a, v.b);
  }
  if (!PERIODIC && last) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r == cnt - 1) {
        const V2<double> v = chunk_edge(K.Mr, x[r], br0, br1);
        put(n - 1, v.a, v.b);
      }
  }
}

// f at the nodes of a chunk (v(k): node k of the line) and the closures.
template <typename T, int R, bool PERIODIC, typename V>
__device__ __forceinline__ void chunk_load(const CcdArgs& a, const ChunkConst<T, R>& K, const V* f, int64_t step,
                                           int q, bool last, int cnt, T (&fv)[R + 2], double& bl0, double& bl1,
                                           double& br0, double& br1) {
  const int j0 = q * R;
  if (PERIODIC) {
    fv[0] = f[(int64_t)(q == 0 ? a.n_rows - 1 : j0 - 1) * step];
    const V* end = f + (last ? 0 : (int64_t)(j0 + R) * step);   // the node after the rows
    const V* p = f + (int64_t)j0 * step;
    if (cnt == R) {
#pragma unroll
      for (int i = 1; i < R + 1; ++i, p += step) fv[i] = *p;
      fv[R + 1] = *end;
    } else {
#pragma unroll
      for (int i = 1; i < R + 2; ++i, p += step) fv[i] = *(i <= cnt ? p : end);
    }
  } else {
    const V* p = f + (int64_t)j0 * step;
    if (cnt == R) {
#pragma unroll
      for (int i = 0; i < R + 2; ++i, p += step) fv[i] = *p;
    } else {
#pragma unroll
      for (int i = 0; i < R + 2; ++i, p += step) fv[i] = *(i < cnt + 2 ? p : f);
    }
    if (q == 0) {
      if (a.ovl) { bl0 = a.bcl0; bl1 = a.bcl1; }
      else chunk_closure(K.cIl, K.cII, f, step, bl0, bl1);
    }
    if (last) {
      if (a.ovr) { br0 = a.bcr0; br1 = a.bcr1; }
      else chunk_closure(K.cIr, K.cII, f + (int64_t)(a.n - 1) * step, -step, br0, br1);
    }
  }
}

enum { kChunkDirect = 0, kChunkStride = 1, kChunkSteal = 2 };

// Tiles dealt out as blocks become free (kChunkSteal): the launch has a block per
// tile, and a running block asks for the first one that has not started to be
// cancelled and solves its tile instead (cluster launch control).  Like
// a fixed stride through the tiles this lets a block copy its next tile early,
// but the tiles in work stay next to each other.  With the stride the SMs drift
// apart, and neighbouring tiles, which share the sectors at the ends of their
// rows and the pages the rows lie in, no longer meet in the caches: fields of more
// than 2 GB in and out took a third longer a node on axis 0 (periodic 417^3
// 5.7 ns, 449^3 7.4; 5.4 dealt out).
__device__ __forceinline__ void steal_ask(uint4* answer, unsigned long long* bar) {
  const unsigned int b = (unsigned int)__cvta_generic_to_shared(bar);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the last answer has been read
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;" ::"r"(b) : "memory");
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   (unsigned int)__cvta_generic_to_shared(answer)),
               "r"(b)
               : "memory");
}
__device__ __forceinline__ bool steal_arrived(unsigned long long* bar, unsigned int phase) {
  unsigned int ok;
  asm volatile("{\n .reg .pred w;\n mbarrier.try_wait.parity.shared::cta.b64 w, [%1], %2;\n selp.u32 %0, 1, 0, w;\n}"
               : "=r"(ok)
               : "r"((unsigned int)__cvta_generic_to_shared(bar)), "r"(phase)
               : "memory");
  return ok != 0;
}
// the tile taken over, -1: none was left
__device__ __forceinline__ int steal_answer(const uint4* answer) {
  int tile;
  asm volatile(
      "{\n .reg .pred w;\n .reg .b128 h;\n ld.shared.b128 h, [%1];\n mov.u32 %0, -1;\n"
      " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 w, h;\n"
      " @w clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, h;\n}"
      : "=r"(tile)
      : "r"((unsigned int)__cvta_generic_to_shared(answer))
      : "memory");
  return tile;
}
constexpr int kStealSpins = 1 << 22;   // polls of an answer, each up to some microseconds

// Strided axes: thread (l, q) = q TL + l of a block owns chunk q of line
// L0 + l (lanes on adjacent lines).  STAGE: a block has one tile of TL lines and a
// thread loads its rows straight into registers, or a block takes several tiles in
// turn, by a fixed stride or dealt out, and copies the next tile's f into shared
// memory while it solves the present one.  POW2: TL is a power of two (the
// division by any other TL costs a block's start 2 %, FP32 epilogues 6-9 %).
// THREADS: most threads of a block, 512 or (FP32, 64 registers a thread) 1024.
template <typename T, int R, bool PERIODIC, int EPI, int STAGE, bool POW2, int THREADS>
__global__ void __launch_bounds__(THREADS)
    ccd_chunk_strided_kernel(const __grid_constant__ CcdArgs a, const __grid_constant__ ChunkConst<T, R> K,
                             const T* __restrict__ gtab, int Q) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool STAGED = STAGE != kChunkDirect, STEAL = STAGE == kChunkSteal;
  const int t = threadIdx.x, TL = a.TL;
  const int q = POW2 ? t >> a.tl_shift : t * a.tl_inv >> 16, l = POW2 ? t & (TL - 1) : t - q * TL;
  T* G = reinterpret_cast<T*>(smem_raw);
  T* e = G + 4 * (kChunkHead + R);
  T* poison = e + 4 * blockDim.x;   // [TL]
  T* fs = poison + TL;              // STAGED: [n][TL]
  const int n = a.n;
  const int64_t inner = a.inner;
  const int cnt = min(R, a.n_rows - q * R);
  const bool last = q == Q - 1;
  if (!PERIODIC)
    for (int i = t; i < 4 * (kChunkHead + R); i += blockDim.x) G[i] = gtab[i];
  // element 0 of this thread's line in a tile, < 0: no line
  auto base_of = [&](int tile) -> int64_t {
    const int64_t L = (int64_t)tile * TL + l;
    if (L >= a.n_lines) return -1;
    const unsigned o = (unsigned)L / (unsigned)inner;
    return (int64_t)o * n * inner + (L - (int64_t)o * inner);
  };
  // rows q, q + rows, ... of the thread's line (idle threads of the block take part)
  const int rows = POW2 ? (int)blockDim.x >> a.tl_shift : (int)blockDim.x * a.tl_inv >> 16;
  auto fetch = [&](int64_t b) {
    if (b >= 0 && (POW2 || q < rows)) {
      const T* src = static_cast<const T*>(a.f) + b + (int64_t)q * inner;
      const int64_t step = (int64_t)rows * inner;
      for (int k = q; k < n; k += rows, src += step) cp_async<sizeof(T)>(fs + k * TL + l, src, true);
    }
    cp_async_commit();
  };
  int tile = blockIdx.x;
  int64_t base = base_of(tile);
  __shared__ uint4 next_answer;
  __shared__ __align__(8) unsigned long long next_bar;
  unsigned int phase = 0;
  if (STAGED) {
    if (STEAL && t == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned int)__cvta_generic_to_shared(&next_bar))
                   : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      steal_ask(&next_answer, &next_bar);
    }
    fetch(base);
  }
  for (;;) {
    const bool act = q < Q && base >= 0;
    T fv[R + 2];
    double bl0 = 0.0, bl1 = 0.0, br0 = 0.0, br1 = 0.0;
    if (STAGED) {
      cp_async_wait<0>();
      __syncthreads();
    }
    if (act) {
      if (STAGED) chunk_load<T, R, PERIODIC>(a, K, fs + l, TL, q, last, cnt, fv, bl0, bl1, br0, br1);
      else chunk_load<T, R, PERIODIC>(a, K, static_cast<const T*>(a.f) + base, inner, q, last, cnt, fv, bl0, bl1, br0, br1);
    } else {
#pragma unroll
      for (int i = 0; i < R + 2; ++i) fv[i] = T(0);
    }
    int next = tile + gridDim.x;
    int64_t nbase = -1;
    if constexpr (STEAL) {
      bool in = false;
      for (int spins = 0; spins < kStealSpins && !in; ++spins) in = steal_arrived(&next_bar, phase);
      phase ^= 1u;
      next = in ? steal_answer(&next_answer) : -1;
      if (__syncthreads_or(!in)) {   // every thread has its rows, and the answer
        // none came: these lines become NaN from end to end, and the block ends
        // once the answer is in, or after as long again
        fv[1] = T(NAN);
        for (int spins = 0; spins < kStealSpins && !steal_arrived(&next_bar, phase ^ 1u); ++spins) {}
        next = -1;
      }
      if (next >= 0) {
        nbase = base_of(next);
        fetch(nbase);
        if (t == 0) steal_ask(&next_answer, &next_bar);
      }
    } else if (STAGED && next < a.n_tiles) {
      nbase = base_of(next);
      __syncthreads();   // every thread has its rows
      fetch(nbase);
    }
    V2<T> x[R];
    chunk_solve<T, R, PERIODIC>(K, fv, q, Q, cnt, bl0, bl1, br0, br1, e, blockDim.x, t, TL, poison + l, G, x);
    if (act) chunk_store<T, R, PERIODIC, EPI>(a, K, x, base, inner, q, last, cnt, bl0, bl1, br0, br1);
    if (!STAGED || (STEAL ? next < 0 : next >= a.n_tiles)) return;
    tile = next;
    base = nbase;
  }
}

// The contiguous axis: a block's TL lines are one run of memory, staged
// through shared memory both ways; threads as on the strided axes (lanes on
// adjacent lines), so that only the warps of the first and last chunks pay for
// the walls.  The lines' pitch in shared memory is n, or n + 1 where n would
// make a warp's accesses collide in the banks; with a pitch of n the run is
// copied in 16-byte pieces where it starts on 16 bytes (`vec`).
template <typename T, int R, bool PERIODIC, bool PLAIN>
__global__ void __launch_bounds__(512, PLAIN ? 0 : 8 / sizeof(T))
    ccd_chunk_contig_kernel(const __grid_constant__ CcdArgs a, const __grid_constant__ ChunkConst<T, R> K,
                            const T* __restrict__ gtab, int Q, int pitch, int vec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x, TL = a.TL, n = a.n;
  const int q = t >> a.tl_shift, l = t & (TL - 1);
  const int tile_len = (TL * pitch + 3) & ~3;
  T* s1 = reinterpret_cast<T*>(smem_raw);          // f, then d1 [TL][pitch]
  T* s2 = s1 + tile_len;                           // d2 [TL][pitch]
  T* G = s2 + tile_len;
  T* e = G + 4 * (kChunkHead + R);
  T* poison = e + 4 * blockDim.x;                  // [TL]
  constexpr int VW = 16 / sizeof(T);
  const int64_t L0 = (int64_t)blockIdx.x * TL, g0 = L0 * n;
  const int nl = (int)min((int64_t)TL, a.n_lines - L0), tot = nl * n;
  const T* __restrict__ f = static_cast<const T*>(a.f) + g0;
  const int nv = vec ? tot / VW : 0;   // 16-byte pieces, then the rest
  // visit element i of the run as (line, node), i = t, t + threads, ...
  auto each = [&](int from, auto&& fn) {
    int i = from + t, ll = i / n, k = i - ll * n;
    const int dl = blockDim.x / n, dk = blockDim.x - dl * n;
    for (; i < tot; i += blockDim.x) {
      fn(i, ll * pitch + k, k);
      ll += dl;
      k += dk;
      if (k >= n) { k -= n; ++ll; }
    }
  };
  for (int i = t; i < nv; i += blockDim.x) cp_async<16>(s1 + i * VW, f + i * VW, true);
  each(nv * VW, [&](int i, int si, int) { cp_async<sizeof(T)>(s1 + si, f + i, true); });
  cp_async_commit();
  if (!PERIODIC)
    for (int i = t; i < 4 * (kChunkHead + R); i += blockDim.x) G[i] = gtab[i];
  const bool act = q < Q && l < nl, last = q == Q - 1;
  const int cnt = min(R, a.n_rows - q * R);
  T fv[R + 2];
  double bl0 = 0.0, bl1 = 0.0, br0 = 0.0, br1 = 0.0;
  T* sl1 = s1 + l * pitch;
  T* sl2 = s2 + l * pitch;
  cp_async_wait<0>();
  __syncthreads();
  if (act) {
    chunk_load<T, R, PERIODIC>(a, K, sl1, 1, q, last, cnt, fv, bl0, bl1, br0, br1);
  } else {
#pragma unroll
    for (int i = 0; i < R + 2; ++i) fv[i] = T(0);
  }
  V2<T> x[R];
  chunk_solve<T, R, PERIODIC>(K, fv, q, Q, cnt, bl0, bl1, br0, br1, e, blockDim.x, t, TL, poison + l, G, x);
  if (act) {   // f has been read by all (the barriers in between)
    const int k0 = q * R + (PERIODIC ? 0 : 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r < cnt) {
        sl1[k0 + r] = x[r].a;
        sl2[k0 + r] = x[r].b;
      }
      if (!PERIODIC && last && r == cnt - 1) {
        const V2<double> v = chunk_edge(K.Mr, x[r], br0, br1);
        sl1[n - 1] = (T)v.a;
        sl2[n - 1] = (T)v.b;
      }
    }
    if (q == 0) {
      const V2<double> v =
          PERIODIC ? V2<double>{(double)x[0].a, (double)x[0].b} : chunk_edge(K.Ml, x[0], bl0, bl1);
      const int k = PERIODIC ? n - 1 : 0;
      sl1[k] = (T)v.a;
      sl2[k] = (T)v.b;
    }
  }
  __syncthreads();
  if (PLAIN) {
    auto out = [&](void* dst, const T* src) {
      T* d = static_cast<T*>(dst) + g0;
      for (int i = t; i < nv; i += blockDim.x)
        __stcs(reinterpret_cast<float4*>(d) + i, reinterpret_cast<const float4*>(src)[i]);
      each(nv * VW, [&](int i, int si, int) { __stcs(d + i, src[si]); });
    };
    if (a.d1) out(a.d1, s1);
    if (a.d2) out(a.d2, s2);
  } else {
    const double* __restrict__ J = a.J;
    auto metric = [&](int k, double& o1, double& o2) {
      if (J) {
        const double Jk = J[k], dJk = J[n + k];
        o2 = Jk * Jk * o2 + Jk * dJk * o1;
        o1 = Jk * o1;
      }
    };
    if (!a.cr_out && !a.vd_out) {
      each(0, [&](int i, int si, int k) {
        double o1 = (double)s1[si], o2 = (double)s2[si];
        metric(k, o1, o2);
        if (a.d1) static_cast<T*>(a.d1)[g0 + i] = (T)o1;
        if (a.d2) static_cast<T*>(a.d2)[g0 + i] = (T)o2;
      });
      return;
    }
    // The operands of a batch of elements first, then its stores (the output may
    // be an operand, so a load cannot pass an earlier element's store, and the
    // few threads of a small field would wait for every load by itself: 65^2
    // corrector 12.6 -> 8.8 us, variable-density term 16.1 -> 9.9, 193^3 130 -> 69
    // and 187 -> 79).
    constexpr int E = sizeof(T) == 4 ? 4 : 8;   // FP32: two blocks of 64 registers a thread
    const T* pa = static_cast<const T*>(a.cr_out ? a.cr_u : a.vd_rho) + g0;
    const T* pb = static_cast<const T*>(a.cr_out ? a.cr_rho : a.vd_drho) + g0;
    T* po = static_cast<T*>(a.cr_out ? a.cr_out : a.vd_out) + g0;
    const bool acc = a.vd_out && a.vd_accumulate;
    int ll = t / n, k = t - ll * n;
    const int dl = blockDim.x / n, dk = blockDim.x - dl * n;
    for (int i0 = t; i0 < tot; i0 += E * blockDim.x) {
      T ua[E], ub[E], uc[E];
      int kk[E], si[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int i = i0 + e * blockDim.x;
        kk[e] = k;
        si[e] = ll * pitch + k;
        if (i < tot) {
          ua[e] = pa[i];
          ub[e] = pb[i];
          uc[e] = acc ? po[i] : T(0);
        }
        ll += dl;
        k += dk;
        if (k >= n) { k -= n; ++ll; }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int i = i0 + e * blockDim.x;
        if (i >= tot) break;
        double o1 = (double)s1[si[e]], o2 = (double)s2[si[e]], v = (double)ua[e];
        const double b = (double)ub[e];
        metric(kk[e], o1, o2);
        if (a.cr_out) {
          if (!(a.cr_wall && (kk[e] == 0 || kk[e] == n - 1))) v = __dsub_rn(v, __dmul_rn(a.cr_dt / b, o1));
        } else {
          v = o2 / v - (b / (v * v)) * o1;
          if (acc) v = (double)uc[e] + v;
        }
        po[i] = (T)v;
      }
    }
  }
}

}  // namespace
