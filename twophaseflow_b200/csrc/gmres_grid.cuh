// Restarted GMRES of a 2-D system in one launch (included by ppe.cu).
//
// The algorithm of gmres.cuh (SciPy's left-preconditioned gmres with its
// inner-tolerance control, classical Gram-Schmidt with a conditional second
// pass), run start to end by one cooperative grid.
//
// What bounds it: a column of a small system is a handful of dependent steps
// of well under a microsecond of work each.  As kernels (operator, two line
// solves, three Gram-Schmidt kernels, scaling: 7 launches chained by
// programmatic launches and replayed from a graph) a column took 60 us at 64^2,
// almost all of it launches, last-block reductions and their fences.  Here a
// block keeps a few grid rows, its part of the basis (in shared memory where
// the whole cycle fits), its line factors and a copy of the Hessenberg matrix;
// what blocks exchange -- edge rows, transposed fields for the line solves
// across rows, partial inner products -- travels as FlagSlots (a value and its
// epoch, polled by the reader), about 1 us a step and five to six steps a
// column.  Every block sums the same partials in the same order, so all take
// the same decisions without being told.  The Givens rotations of a column, a
// serial chain, run in the last warp while the others wait for the next
// column's line solutions.
//
// Measured per column, restart 80, line preconditioner (kernels of gmres.cuh ->
// here): 33^2 56.8 -> 14.1 us, 65^2 58.7 -> 13.2 us, 129 x 97 65.4 -> 13.1 us,
// 201^2 81.0 -> 22.8 us (basis in global memory).
#pragma once

namespace {

constexpr int kGgThreads = 288, kGgWarps = kGgThreads / 32;   // two rows of 129 nodes, four of 65
constexpr int kGgMaxGrid = 148;
constexpr int kGgLane[5] = {2, 3, 5, 9, 17};   // rows per lane of a line solve: lines of up to 544 nodes

struct GmresGridOut {
  long long inner, applies;
  double bnrm2, rnorm;
  int converged, pad;
};

struct GmresGridArgs {
  Grid3 g;
  Geo geo;
  const double *s0, *s1;        // face couplings
  const double *lo[2], *den[2], *cp[2];   // Thomas factors per axis
  const double* dinvL;
  int precond;
  const double* b;              // right-hand side, 0 at the pin
  double* x;                    // x0 in, solution out
  double* V;                    // basis [m][n]; unused where it is in shared memory
  FlagSlot *wt, *zt;            // [2][n]: operator output / column solutions
  FlagSlot* edges;              // [2][G][2][n1]: first / last row of a block
  FlagSlot* dots;               // [2][G][ld]: partial inner products
  int ld;                       // m + 2 rounded up to whole lines
  int* err;
  GmresGridOut* out;
  double tol;
  long long maxiter;
  int m, rows, x_nonzero;
  int k;                        // rows per lane of a line: one of kGgLane
};

// shared-memory doubles besides the basis
inline size_t gg_smem_doubles(int n0, int n1, int rows, int G, int m, bool line) {
  const size_t nb = (size_t)rows * n1, ncol = (size_t)(n1 + G - 1) / G + 1;
  const size_t ld = ((size_t)m + 2 + 7) / 8 * 8;
  return (size_t)(rows + 2) * n1 + 4 * nb + (size_t)m * (m + 1) / 2 + 2 * (size_t)m + 4 * ((size_t)m + 2) +
         kGgWarps * ld + 32 + (line ? 3 * (rows * (size_t)n1 + ncol * (size_t)n0) : 0);
}

// T^-1 r along one line by one warp: lane l holds rows [l K, l K + K).  f: the
// line's factors {1 / den, lo / den, c'} in shared memory.  Both sweeps are
// affine recurrences, composed per lane, scanned over the warp and then rerun
// from the value that enters the lane, as in thomas_warp_line, with the
// divisions by den made once per solve.
template <int K>
__device__ __forceinline__ void gg_line(const double* f, int n, int lane, double (&r)[K]) {
  const unsigned m = 0xffffffffu;
  const int i0 = lane * K;
  double A = 1.0, B = 0.0;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int i = i0 + q;
    if (i < n) {
      const double mi = f[3 * i + 1];
      r[q] *= f[3 * i];
      B = fma(-mi, B, r[q]);
      A *= -mi;
    }
  }
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const double Ap = __shfl_up_sync(m, A, s), Bp = __shfl_up_sync(m, B, s);
    if (lane >= s) {
      B = fma(A, Bp, B);
      A *= Ap;
    }
  }
  double y = __shfl_up_sync(m, B, 1);
  if (lane == 0) y = 0.0;
  double C = 1.0, D = 0.0;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int i = i0 + q;
    if (i < n) {
      y = fma(-f[3 * i + 1], y, r[q]);
      r[q] = y;
    }
  }
#pragma unroll
  for (int q = K - 1; q >= 0; --q) {
    const int i = i0 + q;
    if (i < n) {
      const double c = f[3 * i + 2];   // 0 on the last row
      D = fma(-c, D, r[q]);
      C *= -c;
    }
  }
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const double Cn = __shfl_down_sync(m, C, s), Dn = __shfl_down_sync(m, D, s);
    if (lane + s < 32) {
      D = fma(C, Dn, D);
      C *= Cn;
    }
  }
  double xx = __shfl_down_sync(m, D, 1);
  if (lane == 31) xx = 0.0;
#pragma unroll
  for (int q = K - 1; q >= 0; --q) {
    const int i = i0 + q;
    if (i < n) {
      xx = fma(-f[3 * i + 2], xx, r[q]);
      r[q] = xx;
    }
  }
}

// One polled slot per index [0, count): p(i) its address, got(i, value) called
// with what arrived; N polls of a thread in flight at a time.  Bounded.
template <int N, typename P, typename F>
__device__ __forceinline__ bool gg_poll(int first, int step, int count, unsigned int tag, int* err, P&& p, F&& got) {
  bool ok = true;
  for (int i0 = first; i0 < count && ok; i0 += N * step) {
    FlagSlot q[N];
    unsigned need = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      q[k] = {0, 0};
      if (i0 + k * step < count) need |= 1u << k;
    }
    for (long long spins = 0; need;) {
#pragma unroll
      for (int k = 0; k < N; ++k) slot_load(p(i0 + k * step), need & (1u << k), q[k]);
#pragma unroll
      for (int k = 0; k < N; ++k)
        if (slot_ready(q[k], tag)) need &= ~(1u << k);
      if (++spins > kSpinLimit) { atomicExch(err, 1); ok = false; break; }
      if ((spins & 1023) == 0 && *(volatile int*)err) { ok = false; break; }
    }
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (i0 + k * step < count) got(i0 + k * step, slot_value(q[k]));
  }
  return ok;
}

// givens_rot by one square root and one division where f^2 + g^2 is safe
__device__ __forceinline__ void gg_givens(double f, double g, double& c, double& s, double& r) {
  const double ff = fabs(f), gg = fabs(g);
  if (!(ff > 1e-140 && ff < 1e140 && gg > 1e-140 && gg < 1e140)) {
    givens_rot(f, g, c, s, r);
    return;
  }
  const double d = sqrt(fma(f, f, g * g)), inv = 1.0 / d;
  c = ff * inv;
  r = copysign(d, f);
  s = g * copysign(inv, f);
}

// VS: the basis is in shared memory
template <bool VS>
__global__ void __launch_bounds__(kGgThreads, 1) gmres_grid_kernel(const __grid_constant__ GmresGridArgs a) {
  extern __shared__ __align__(16) unsigned char gg_smem[];
  const Grid3& g = a.g;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, bid = blockIdx.x, G = gridDim.x;
  const int n = g.ndof, n0 = g.n0, n1 = g.n1, m = a.m, ld = a.ld;
  const int row0 = bid * a.rows, rows = min(a.rows, n0 - row0), nb = rows * n1, base = row0 * n1, NB = a.rows * n1;
  const int col0 = (int)((long long)bid * n1 / G), ncol = (int)((long long)(bid + 1) * n1 / G) - col0;
  const int ncol_max = (n1 + G - 1) / G + 1;
  const bool line = a.precond == TPF_PRECOND_LINE;
  double* giv = reinterpret_cast<double*>(gg_smem);  // (cos, sin) of the columns' rotations
  double* vh = giv + 2 * m;                          // a field with a halo row either side [rows + 2][n1]
  double* w = vh + (size_t)(a.rows + 2) * n1;        // own nodes
  double* z = w + NB;
  double* zr = z + NB;
  double* R = zr + NB;                               // Hessenberg columns, rotated: column j at j (j + 1) / 2
  double* S = R + (size_t)m * (m + 1) / 2;
  double* yv = S + (m + 2);
  double* h1c = yv + (m + 2);                        // the column's coefficients
  double* tot = h1c + (m + 2);                       // totals of an exchange
  double* part = tot + (m + 2);                      // [warps][ld]
  double* red = part + kGgWarps * ld;                // 32
  double* iw = red + 32;                             // 1 / control volume of the own nodes
  double* fac = iw + NB;                             // line factors: rows, then columns
  double* V = VS ? fac + (line ? 3 * ((size_t)a.rows * n1 + (size_t)ncol_max * n0) : 0) : a.V + base;
  const size_t ldv = VS ? (size_t)NB : (size_t)n;
  __shared__ int s_flag[2];                          // the cycle has ended; it ended by breakdown
  __shared__ double s_num[4];                        // scale of the new basis vector, its norm, presid

  if (line) {
    for (int i = t; i < rows * n1; i += kGgThreads) {
      const double inv = 1.0 / a.den[1][base + i];
      fac[3 * i] = inv;
      fac[3 * i + 1] = i % n1 == 0 ? 0.0 : a.lo[1][base + i] * inv;
      fac[3 * i + 2] = i % n1 == n1 - 1 ? 0.0 : a.cp[1][base + i];
    }
    double* fc = fac + 3 * (size_t)a.rows * n1;
    for (int i = t; i < ncol * n0; i += kGgThreads) {
      const int c = i / n0, k = i - c * n0, e = k * n1 + col0 + c;
      const double inv = 1.0 / a.den[0][e];
      fc[3 * i] = inv;
      fc[3 * i + 1] = k == 0 ? 0.0 : a.lo[0][e] * inv;
      fc[3 * i + 2] = k == n0 - 1 ? 0.0 : a.cp[0][e];
    }
  }
  for (int i = t; i < nb; i += kGgThreads) iw[i] = 1.0 / (a.geo.dv[0][row0 + i / n1] * a.geo.dv[1][i % n1]);
  unsigned int ep = 0;
  bool ok = true;
  unsigned int n_dots = 0, n_edges = 0, n_pre = 0;   // uses of the buffers so far
  auto agree = [&] { ok = __syncthreads_and(ok) != 0; };

  // ---- exchanges ------------------------------------------------------------------
  auto put_edges = [&](const double* f, unsigned int tag) {   // f: own nodes
    FlagSlot* e = a.edges + ((size_t)(n_edges & 1) * G + bid) * 2 * n1;
    for (int i = t; i < 2 * n1; i += kGgThreads)
      slot_store(e + i, i < n1 ? f[i] : f[nb - n1 + (i - n1)], tag);
  };
  // entry i of the halo rows of vh: n1 nodes before the block's rows, n1 after
  auto edge_slot = [&](int i) -> const FlagSlot* {
    const FlagSlot* e = a.edges + (size_t)(n_edges & 1) * G * 2 * n1;
    return i < n1 ? e + ((size_t)(bid - 1) * 2 + 1) * n1 + i : e + (size_t)(bid + 1) * 2 * n1 + (i - n1);
  };
  auto edge_live = [&](int i) { return i < 2 * n1 && (i < n1 ? bid > 0 : bid < G - 1); };
  auto edge_set = [&](int i, double v) { vh[i < n1 ? i : rows * n1 + i] = v; };
  // halo entries from `first` on, into vh
  auto get_edges = [&](int first, unsigned int tag) {
    for (int i = first; i < 2 * n1; i += kGgThreads) {
      FlagSlot q{0, 0};
      bool need = edge_live(i);
      for (long long spins = 0; need && ok;) {
        slot_load(edge_slot(i), true, q);
        need = !slot_ready(q, tag);
        if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; }
        if ((spins & 1023) == 0 && *(volatile int*)a.err) ok = false;
      }
      edge_set(i, slot_value(q));   // outside the domain: 0
    }
    ++n_edges;
  };
  // totals of `nt` per-block values, published by put(j, value), into tot
  auto put_dot = [&](int j, double v, unsigned int tag) {
    slot_store(a.dots + ((size_t)(n_dots & 1) * G + bid) * ld + j, v, tag);
  };
  auto get_dots = [&](int nt, unsigned int tag) {
    const FlagSlot* d = a.dots + (size_t)(n_dots & 1) * G * ld;
    // warp w: blocks w, w + warps, ...; a lane the values j, j + 32, j + 64,
    // four blocks' worth of polls in flight
    for (int j0 = lane; j0 - lane < nt; j0 += 96) {
      double s[3] = {0.0, 0.0, 0.0};
      for (int b0 = wid; b0 < G; b0 += 4 * kGgWarps) {
        FlagSlot q[12];
        unsigned need = 0;
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          q[k] = {0, 0};
          if (b0 + (k / 3) * kGgWarps < G && j0 + 32 * (k % 3) < nt) need |= 1u << k;
        }
        const FlagSlot* p = d + (size_t)b0 * ld + j0;
        for (long long spins = 0; need && ok;) {
#pragma unroll
          for (int k = 0; k < 12; ++k)
            slot_load(p + (size_t)(k / 3) * kGgWarps * ld + 32 * (k % 3), need & (1u << k), q[k]);
#pragma unroll
          for (int k = 0; k < 12; ++k)
            if (slot_ready(q[k], tag)) need &= ~(1u << k);
          if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; }
          if ((spins & 1023) == 0 && *(volatile int*)a.err) ok = false;
        }
#pragma unroll
        for (int k = 0; k < 12; ++k) s[k % 3] += slot_value(q[k]);   // a slot not asked for reads as 0
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (j0 + 32 * k < nt) part[wid * ld + j0 + 32 * k] = s[k];
    }
    agree();
    for (int j = t; j < nt; j += kGgThreads) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < kGgWarps; ++k) s += part[k * ld + j];
      tot[j] = s;
    }
    ++n_dots;
    __syncthreads();
  };
  // sqrt of the total of a per-thread value (one slot per block); edges of f ride along (NULL: none)
  auto norm = [&](double v, const double* f) -> double {
    ++ep;
    if (f) put_edges(f, ep);
    v = tpf::warp_sum(v);
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (t == 0) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < kGgWarps; ++k) s += red[k];
      put_dot(0, s, ep);
    }
    // one block's sum and the first two halo entries of this thread in one wait
    const FlagSlot* d = a.dots + (size_t)(n_dots & 1) * G * ld + (size_t)t * ld;
    FlagSlot q[3] = {{0, 0}, {0, 0}, {0, 0}};
    unsigned need = t < G ? 1u : 0u;
    if (f && edge_live(t)) need |= 2u;
    if (f && edge_live(t + kGgThreads)) need |= 4u;
    for (long long spins = 0; need && ok;) {
      slot_load(d, need & 1u, q[0]);
      slot_load(edge_slot(t), need & 2u, q[1]);
      slot_load(edge_slot(t + kGgThreads), need & 4u, q[2]);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (slot_ready(q[k], ep)) need &= ~(1u << k);
      if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; }
      if ((spins & 1023) == 0 && *(volatile int*)a.err) ok = false;
    }
    ++n_dots;
    if (f) {
      if (t < 2 * n1) edge_set(t, slot_value(q[1]));
      if (t + kGgThreads < 2 * n1) edge_set(t + kGgThreads, slot_value(q[2]));
      get_edges(t + 2 * kGgThreads, ep);
    }
    __syncwarp();
    double s = tpf::warp_sum(slot_value(q[0]));
    if (lane == 0) red[16 + wid] = s;
    agree();
    s = 0.0;
#pragma unroll
    for (int k = 0; k < kGgWarps; ++k) s += red[16 + k];
    __syncthreads();
    return sqrt(s);
  };

  // ---- operator, residual and preconditioner ---------------------------------------
  // (L v)_i of own node i of the field in vh
  auto apply = [&](int i) -> double {
    const int idx = base + i, i0 = row0 + i / n1, i1 = i - (i / n1) * n1;
    const double v = vh[n1 + i];
    if (idx == g.pin) return v;
    const double sm0 = i0 > 0 ? __ldg(a.s0 + idx - n1) : 0.0, sp0 = __ldg(a.s0 + idx);
    const double sm1 = i1 > 0 ? __ldg(a.s1 + idx - 1) : 0.0, sp1 = __ldg(a.s1 + idx);
    const double d = (sm0 + sp0) + (sm1 + sp1);
    // neighbours outside the domain: their couplings are 0, the values read are finite
    const double off = sm0 * vh[i] + sp0 * vh[2 * n1 + i] + sm1 * vh[i1 > 0 ? n1 + i - 1 : n1 + i] +
                       sp1 * vh[i1 < n1 - 1 ? n1 + i + 1 : n1 + i];
    return (off - d * v) * iw[i];
  };
  // z = M w; w complete in every thread's view (a barrier before), z so on return.
  // For the line solves w goes out to the blocks that own its columns.  `aside`
  // runs in the last warp while the columns' solutions travel back.
  auto precondition = [&](auto&& aside) {
    if (!line) {
      if (wid == kGgWarps - 1) aside();
      for (int i = t; i < nb; i += kGgThreads) {
        const int idx = base + i;
        z[i] = a.precond == TPF_PRECOND_JACOBI ? (idx == g.pin ? 0.0 : w[i] * a.dinvL[idx]) : w[i];
      }
      __syncthreads();
      return;
    }
    ++ep;
    FlagSlot* wt = a.wt + (size_t)(n_pre & 1) * n;
    FlagSlot* zt = a.zt + (size_t)(n_pre & 1) * n;
    ++n_pre;
    for (int i = t; i < nb; i += kGgThreads) slot_store(wt + base + i, base + i == g.pin ? 0.0 : w[i], ep);
    auto lines = [&](auto kk) {
      constexpr int K = decltype(kk)::value;
      const int i0 = lane * K;
      for (int li = wid; li < rows + ncol; li += kGgWarps) {
        double r[K];
        if (li < rows) {   // along the row: all of it is here
#pragma unroll
          for (int q = 0; q < K; ++q)
            r[q] = i0 + q < n1 && base + li * n1 + i0 + q != g.pin ? w[li * n1 + i0 + q] : 0.0;
          gg_line<K>(fac + 3 * (size_t)li * n1, n1, lane, r);
#pragma unroll
          for (int q = 0; q < K; ++q)
            if (i0 + q < n1) zr[li * n1 + i0 + q] = r[q];
        } else {           // a column: its values come from every block
          const int c = col0 + (li - rows);
          FlagSlot v[K];
          unsigned need = 0;
#pragma unroll
          for (int q = 0; q < K; ++q) {
            v[q] = {0, 0};
            if (i0 + q < n0) need |= 1u << q;
          }
          for (long long spins = 0; need && ok;) {
#pragma unroll
            for (int q = 0; q < K; ++q) slot_load(wt + (size_t)(i0 + q) * n1 + c, need & (1u << q), v[q]);
#pragma unroll
            for (int q = 0; q < K; ++q)
              if (slot_ready(v[q], ep)) need &= ~(1u << q);
            if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; }
            if ((spins & 1023) == 0 && *(volatile int*)a.err) ok = false;
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < K; ++q) r[q] = slot_value(v[q]);
          gg_line<K>(fac + 3 * ((size_t)a.rows * n1 + (size_t)(li - rows) * n0), n0, lane, r);
#pragma unroll
          for (int q = 0; q < K; ++q)
            if (i0 + q < n0) slot_store(zt + (size_t)(i0 + q) * n1 + c, r[q], ep);
        }
      }
    };
    switch (a.k) {
      case kGgLane[0]: lines(std::integral_constant<int, kGgLane[0]>{}); break;
      case kGgLane[1]: lines(std::integral_constant<int, kGgLane[1]>{}); break;
      case kGgLane[2]: lines(std::integral_constant<int, kGgLane[2]>{}); break;
      case kGgLane[3]: lines(std::integral_constant<int, kGgLane[3]>{}); break;
      default: lines(std::integral_constant<int, kGgLane[4]>{}); break;
    }
    __syncthreads();   // zr
    if (wid == kGgWarps - 1) aside();
    ok = ok && gg_poll<2>(t, kGgThreads, nb, ep, a.err, [&](int i) { return zt + base + i; },
                          [&](int i, double v) { z[i] = base + i == g.pin ? 0.0 : (v + zr[i]) * 0.5; });
    agree();
  };
  // partial inner products <V_j, z>, j < nv, and <z, z> (zz) of this block, published
  auto dots = [&](int nv, bool zz, unsigned int tag) {
    const int nt = nv + (zz ? 1 : 0);
    const unsigned msk = 0xffffffffu;
    for (int j0 = 8 * wid; j0 < nt; j0 += 8 * kGgWarps) {
      double acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.0;
      const double* v[8];   // <z, z> and the unused ones: z itself
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = j0 + q < nv ? V + (size_t)(j0 + q) * ldv : z;
#pragma unroll 2
      for (int i = lane; i < nb; i += 32) {
        const double zi = z[i];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fma(v[q][i], zi, acc[q]);
      }
      const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
      double x[4], y[2];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        x[q] = (h16 ? acc[q + 4] : acc[q]) + __shfl_xor_sync(msk, h16 ? acc[q] : acc[q + 4], 16);
#pragma unroll
      for (int q = 0; q < 2; ++q) y[q] = (h8 ? x[q + 2] : x[q]) + __shfl_xor_sync(msk, h8 ? x[q] : x[q + 2], 8);
      double s = (h4 ? y[1] : y[0]) + __shfl_xor_sync(msk, h4 ? y[0] : y[1], 4);
      s += __shfl_xor_sync(msk, s, 2);
      s += __shfl_xor_sync(msk, s, 1);
      const int j = j0 + (lane >> 2);
      if ((lane & 3) == 0 && j < nt) put_dot(j, s, tag);
    }
  };
  // z -= sum_j tot_j V_j (j < nv); the sum of squares of this thread's nodes
  auto update = [&](int nv) -> double {
    double ss = 0.0;
    for (int i = t; i < nb; i += kGgThreads) {
      double c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
      int j = 0;
      for (; j + 4 <= nv; j += 4) {
        c0 = fma(tot[j], V[(size_t)j * ldv + i], c0);
        c1 = fma(tot[j + 1], V[(size_t)(j + 1) * ldv + i], c1);
        c2 = fma(tot[j + 2], V[(size_t)(j + 2) * ldv + i], c2);
        c3 = fma(tot[j + 3], V[(size_t)(j + 3) * ldv + i], c3);
      }
      for (; j < nv; ++j) c0 = fma(tot[j], V[(size_t)j * ldv + i], c0);
      const double v = z[i] - ((c0 + c1) + (c2 + c3));
      z[i] = v;
      ss = fma(v, v, ss);
    }
    return ss;
  };
  auto square = [&](const double* f) -> double {
    double s = 0.0;
    for (int i = t; i < nb; i += kGgThreads) s = fma(f[i], f[i], s);
    return s;
  };
  // residual b - L x of the iterate into w; its norm
  auto residual = [&]() -> double {
    ++ep;
    for (int i = t; i < nb; i += kGgThreads) vh[n1 + i] = a.x[base + i];
    __syncthreads();
    put_edges(vh + n1, ep);
    get_edges(t, ep);
    agree();
    for (int i = t; i < nb; i += kGgThreads) w[i] = a.b[base + i] - apply(i);
    __syncthreads();
    return norm(square(w), nullptr);
  };

  // ---- the solve --------------------------------------------------------------------
  long long inner = 0, applies = 0;
  double rnorm = INFINITY;
  bool converged = false;
  for (int i = t; i < nb; i += kGgThreads) w[i] = a.b[base + i];
  __syncthreads();
  const double bnrm2 = norm(square(w), nullptr);
  auto finish = [&] {
    if (bid == 0 && t == 0) *a.out = {inner, applies, bnrm2, rnorm, converged ? 1 : 0, 0};
  };
  if (!ok) return;
  if (bnrm2 == 0.0) {
    for (int i = t; i < nb; i += kGgThreads) a.x[base + i] = 0.0;
    converged = true;
    rnorm = 0.0;
    finish();
    return;
  }
  const double atol = a.tol * bnrm2, eps = 2.220446049250313e-16;
  precondition([] {});
  const double mb = norm(square(z), nullptr);
  double factor = 1.0, ptol = mb * fmin(factor, atol / bnrm2);
  if (a.maxiter == 0) {
    // no cycle, and as in SciPy no look at the initial guess either
  } else if (ok && a.x_nonzero) {
    rnorm = residual();
    ++applies;
    converged = rnorm < atol;
  } else {
    // w = b still, and r0 = ||b|| < atol only where tol > 1
    converged = bnrm2 < atol;
    if (converged) rnorm = bnrm2;
  }
  for (long long cycle = 0; ok && !converged && cycle < a.maxiter; ++cycle) {
    // v0 = M r / ||M r||, with its edges
    precondition([] {});
    const double v0n = norm(square(z), z);
    if (!ok) break;
    double scal = 1.0 / v0n;
    for (int k = t; k < m + 1; k += kGgThreads) S[k] = k == 0 ? v0n : 0.0;
    if (t < 2) s_flag[t] = 0;
    int ncols = 0;
    __syncthreads();
    double h1 = 0.0, h0 = 0.0;   // norms of the column that waits for its Givens step
    for (int col = 0;; ++col) {
      // basis vector `col` from z, its halo rows scaled alike
      for (int i = t; i < nb; i += kGgThreads) {
        const double v = z[i] * scal;
        if (col < m) V[(size_t)col * ldv + i] = v;
        vh[n1 + i] = v;
      }
      for (int i = t; i < 2 * n1; i += kGgThreads) {
        double* e = i < n1 ? vh + i : vh + (rows + 1) * n1 + (i - n1);
        *e *= scal;
      }
      __syncthreads();
      for (int i = t; i < nb; i += kGgThreads) w[i] = apply(i);
      __syncthreads();
      // the Givens step of the column before runs beside this column's
      // preconditioner; where it ends the cycle, this column is dropped
      precondition([&] {
        if (col == 0) return;
        const int k = col - 1;
        double* hc = R + (size_t)k * (k + 1) / 2;
        const bool breakdown = h1 <= eps * h0;
        // all lanes run the chain on values fetched eight rotations ahead
        double cur = h1c[0];
        const double2* gv = reinterpret_cast<const double2*>(giv);
        auto rotate = [&](int j, double2 cs, double nx) {
          const double o = fma(cs.x, cur, cs.y * nx);
          cur = fma(-cs.y, cur, cs.x * nx);
          if (lane == 0) hc[j] = o;
        };
        int j = 0;
        for (; j + 8 <= k; j += 8) {
          double2 cs[8];
          double nx[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            cs[q] = gv[j + q];
            nx[q] = h1c[j + q + 1];
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) rotate(j + q, cs[q], nx[q]);
        }
        for (; j < k; ++j) rotate(j, gv[j], h1c[j + 1]);
        if (lane == 0) {
          double c, sn, mag;
          gg_givens(cur, breakdown ? 0.0 : h1, c, sn, mag);
          giv[2 * k] = c;
          giv[2 * k + 1] = sn;
          hc[k] = mag;
          const double ts = -sn * S[k];
          S[k] = c * S[k];
          S[k + 1] = ts;
          s_num[0] = fabs(ts);
          s_flag[0] = fabs(ts) <= ptol || breakdown || col == m ? 1 : 0;
          s_flag[1] = breakdown ? 1 : 0;
        }
        __syncwarp();
      });
      ncols = col;
      if (s_flag[0]) break;
      // first pass; all of h, ||w||
      ++ep;
      dots(col + 1, true, ep);
      get_dots(col + 2, ep);
      double proj = 0.0;
      for (int j = lane; j <= col; j += 32) proj = fma(tot[j], tot[j], proj);
      proj = tpf::warp_sum(proj);
      const double sw = tot[col + 1];
      h0 = sqrt(sw);
      const bool again = sw - proj < 0.5 * sw;
      for (int j = t; j <= col; j += kGgThreads) h1c[j] = tot[j];
      double ss = update(col + 1);
      if (again) {
        __syncthreads();
        ++ep;
        dots(col + 1, false, ep);
        get_dots(col + 1, ep);
        for (int j = t; j <= col; j += kGgThreads) h1c[j] += tot[j];
        ss = update(col + 1);
      }
      __syncthreads();
      h1 = norm(ss, z);
      if (!ok) break;
      scal = h1 <= eps * h0 ? 1.0 : 1.0 / h1;
      ++inner;
      ++applies;
    }
    if (!ok) break;
    const double presid = s_num[0];
    const bool breakdown = s_flag[1] != 0;
    // y = R^-1 S (column by column, as SciPy's trsv), x += V y
    const int last = ncols - 1;
    for (int k = t; k <= last; k += kGgThreads) yv[k] = S[k];
    __syncthreads();
    if (t < 32) {
      if (lane == 0 && R[(size_t)last * (last + 1) / 2 + last] == 0.0) yv[last] = 0.0;
      __syncwarp();
      for (int k = last; k > 0; --k) {
        const double* hc = R + (size_t)k * (k + 1) / 2;
        double yk = yv[k];
        if (yk != 0.0) {
          yk /= hc[k];
          __syncwarp();
          if (lane == 0) yv[k] = yk;
          for (int q = lane; q < k; q += 32) yv[q] -= yk * hc[q];
        }
        __syncwarp();
      }
      if (lane == 0 && yv[0] != 0.0) yv[0] /= R[0];
    }
    __syncthreads();
    for (int i = t; i < nb; i += kGgThreads) {
      double c0 = 0.0, c1 = 0.0;
      int j = 0;
      for (; j + 2 <= ncols; j += 2) {
        c0 = fma(yv[j], V[(size_t)j * ldv + i], c0);
        c1 = fma(yv[j + 1], V[(size_t)(j + 1) * ldv + i], c1);
      }
      if (j < ncols) c0 = fma(yv[j], V[(size_t)j * ldv + i], c0);
      a.x[base + i] += c0 + c1;
    }
    rnorm = residual();   // each thread reads back its own nodes of x
    ++applies;
    if (!ok) break;
    if (rnorm <= atol) { converged = true; break; }
    if (breakdown) break;
    if (presid <= ptol) factor = fmax(eps, 0.25 * factor);
    else factor = fmin(1.0, 1.5 * factor);
    ptol = presid * fmin(factor, atol / rnorm);
  }
  finish();
}

}  // namespace
