// FP64 Jacobi-PCG of systems too large to stay on chip (3-D grids, large 2-D
// ones) in one cooperative launch (included by ppe.cu).
//
// The textbook recurrences with SciPy's stopping rule, two passes an iteration:
//   A  p = z + beta p, w = S p, (p, w); x += alpha p of the iteration before
//   B  r -= alpha w, z = M r, (r, z), (r, r)
// Pass A marches: the (axis 1, axis 2) plane is cut into tiles of T <= 512
// consecutive columns, a unit is one tile of one plane, and a block takes a
// contiguous range of the units, tile by tile along axis 0.  A step brings the
// next plane's z and p (the tile and the columns a row of axis 2 to either
// side, where p is recomputed rather than exchanged), x and the couplings into
// a ring of shared-memory stages with bulk copies; p of a plane sits in
// shared memory for its in-plane neighbours and in registers for the planes
// above and below.  Pass B touches the block's own nodes only, so w stays in
// shared memory where the block's share fits, and what separates the passes is
// one sum over the grid each (FlagSlots; the one after B also publishes z and p).
// Per node and iteration 9 loads and 5 stores instead of the 11 and 6 of the
// two streaming kernels, and no launches between them.
//
// Measured (streaming kernels -> here, us an iteration): 129^3 66.3 -> 43.9 (the
// 112 B a node moves pass at 5.5 TB/s), 97^3 27.5 -> 19.9, 65^3 18.4 -> 11.0,
// 25^3 9.5 -> 7.5.  Small grids are bound by the two sums (2 us each with their
// fences) and by the steps' latency, about 0.5 us each.
#pragma once

namespace {

constexpr int kMarchT = 512;        // threads that compute, and most columns of a tile
constexpr int kMarchWarps = kMarchT / 32;
constexpr int kMarchGrid = 160;     // most blocks: three sums of each fit the polling threads
constexpr int kMarchBatch = 4;      // nodes a thread of pass B has in flight (97^3: 19.8 us; 6: 22.0, 8: 23.0)
constexpr int kMarchCopies = 6;     // fields of a step
constexpr int kMarchStages = 6;     // most stages

struct MarchArgs {
  Grid3 g;
  const double *s0, *s1, *s2;   // couplings to the next node per axis, 0 on the last
  const double* dinv;           // M, 1 at the pin
  const double* b;
  double *x, *r, *z, *w;
  double* p[2];
  FlagSlot* slots;              // [2 parity][G][kBandLine]
  int* err;
  SolveStatus* st;
  double tol;
  long long maxiter;
  int x_nonzero;
  int T, tiles, units, most;    // columns of a tile, tiles of a plane, units, most units of a block
  int stages, w_on_chip;
};

__host__ __device__ inline int march_even(int n) { return (n + 1) & ~1; }
// doubles of a stage: x, s0, s2 (tile and two nodes), s1 (tile and the lower
// halo), z and p (tile and both halos).  Copies start on an even node of the
// field, so a plane that starts on an odd one sits one entry to the right.
constexpr int kMarchX = 0, kMarchS0 = kMarchT + 2, kMarchS2 = 2 * (kMarchT + 2), kMarchZ = 3 * (kMarchT + 2) + 2;
struct MarchStage {
  int p, s1, size;   // z is at kMarchZ
  __host__ __device__ MarchStage(int T, int h) {
    const int full = march_even(T + 2 * h + 2);
    p = kMarchZ + full;
    s1 = p + full;
    size = s1 + march_even(T + h + 2);
  }
};

// a tile: columns [j0, j1) of the plane, fields with halo from lz to hz, s2 from l2
// (lz, j0, l2 even)
struct MarchTile {
  int j0, j1, lz, hz, l2;
  __device__ __forceinline__ MarchTile(int tile, int T, int h, int plane)
      : j0(tile * T), j1(min(j0 + T, plane)), lz(max(j0 - h, 0) & ~1), hz(min(j1 + h, plane)), l2(max(j0 - 2, 0)) {}
};

// elements [from, from + n) of src to dst (both even; the fields have a node of
// slack behind them); `bar` sees the bytes arrive
__device__ __forceinline__ void march_copy(unsigned int dst, const double* src, int from, int n, unsigned int bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src + from), "r"(8 * n), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool march_arrived(unsigned int bar, unsigned int phase) {
  unsigned int ok;
  asm volatile("{\n .reg .pred w;\n mbarrier.try_wait.parity.shared::cta.b64 w, [%1], %2;\n selp.u32 %0, 1, 0, w;\n}"
               : "=r"(ok)
               : "r"(bar), "r"(phase)
               : "memory");
  return ok != 0;
}
// what this thread wrote or saw written to global memory is visible to its bulk copies too
__device__ __forceinline__ void march_proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }

template <bool HAS2>
__global__ void __launch_bounds__(kMarchT, 1) march_pcg_kernel(const __grid_constant__ MarchArgs a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double own[3][kMarchWarps], vals[3][kMarchGrid], tot[3];
  __shared__ __align__(8) unsigned long long full[kMarchStages];
  const Grid3& g = a.g;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, G = gridDim.x, bid = blockIdx.x;
  const int n0 = g.n0, plane = g.st0, h = g.n2, T = a.T, S = a.stages;
  const int u0 = (int)((long long)a.units * bid / G), u1 = (int)((long long)a.units * (bid + 1) / G);
  const MarchStage L(T, h);
  const int np = T + 2 * h;
  double* const pn = sm + (size_t)S * L.size;       // [2][np]
  double* const won = pn + 2 * (size_t)march_even(np);   // [units of the block][T], or unused
  const unsigned int bars = (unsigned int)__cvta_generic_to_shared(full), ring = (unsigned int)__cvta_generic_to_shared(sm);
  unsigned int ep = 0, phases = 0;   // phases: the parity each stage's barrier shows next
  bool ok = true;                    // no wait has run out
  if (t == 0) {
    for (int k = 0; k < S; ++k) 
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8 * k), "n"(kMarchCopies) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  // totals over the grid of NV values per thread, in tot; `publish`: what this
  // block wrote to global memory before is visible to all blocks afterwards
  auto total = [&](auto& v, bool publish) -> bool {
    constexpr int NV = sizeof(v) / sizeof(double);
    ++ep;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const double s = tpf::warp_sum(v[k]);
      if (lane == 0) own[k][wid] = s;
    }
    FlagSlot* const set = a.slots + (size_t)(ep & 1) * G * kBandLine;
    if (publish) march_proxy_fence();
    __syncthreads();
    if (t < NV) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < kMarchWarps; ++k) s += own[t][k];
      if (publish) __threadfence();
      slot_store(set + (size_t)bid * kBandLine + t, s, ep);
    }
    if (t < NV * G) {
      const int k = t % NV, c = t / NV;
      FlagSlot q{0, 0};
      for (long long spins = 0;;) {
        slot_load(set + (size_t)c * kBandLine + k, true, q);
        if (slot_ready(q, ep) || !ok) break;
        if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; break; }
        if ((spins & 1023) == 0 && *(volatile int*)a.err) { ok = false; break; }
      }
      vals[k][c] = slot_value(q);
      if (publish) __threadfence();
    }
    ok = __syncthreads_and(ok) != 0;
    if (publish) march_proxy_fence();
    if (wid < NV) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < kMarchGrid / 32; ++k)
        if (lane + 32 * k < G) s += vals[wid][lane + 32 * k];
      s = tpf::warp_sum(s);
      if (lane == 0) tot[wid] = s;
    }
    __syncthreads();
    return ok;
  };

  // pass A: p = zs + beta pold (to pnew), x += alpha pold, w = S p; returns the thread's (p, w).
  // Steps: per segment of a tile, plane lo - 1 .. hi.
  int slot = 0;   // stage of the step
  auto march = [&](const double* zs, const double* pold, double beta, double alpha, double* pnew) -> double {
    // Copies: warp k of the last six issues copy k of a step, S - 1 steps ahead: z, p, x of the
    // plane, then s0, s1, s2 of the plane before (the couplings the step's row uses)
    const int role = wid - (kMarchWarps - kMarchCopies), back = role >= 3 ? 1 : 0;
    const double* const src = role == 0 ? zs : role == 1 ? pold : role == 2 ? a.x : role == 3 ? a.s0
                                                                     : role == 4 ? a.s1 : a.s2;
    const int place = role == 0 ? kMarchZ : role == 1 ? L.p : role == 2 ? kMarchX : role == 3 ? kMarchS0
                                                                 : role == 4 ? L.s1 : kMarchS2;
    int iu = u0, ilo = 0, ihi = 0, iq = 0, fill = slot, from = 0, upto = 0, j0 = 0, j1 = 0;
    auto enter = [&] {
      const int tile = iu / n0;
      ilo = iu - tile * n0;
      ihi = min(n0, ilo + (u1 - iu));
      iq = ilo - 1;
      const MarchTile it(tile, T, h, plane);
      j0 = it.j0;
      j1 = it.j1;
      from = role == 0 || role == 1 || role == 4 ? it.lz : role == 5 ? it.l2 : it.j0;
      upto = role < 2 ? it.hz : it.j1;
    };
    auto issue = [&] {
      if (role < 0 || iu >= u1) return;
      if (lane == 0) {
        const unsigned int bar = bars + 8u * fill;
        const int q = iq - back, base = q * plane, odd = base & 1;
        const bool full = iq >= ilo && iq < ihi;   // the step's plane is the block's
        // z and p of a plane that is not are for the columns above and below only
        const int f = role < 2 && !full ? j0 : from, e = role < 2 && !full ? j1 : upto;
        const bool on = q >= 0 && q < n0 && (role < 2 || (role == 2 ? full : role == 3 ? iq >= ilo : iq > ilo));
        const int n = on && (HAS2 || role < 5) ? march_even(e - f + odd) : 0;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(8 * n) : "memory");
        if (n) march_copy(ring + 8u * (unsigned int)(fill * L.size + place + (f - from)), src, base - odd + f, n, bar);
      }
      __syncwarp();
      if (++iq > ihi) {
        iu += ihi - ilo;
        if (iu < u1) enter();
      }
      fill = fill + 1 == S ? 0 : fill + 1;
    };
    if (iu < u1) enter();
    for (int k = 0; k + 1 < S; ++k) issue();
    double pw = 0.0;
    double *cur = pn, *old = pn + march_even(np);
    for (int u = u0; u < u1;) {
      const int tile = u / n0, lo = u - tile * n0, hi = min(n0, lo + (u1 - u));
      const MarchTile T0(tile, T, h, plane);
      const int own_n = T0.j1 - T0.j0, j = T0.j0 + t;
      const bool mine = t < own_n, lo1 = j >= h, lo2 = j > 0;
      const int pin_q = j == g.pin % plane ? g.pin / plane : -1;
      // places in a stage: z, s1, s2 of the column; the first halo column this thread refreshes
      const int jz = kMarchZ + (j - T0.lz), dp = L.p - kMarchZ, j1 = L.s1 + (j - T0.lz), j2 = kMarchS2 + (j - T0.l2);
      auto halo = [&](int e, int& c, int& k) {
        c = e < h ? e : own_n + e;
        const int jj = T0.j0 - h + c;
        k = jj >= 0 && jj < plane ? kMarchZ + (jj - T0.lz) : -1;
      };
      int hc, hk;
      halo(t, hc, hk);
      double pm = 0.0, pc = 0.0, pp = 0.0, s0m = 0.0;
      double* xq = a.x + ((lo - 1) * plane + j);
      double* dq = pnew + ((lo - 1) * plane + j);
      double* wq = a.w_on_chip ? won + (size_t)(u - u0) * T + t : a.w + (lo * plane + j);
      const int wstep = a.w_on_chip ? T : plane;
      int odd = ((lo - 1) * plane) & 1;
      // plane q: FIRST: lo - 1, LAST: hi (their p only, for the neighbour planes), else owned;
      // then the row of plane q - 1, if that is owned
      auto step = [&](int q, auto kind) {
        constexpr int K = decltype(kind)::value;   // 0: lo - 1, 1: lo, 2: between, 3: hi
        __syncthreads();
        issue();
        for (long long spins = 0; ok && !march_arrived(bars + 8 * slot, phases >> slot & 1u);)
          if (++spins > kSpinLimit) { atomicExch(a.err, 1); ok = false; }
        const double* const st = sm + slot * L.size;
        const int podd = (odd ^ plane) & 1;   // of plane q - 1
        pm = pc;
        pc = pp;
        pp = 0.0;
        if (mine && (K == 1 || K == 2 || (K == 0 && q >= 0) || (K == 3 && q < n0))) {
          const double po = st[jz + dp + odd];
          pp = fma(beta, po, st[jz + odd]);
          if (K == 1 || K == 2) {
            cur[h + t] = pp;
            *xq = fma(alpha, po, st[kMarchX + odd + t]);
            *dq = pp;
          }
        }
        if ((K == 1 || K == 2) && t < 2 * h) {
          cur[hc] = hk >= 0 ? fma(beta, st[hk + dp + odd], st[hk + odd]) : 0.0;
          for (int e = t + kMarchT; e < 2 * h; e += kMarchT) {
            int c, k;
            halo(e, c, k);
            cur[c] = k >= 0 ? fma(beta, st[k + dp + odd], st[k + odd]) : 0.0;
          }
        }
        if (mine && (K >= 2 || (K == 1 && q > 0))) {
          const double s0p = st[kMarchS0 + podd + t];
          if (K >= 2) {
            const double s1m = lo1 ? st[j1 - h + podd] : 0.0, s1p = st[j1 + podd];
            double d = (s0m + s0p) + (s1m + s1p);
            // beyond the walls of axis 1 p reads as 0; across those of axis 2 the coupling is a stored 0
            double acc = s0m * pm + s0p * pp + s1m * old[t] + s1p * old[t + 2 * h];
            if (HAS2) {
              const double s2m = lo2 ? st[j2 - 1 + podd] : 0.0, s2p = st[j2 + podd];
              d += s2m + s2p;
              acc += s2m * old[h + t - 1] + s2p * old[h + t + 1];
            }
            const double w = q - 1 == pin_q ? pc : d * pc - acc;
            *wq = w;
            wq += wstep;
            pw = fma(pc, w, pw);
          }
          s0m = s0p;
        }
        phases ^= 1u << slot;
        slot = slot + 1 == S ? 0 : slot + 1;
        double* const other = cur;
        cur = old;
        old = other;
        odd = podd;
        xq += plane;
        dq += plane;
      };
      step(lo - 1, std::integral_constant<int, 0>{});
      step(lo, std::integral_constant<int, 1>{});
      for (int q = lo + 1; q < hi; ++q) step(q, std::integral_constant<int, 2>{});
      step(hi, std::integral_constant<int, 3>{});
      u += hi - lo;
    }
    return pw;
  };

  // the block's nodes in batches: f(local unit, node, valid)
  auto nodes = [&](auto&& f) {
    int u = u0, tile = u0 / n0, i = u0 - tile * n0;
    while (u < u1) {
      int idx[kMarchBatch], loc[kMarchBatch];
      unsigned on = 0;
#pragma unroll
      for (int k = 0; k < kMarchBatch; ++k) {
        const int j = tile * T + t;
        if (u < u1 && t < T && j < plane) on |= 1u << k;
        idx[k] = i * plane + j;
        loc[k] = (u - u0) * T + t;
        if (++i == n0) { i = 0; ++tile; }
        ++u;
      }
      f(idx, loc, on);
    }
  };

  bool live = true;
  double rz = 0.0, rr = 0.0, bb = 0.0;
  if (a.x_nonzero) march(a.x, a.x, 0.0, 0.0, a.p[1]);   // w = S x
  {
    double red[3] = {0.0, 0.0, 0.0};
    nodes([&](const int (&idx)[kMarchBatch], const int (&loc)[kMarchBatch], unsigned on) {
#pragma unroll
      for (int k = 0; k < kMarchBatch; ++k)
        if (on & (1u << k)) {
          const int i = idx[k];
          const double bi = a.b[i];
          const double ri = a.x_nonzero ? bi - (a.w_on_chip ? won[loc[k]] : a.w[i]) : bi;
          const double zi = i == g.pin ? 0.0 : a.dinv[i] * ri;
          a.r[i] = ri;
          a.z[i] = zi;
          red[0] = fma(ri, zi, red[0]);
          red[1] = fma(ri, ri, red[1]);
          red[2] = fma(bi, bi, red[2]);
        }
    });
    live = total(red, true);
    rz = tot[0];
    rr = tot[1];
    bb = tot[2];
  }
  const double atol = a.tol * sqrt(bb), atol2 = atol * atol;
  long long it = 0;
  bool conv = bb == 0.0 || rr < atol2;
  double alpha = 0.0, beta = 0.0;
  int cur = 0;   // p[cur]: the newest direction
  while (live && !conv && it < a.maxiter) {
    double red[1] = {march(a.z, it ? a.p[cur] : a.z, beta, alpha, a.p[cur ^ 1])};
    cur ^= 1;
    if (!(live = total(red, false))) break;
    alpha = rz / tot[0];
    double red2[2] = {0.0, 0.0};
    nodes([&](const int (&idx)[kMarchBatch], const int (&loc)[kMarchBatch], unsigned on) {
      double ri[kMarchBatch], wi[kMarchBatch], di[kMarchBatch];
#pragma unroll
      for (int k = 0; k < kMarchBatch; ++k)
        if (on & (1u << k)) {
          ri[k] = a.r[idx[k]];
          di[k] = a.dinv[idx[k]];
          wi[k] = a.w_on_chip ? won[loc[k]] : a.w[idx[k]];
        }
#pragma unroll
      for (int k = 0; k < kMarchBatch; ++k)
        if (on & (1u << k)) {
          const double rn = ri[k] - alpha * wi[k], zn = idx[k] == g.pin ? 0.0 : di[k] * rn;
          a.r[idx[k]] = rn;
          a.z[idx[k]] = zn;
          red2[0] = fma(rn, zn, red2[0]);
          red2[1] = fma(rn, rn, red2[1]);
        }
    });
    if (!(live = total(red2, true))) break;
    beta = tot[0] / rz;
    rz = tot[0];
    rr = tot[1];
    ++it;
    conv = rr < atol2;
  }
  if (!live) {   // a wait ran out: leave once the copies are in, or after as long again
    for (int k = 0; k < S; ++k)
      for (long long spins = 0; spins < kSpinLimit && !march_arrived(bars + 8 * k, (phases >> k & 1u) ^ 1u); ++spins) {}
    return;
  }
  if (it > 0 || bb == 0.0) {   // the step x still owes
    nodes([&](const int (&idx)[kMarchBatch], const int (&)[kMarchBatch], unsigned on) {
#pragma unroll
      for (int k = 0; k < kMarchBatch; ++k)
        if (on & (1u << k)) a.x[idx[k]] = bb == 0.0 ? 0.0 : fma(alpha, a.p[cur][idx[k]], a.x[idx[k]]);
    });
  }
  if (bid == 0 && t == 0) {
    a.st->iters = it;
    a.st->applies = bb == 0.0 ? 0 : it + 1 + (a.x_nonzero ? 1 : 0);   // as the other PCG kernels count
    a.st->refinements = 0;
    a.st->rr = rr;
    a.st->bb = bb;
    a.st->converged = conv ? 1 : 0;
  }
}

}  // namespace
