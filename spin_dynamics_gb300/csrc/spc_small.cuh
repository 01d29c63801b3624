// Small systems: one CTA carries one sample's whole propagation -- every
// Krylov build, expm, projector Gram, dt loop and psi update until t_end --
// in a single launch (trace_sampling_para's per-sample loop,
// src/qm_dynamics.f90:322-378, with the CTA's threads over rows).
//
// Why: a system of a few hundred rows gives the tiled path (32 samples per
// tile, one launch per phase) kernels of microseconds, so a build round of
// ~90 launches is bound by launch and synchronisation latency, not by the
// FP64 pipe. Here a sample's build is ~1e6 DFMA on its own SM with
// block-level barriers only. Used (SPC_SAMPLE_AUTO) when every job has at
// most SMALL_NMAX rows, m <= 32, a small estimated build and the samples fill
// at most two waves of CTAs (small_path_fits).
//
// Calls with few samples give each sample a cluster of two CTAs instead
// (k_small_pair, below).
//
// Per sample the arithmetic is the tiled path's: the entries of k_spmm's rows,
// real-coefficient Lanczos on the Hermitian part (orthonormality checked from
// the projector Grams, MGS rebuild when it fails) or MGS, expm_one, the four
// Hermitian projector Grams, the reference's dt-loop semantics. Reductions are
// integer or two-level in a fixed order, so results repeat bit for bit; they
// differ from the tiled path's by rounding.
// Control flow is uniform across the CTA: every barrier is reached by all
// threads, and a sample leaves the loop only when the whole CTA does.
#define SMALL_THREADS 256
#define SMALL_WARPS (SMALL_THREADS / 32)
#define SMALL_MAX_M 32
#define SMALL_NMAX 2048
#define SMALL_GRAM_R(mt) ((mt) == 1 ? 32 : 16)  // rows per chunk of the Grams: two CTAs' scratch in an SM at m = 20
#define SMALL_STATIC 12288  // at least the kernels' static shared memory

struct SmallJob {
  int n, Z, me;            // rows, nuclear rows, Krylov dimension min(m, n)
  const int* rowptr;       // execution-order CSR (k_split_rows)
  const int* split;
  const int* col;
  const double2* val;
  const double* kappa;     // non-null: the copy holds A of A - i*kappa*1
  int rexp;                // ||H|| <= 2^rexp
  const double2* zk;       // M x Z sample vectors of the job
};

// Sum over the CTA of values whose absolute sum is at most 2^e, or with NORM its
// square root and that root's reciprocal (0 for a zero sum): every thread gets
// {sum or root, reciprocal}. A double add's latency is 109 clocks with its
// shuffle, eight of them in a row and 1010 more for a square root and a division;
// as integer multiples of 2^(e - 110) (acc_add's pair of words) a level takes a
// third of that. A square that is not zero counts as one unit at least, so that
// only a zero vector has a zero norm (small_norm). red: SMALL_WARPS pairs and the result, two sets that the
// calls use in turn (`turn`). Called by all threads; one result per two barriers.
//
// A sample's rows may be spread over a cluster of up to SMALL_TEAM CTAs (CL):
// every CTA then sends its partials to all of them and adds the same numbers in
// the same order.
#define SMALL_TEAM 4
struct SmallRed {
  longlong2 part[2][SMALL_TEAM * SMALL_WARPS];
  double2 out[2];
};
struct SmallTeam {
  int rank, size;
};
template <bool NORM, bool CL = false>
__device__ __forceinline__ double2 block_sum(double v, int e, SmallRed& red, int& turn, SmallTeam team = {0, 1}) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long b = __double_as_longlong(v);
  const int ex = (int)(b >> 52) & 0x7ff;
  const bool bad = ex != 0 && ex - 1023 > e + 1;  // NaN, infinities, a broken bound
  long long hi = 0, lo = 0;
  if (ex != 0 && !bad) {
    const acc_t man = (b & 0xfffffffffffffll) | (1ull << 52);
    const int sh = ex - 965 - e;
    if (sh >= 0) {
      lo = (long long)((man << sh) & ((1ull << 50) - 1));
      hi = (long long)(sh >= 50 ? man << (sh - 50) : man >> (50 - sh));
    } else {
      acc_t u = sh < -62 ? 0 : ((man >> (-sh - 1)) + 1) >> 1;
      if (NORM && u == 0) u = 1;
      lo = (long long)(u & ((1ull << 50) - 1));
      hi = (long long)(u >> 50);
    }
    if (b < 0) {
      lo = -lo;
      hi = -hi;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    hi += __shfl_xor_sync(0xffffffffu, hi, o);
    lo += __shfl_xor_sync(0xffffffffu, lo, o);
  }
  if (__any_sync(0xffffffffu, bad)) hi = LLONG_MIN;
  if (CL) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (lane < team.size)
      cluster.map_shared_rank(&red, lane)->part[turn][team.rank * SMALL_WARPS + warp] = make_longlong2(hi, lo);
    cluster.sync();
  } else {
    if (lane == 0) red.part[turn][warp] = make_longlong2(hi, lo);
    __syncthreads();
  }
  if (warp == 0) {
    const int np = CL ? team.size * SMALL_WARPS : SMALL_WARPS;
    const longlong2 x = red.part[turn][lane & (np - 1)];
    hi = x.x;
    lo = x.y;
    const bool nan = __any_sync(0xffffffffu, hi == LLONG_MIN);
#pragma unroll
    for (int o = CL ? 16 : SMALL_WARPS / 2; o > 0; o >>= 1) {
      if (CL && o >= np) continue;
      hi += __shfl_xor_sync(0xffffffffu, hi, o);
      lo += __shfl_xor_sync(0xffffffffu, lo, o);
    }
    double s = ldexp(fma((double)hi, 1125899906842624.0, (double)lo), e - 110);
    if (nan) s = __longlong_as_double(0x7ff8000000000000ll);
    double r = 0.0;
    if (NORM) {
      // root and reciprocal from one inverse root, the root corrected to its
      // last bit
      r = s > 0.0 ? rsqrt(s) : (s == 0.0 ? 0.0 : s);
      const double q = s * r;
      s = fma(fma(-q, q, s), 0.5 * r, q);
    }
    if (lane == 0) red.out[turn] = make_double2(s, r);
  }
  __syncthreads();
  const double2 res = red.out[turn];
  turn ^= 1;
  return res;
}

// {root, reciprocal} of a sum of squares bounded by 2^e: taken again in finer
// units where the first ones left fewer bits than a double's (a vector far
// below the bound on ||H||).
template <bool CL>
__device__ __forceinline__ double2 small_norm(double v, int e, SmallRed& red, int& turn, SmallTeam team) {
  for (;;) {
    const double2 r = block_sum<true, CL>(v, e, red, turn, team);
    const int top = 2 * (((__double2hiint(r.x) >> 20) & 0x7ff) - 1023) + 3;  // the sum is below 2^top
    if (!(r.x > 0.0) || top >= e - 44 || e < -1000) return r;
    e = top;
  }
}

// Real sum over the CTA in doubles, its root and reciprocal: for a value of any
// size (a state's norm). Called by all threads.
__device__ __forceinline__ double2 block_norm(double v, SmallRed& red, int& turn) {
  double* part = reinterpret_cast<double*>(red.part[turn]);
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double x = threadIdx.x < SMALL_WARPS ? part[threadIdx.x] : 0.0;
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    if (threadIdx.x == 0) {
      const double b = sqrt(x);
      red.out[turn] = make_double2(b, b > 0.0 ? 1.0 / b : 0.0);
    }
  }
  __syncthreads();
  const double2 res = red.out[turn];
  turn ^= 1;
  return res;
}

// Vectors are taken by components: thread idx has component idx & 1 (real,
// imaginary) of row idx / 2, the order in memory. A warp instruction of FP64
// holds its scheduler's pipe for 64 clocks whatever the lanes in use, and the
// 288 rows of a small pair are nine warps on four schedulers (three on one);
// as 576 components they are five half-rows at most against six, and where rows
// are few a row's chain of multiply-adds is half as long: 64 samples at dim 288,
// m = 20, 5000 steps 24.3 -> 22.1 ms; dim 48, m = 10 1.98 -> 1.88 ms.
__device__ __forceinline__ double flip(double v, bool neg) {
  return __hiloint2double(__double2hiint(v) ^ (neg ? (int)0x80000000 : 0), __double2loint(v));
}
// component im of a + v q for the complex v, q
__device__ __forceinline__ double half_fma(double2 v, double2 q, bool im, double a) {
  a = fma(v.x, im ? q.y : q.x, a);
  return fma(flip(v.y, !im), im ? q.x : q.y, a);
}

// Component idx of H x. Entries are taken four at a time, all loads before the
// sums: a row has 4 to 20 entries, and their latency, not their arithmetic, is
// a row's time. shift adds -i*kappa*x_r.
__device__ __forceinline__ double small_half(const SmallJob& J, const double2* __restrict__ x, int idx, bool shift,
                                             double kap) {
  const int r = idx >> 1;
  const bool im = (idx & 1) != 0;
  const int k0 = __ldg(J.rowptr + r), ks = __ldg(J.split + r), k1 = __ldg(J.rowptr + r + 1);
  const double* xd = reinterpret_cast<const double*>(x) + (idx & 1);
  double a0 = 0.0, a1 = 0.0;
  for (int k = k0; k < ks; k += 4) {
    double2 v[4], q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = k + u < ks;
      v[u] = in ? __ldg(J.val + k + u) : cz();
      q[u] = x[in ? __ldg(J.col + k + u) : r];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < ks) {
        if (u & 1)
          a1 = half_fma(v[u], q[u], im, a1);
        else
          a0 = half_fma(v[u], q[u], im, a0);
      }
  }
  for (int k = ks; k < k1; k += 4) {
    double v[4], q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = k + u < k1;
      v[u] = in ? __ldg(&J.val[k + u].x) : 0.0;
      q[u] = xd[2 * (in ? __ldg(J.col + k + u) : r)];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < k1) {
        if (u & 1)
          a1 = fma(v[u], q[u], a1);
        else
          a0 = fma(v[u], q[u], a0);
      }
  }
  double y = a0 + a1;
  if (shift) {
    const double2 xr = x[r];
    y = fma(flip(kap, im), im ? xr.x : xr.y, y);
  }
  return y;
}

// Row r of H x, both components by one thread: from SMALL_WIDE rows on, where every
// scheduler has rows enough and a row's entries loaded twice cost more than the
// halves even out. 120 samples, m = 8, 40 steps of 1 ns, components -> rows: dim
// 576 even; dim 1152 general 3.67 -> 3.31, isotropic MGS 3.37 -> 2.82 ms; dim 1728
// isotropic MGS 4.79 -> 3.83 ms (with a block's dots over all warps, below).
#define SMALL_WIDE 512
__device__ __forceinline__ double2 small_row(const SmallJob& J, const double2* __restrict__ x, int r, bool shift,
                                             double kap) {
  const int k0 = __ldg(J.rowptr + r), ks = __ldg(J.split + r), k1 = __ldg(J.rowptr + r + 1);
  double2 a0 = cz(), a1 = cz();
  for (int k = k0; k < ks; k += 4) {
    double2 v[4], q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = k + u < ks;
      v[u] = in ? __ldg(J.val + k + u) : cz();
      q[u] = x[in ? __ldg(J.col + k + u) : r];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < ks) {
        if (u & 1)
          a1 = cfma(v[u], q[u], a1);
        else
          a0 = cfma(v[u], q[u], a0);
      }
  }
  for (int k = ks; k < k1; k += 4) {
    double v[4];
    double2 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = k + u < k1;
      v[u] = in ? __ldg(&J.val[k + u].x) : 0.0;
      q[u] = x[in ? __ldg(J.col + k + u) : r];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < k1) {
        double2& a = (u & 1) ? a1 : a0;
        a.x = fma(v[u], q[u].x, a.x);
        a.y = fma(v[u], q[u].y, a.y);
      }
  }
  double2 y = cadd(a0, a1);
  if (shift) {
    const double2 xr = x[r];
    y.x = fma(kap, xr.y, y.x);
    y.y = fma(-kap, xr.x, y.y);
  }
  return y;
}

// psi = Q c (:365) by components, over all threads of the CTA
__device__ __forceinline__ void small_psi(int me, int n, const double2* Q, const double2* c, double2* psi) {
  if (n >= SMALL_WIDE) {
    for (int r = threadIdx.x; r < n; r += SMALL_THREADS) {
      double2 a = cz();
      for (int j = 0; j < me; ++j) a = cfma(c[j], Q[(size_t)j * n + r], a);
      psi[r] = a;
    }
    return;
  }
  for (int idx = threadIdx.x; idx < 2 * n; idx += SMALL_THREADS) {
    double a = 0.0;
    for (int j = 0; j < me; ++j) a = half_fma(c[j], Q[(size_t)j * n + (idx >> 1)], (idx & 1) != 0, a);
    reinterpret_cast<double*>(psi)[idx] = a;
  }
}

// The four projector Grams P_t = V_t^H V_t over the Z nuclear rows (k_gram and
// k_proj_reduce of one sample; S and T0 halved): gram_sums per type, the
// CTA's eight warps over the blocks. `top`: high word of the basis' largest
// component; work: gram_smem_bytes. Ends with a barrier. FP64 Grams of 20
// vectors at dim 288 took 124 K clocks, these 90 K (and leave the FP64
// pipes alone).
template <int MT>
__device__ __forceinline__ void small_grams(int m, int me, int n, int Z, unsigned top, const double2* Q, double2* P,
                                            unsigned char* work) {
  constexpr int MP = 16 * MT;
  longlong2* acc64 = reinterpret_cast<longlong2*>(work);
  unsigned* V = reinterpret_cast<unsigned*>(acc64 + 8 * 256);
  const double* Tm = reinterpret_cast<const double*>(V);
  const double unit = gram_unit(top);
  for (int t = 0; t < 4; ++t) {
    gram_sums<MT, SMALL_GRAM_R(MT), false>(t, me, me, (int)(top >> 20), 0, Z, acc64, V, nullptr,
                  [&](int j, int64_t row, int e) { return &Q[(size_t)j * n + (size_t)(e * Z + (int)row)]; });
    double2* Pt = P + (size_t)t * m * m;
    for (int idx = threadIdx.x; idx < MP * MP; idx += SMALL_THREADS) {
      const int i = idx / MP, j = idx % MP;
      if (i > j || j >= me) continue;
      double2 s = gram_entry<MT>(Tm, i, j, unit);
      if (t == 1 || t == 2) s = make_double2(0.5 * s.x, 0.5 * s.y);
      if (i == j && s.y == s.y) s.y = 0.0;
      Pt[i + j * m] = s;
      if (i != j) Pt[j + i * m] = make_double2(s.x, -s.y);
    }
    __syncthreads();
  }
}
__device__ void small_projectors(int m, int me, int n, int Z, unsigned top, const double2* Q, double2* P, void* work) {
  if (me <= 16)
    small_grams<1>(m, me, n, Z, top, Q, P, (unsigned char*)work);
  else
    small_grams<2>(m, me, n, Z, top, Q, P, (unsigned char*)work);
}
__host__ __device__ __forceinline__ size_t small_gram_elems(int m) { return (gram_smem_bytes(m <= 16 ? 1 : 2, SMALL_GRAM_R(m <= 16 ? 1 : 2)) + 15) / 16; }

// Scratch of small_krylov: coefficients of a block of vectors and the products of
// basis vectors within their blocks (k_ortho's recurrence).
struct SmallOrtho {
  double2 h[ORTHO_NB];
  double2 gram[SMALL_MAX_M][ORTHO_NB];  // <Q_j, Q_k>, k < j of j's block
  double part[ORTHO_NB][4];             // a warp's dot and product, where several warps share a vector
  unsigned top;                         // high word of the basis' largest component
};

// One Krylov basis of psi (get_krylov, src/qm_dynamics.f90:432-467): A (m x m,
// zeroed first) gets the tridiagonal (lz: Lanczos on the Hermitian part, real
// coefficients, alpha - i*kappa on the diagonal) or the Hessenberg (MGS),
// Q_0..Q_{me-1} the basis, cA = ||psi|| e_1; p is the work vector. Called by
// all SMALL_THREADS threads of the CTA; thread 0 writes A's last entries (and
// the warps ort.top) after the last barrier, so the caller synchronises before
// reading them.
// MGS in blocks of eight vectors (see k_ortho): warp v sums <Q_v, p> over all
// rows by itself, so a block costs one warp's tree of adds and three barriers
// where a vector at a time cost a CTA sum each. 20 vectors at dim 288: 1.5 M
// clocks a vector at a time, 1.1 M by blocks; dim 48, 10 vectors: 230 K -> 147 K.
// CL: the CTA of a cluster that holds rows [r0, r0 + nl) of every vector (Q and p
// with ns rows); psi (all n rows, in every CTA) becomes the vector that H is
// applied to. Dots and norms are sums over the cluster, and a new vector's rows
// go to every CTA: nblocks + 2 cluster barriers a step.
struct SmallExch {
  double d[2][SMALL_TEAM][SMALL_WARPS][4];  // a block's dots and products of each CTA, two sets in turn
};
template <bool CL = false>
__device__ __forceinline__ void small_krylov(const SmallJob& J, bool lz, bool herm, double kap, int m, double2* A,
                                             double2* cA, double2* Q, double2* p,
                                             std::conditional_t<CL, double2*, const double2*> psi, SmallRed& red,
                                             SmallOrtho& ort, int& turn, SmallTeam team = {0, 1},
                                             SmallExch* ex = nullptr) {
  namespace cg = cooperative_groups;
  const int me = J.me, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = CL ? (J.n + team.size - 1) / team.size : J.n;  // rows of a vector here
  const int r0 = CL ? team.rank * n : 0, nl = CL ? max(0, min(n, J.n - r0)) : n;
  const bool wide = !CL && n >= SMALL_WIDE;  // rows instead of components
  int turn_ex = 0;
  const size_t mm = (size_t)m * m;
  for (int i = tid; i < (int)mm; i += SMALL_THREADS) A[i] = cz();
  double* pd = reinterpret_cast<double*>(p);
  double* Qd = reinterpret_cast<double*>(Q);
  auto* psid = reinterpret_cast<std::conditional_t<CL, double, const double>*>(psi);
  // c = ||psi|| e_1, Q_0 = psi / ||psi|| (get_krylov :440-447)
  double acc = 0.0;
  for (int idx = tid; idx < 2 * J.n; idx += SMALL_THREADS) acc = fma(psid[idx], psid[idx], acc);
  const double2 bn0 = block_norm(acc, red, turn);
  unsigned top = 0;
  if (tid == 0) ort.top = 0;
  for (int idx = tid; idx < 2 * J.n; idx += SMALL_THREADS) {
    const double q = psid[idx] * bn0.y;
    if constexpr (CL) {
      psid[idx] = q;
      if (idx >= 2 * r0 && idx < 2 * (r0 + nl)) Qd[idx - 2 * r0] = q;
    } else {
      Qd[idx] = q;
    }
    top = max(top, (unsigned)__double2hiint(q) & 0x7fffffffu);
  }
  if (tid < m) cA[tid] = tid == 0 ? make_double2(bn0.x, 0.0) : cz();
  if (CL)
    cg::this_cluster().sync();  // every CTA has psi before another one's rows arrive there
  else
    __syncthreads();
  double beta = 0.0;
  for (int i = 0; i < me; ++i) {
    const double2* qi = Q + (size_t)i * n;
    const double2* x = CL ? psi : qi;
    const double* qid = Qd + (size_t)i * 2 * n;
    double alpha = 0.0;
    int na = 0, ja = 0;  // the block whose projection is still to be subtracted
    if (lz) {
      // p = H q_i - beta_{i-1} Q_{i-1}; alpha_i = Re <Q_i, p>
      double a2 = 0.0;
      for (int r = tid; wide && r < n; r += SMALL_THREADS) {
        double2 pv = small_row(J, x, r, false, kap);
        const double2 q = qi[r];
        if (i > 0) {
          const double2 q0 = qi[r - n];
          pv.x = fma(-beta, q0.x, pv.x);
          pv.y = fma(-beta, q0.y, pv.y);
        }
        p[r] = pv;
        a2 = fma(q.y, pv.y, fma(q.x, pv.x, a2));
      }
      for (int idx = tid; !wide && idx < 2 * nl; idx += SMALL_THREADS) {
        double pv = small_half(J, x, idx + 2 * r0, false, kap);
        if (i > 0) pv = fma(-beta, qid[idx - 2 * n], pv);
        pd[idx] = pv;
        a2 = fma(qid[idx], pv, a2);
      }
      alpha = block_sum<false, CL>(a2, J.rexp, red, turn, team).x;
      if (tid == 0) A[i + i * m] = make_double2(alpha, -kap);
      if (i == me - 1) break;
    } else {
      for (int r = tid; wide && r < n; r += SMALL_THREADS) p[r] = small_row(J, x, r, herm, kap);
      for (int idx = tid; !wide && idx < 2 * nl; idx += SMALL_THREADS) pd[idx] = small_half(J, x, idx + 2 * r0, herm, kap);
      // MGS (get_krylov :453-456) by blocks: d_v = <Q_v, p>, h_v from the d_v and
      // the block's basis products, p -= sum_v h_v Q_v
      for (int jb = 0; jb <= i; jb += ORTHO_NB) {
        const int nb = min(ORTHO_NB, i + 1 - jb);
        const bool newest = jb + nb == i + 1;
        __syncthreads();  // p and the last block's coefficients
        // a block of few vectors leaves warps: long ones go to 2, 4 or 8 of them
        const int lw = !wide || nb > 4 ? 0 : (nb > 2 ? 1 : (nb > 1 ? 2 : 3));
        const int wv = warp >> lw;
        if (wv < nb) {
          const double2* qv = Q + (size_t)(jb + wv) * n;
          const bool prod = newest && wv < nb - 1;  // also <Q_v, Q_i>
          double2 d = cz(), gp = cz();
          for (int r = lane + 32 * (warp & ((1 << lw) - 1)); r < nl; r += 32 << lw) {
            const double2 q = qv[r];
            d = cjfma(q, p[r], d);
            if (prod) gp = cjfma(q, qi[r], gp);
          }
          // the four sums, two halves of the lanes at a time
          const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
          double ka = h16 ? gp.x : d.x, kb = h16 ? gp.y : d.y;
          ka += __shfl_xor_sync(0xffffffffu, h16 ? d.x : gp.x, 16);
          kb += __shfl_xor_sync(0xffffffffu, h16 ? d.y : gp.y, 16);
          double v = h8 ? kb : ka;
          v += __shfl_xor_sync(0xffffffffu, h8 ? ka : kb, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          if (CL) {
            if ((lane & 7) < team.size)
              cg::this_cluster().map_shared_rank(ex, lane & 7)->d[turn_ex][team.rank][warp][lane >> 3] = v;
          } else if (lw > 0) {
            if ((lane & 7) == 0) ort.part[warp][lane >> 3] = v;
          } else {
            if (lane == 0) ort.h[warp].x = v;
            if (lane == 8) ort.h[warp].y = v;
            // <Q_i, Q_v> = conj <Q_v, Q_i>
            if (prod && lane == 16) ort.gram[i][warp].x = v;
            if (prod && lane == 24) ort.gram[i][warp].y = -v;
          }
        }
        const int set = turn_ex;
        turn_ex ^= 1;
        if (CL)
          cg::this_cluster().sync();
        else
          __syncthreads();
        if (warp == 0) {
          if (CL || lw > 0) {
            // four lanes a vector: the components in the order of ranks or warps
            const int v = lane >> 2, u = lane & 3;
            if (v < nb) {
              double y;
              if (CL) {
                y = ex->d[set][0][v][u];
                for (int c = 1; c < team.size; ++c) y += ex->d[set][c][v][u];
              } else {
                y = ort.part[v << lw][u];
                for (int c = 1; c < 1 << lw; ++c) y += ort.part[(v << lw) + c][u];
              }
              double* to = reinterpret_cast<double*>(u < 2 ? &ort.h[v] : &ort.gram[i][v]);
              if (u < 2 || (newest && v < nb - 1)) to[u & 1] = u == 3 ? -y : y;
            }
            __syncwarp();
          }
          // first-order corrections where the basis is orthonormal to rounding
          // and the units suit single precision, the recurrence otherwise
          const int v = lane;
          double2 d = v < nb ? ort.h[v] : cz();
          float2 c = make_float2(0.f, 0.f);
          bool big = !single_range(J.rexp);
          if (v < nb)
            for (int k = 0; k < v; ++k) {
              const double2 gv = ort.gram[jb + v][k];
              const float gx = cut_float(gv.x), gy = cut_float(gv.y), hx = cut_float(ort.h[k].x), hy = cut_float(ort.h[k].y);
              big |= !(fabsf(gx) + fabsf(gy) < 4e-9f);
              c.x += gx * hx - gy * hy;
              c.y += gx * hy + gy * hx;
            }
          if (!__any_sync(0xffffffffu, big)) {
            d = make_double2(d.x - wide_any(c.x), d.y - wide_any(c.y));
          } else {
            for (int k = 0; k + 1 < nb; ++k) {
              const double2 hk = make_double2(__shfl_sync(0xffffffffu, d.x, k), __shfl_sync(0xffffffffu, d.y, k));
              if (v > k && v < nb) d = cfms(ort.gram[jb + v][k], hk, d);
            }
          }
          __syncwarp();
          if (v < nb) {
            ort.h[v] = d;
            A[jb + v + i * m] = d;
          }
        }
        __syncthreads();
        if (!newest || i < me - 1) {
          if (newest) {
            ja = jb;
            na = nb;
          } else {
            for (int r = tid; wide && r < n; r += SMALL_THREADS) {
              double2 pv = p[r];
#pragma unroll
              for (int v = 0; v < ORTHO_NB; ++v) pv = cfms(ort.h[v], Q[(size_t)(jb + v) * n + r], pv);
              p[r] = pv;
            }
            for (int idx = tid; !wide && idx < 2 * nl; idx += SMALL_THREADS) {
              const bool im = (idx & 1) != 0;
              double pv = pd[idx];
#pragma unroll
              for (int v = 0; v < ORTHO_NB; ++v) {
                const double2 h = ort.h[v];
                pv = half_fma(make_double2(-h.x, -h.y), Q[(size_t)(jb + v) * n + (idx >> 1)], im, pv);
              }
              pd[idx] = pv;
            }
          }
        }
      }
      if (i == me - 1) break;
    }
    // the last projection, ||p|| and Q_{i+1} = p / ||p||
    double nr = 0.0;
    for (int r = tid; wide && r < n; r += SMALL_THREADS) {
      double2 pv = p[r];
      if (lz) {
        const double2 q = qi[r];
        pv.x = fma(-alpha, q.x, pv.x);
        pv.y = fma(-alpha, q.y, pv.y);
      } else {
        for (int v = 0; v < na; ++v) pv = cfms(ort.h[v], Q[(size_t)(ja + v) * n + r], pv);
      }
      p[r] = pv;
      nr = fma(pv.y, pv.y, fma(pv.x, pv.x, nr));
    }
    for (int idx = tid; !wide && idx < 2 * nl; idx += SMALL_THREADS) {
      double pv = pd[idx];
      if (lz) {
        pv = fma(-alpha, qid[idx], pv);
      } else {
        for (int v = 0; v < na; ++v) {
          const double2 h = ort.h[v];
          pv = half_fma(make_double2(-h.x, -h.y), Q[(size_t)(ja + v) * n + (idx >> 1)], (idx & 1) != 0, pv);
        }
      }
      pd[idx] = pv;
      nr = fma(pv, pv, nr);
    }
    const double2 bn = small_norm<CL>(nr, 2 * J.rexp, red, turn, team);
    beta = bn.x;
    if (tid == 0) {
      A[(i + 1) + i * m] = make_double2(beta, 0.0);
      if (lz) A[i + (i + 1) * m] = make_double2(beta, 0.0);
    }
    double* qn = Qd + (size_t)(i + 1) * 2 * n;
    for (int idx = tid; idx < 2 * nl; idx += SMALL_THREADS) {
      const double q = pd[idx] * bn.y;
      qn[idx] = q;
      if constexpr (CL)
        for (int c = 0; c < team.size; ++c) cg::this_cluster().map_shared_rank(psid, c)[2 * r0 + idx] = q;
      top = max(top, (unsigned)__double2hiint(q) & 0x7fffffffu);
    }
    if (CL)
      cg::this_cluster().sync();
    else
      __syncthreads();
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&ort.top, top);
}

// The Krylov bases of a small system's samples for the yield gradient, one CTA
// per slot with its vectors in shared memory, written in the tiles' layout. The
// tiled build of a step is about 4 m launches of kernels that a few hundred rows
// fill for microseconds: 32 samples at dim 288, m = 16, MGS take 0.72 ms so and
// 0.38 ms here (FP64 issue: 16 complex entries a row and 136 vector pairs).
// Dynamic shared memory: A (m^2), c (m), basis (m n), work and state vector (n each).
// With samples for at most half or a quarter of the SMs a cluster of two or four
// CTAs takes each (`size` CTAs, rows split): 0.38 -> 0.20 ms.
__host__ __device__ __forceinline__ size_t small_basis_elems(int m, int n, int team) {
  return (size_t)m * m + m + (size_t)(m + 1) * ((n + team - 1) / team) + n;
}
template <bool CL>
__global__ void __launch_bounds__(SMALL_THREADS)
    k_small_basis(const TileInfo* __restrict__ tiles, const int* __restrict__ map, const int* __restrict__ scol,
                  const double2* __restrict__ x, int m, int lanczos, int size, double2* __restrict__ Q,
                  double2* __restrict__ Ahess, double2* __restrict__ cvec) {
  extern __shared__ double2 smem[];
  __shared__ SmallRed red;
  __shared__ SmallOrtho ort;
  __shared__ SmallExch ex;
  const int w = CL ? blockIdx.x / size : blockIdx.x;
  if (map[w] < 0) return;  // every CTA of a cluster
  const TileInfo& T = tiles[w / SPC_LANES];
  const SmallJob J{T.n, T.n / 4, T.m, T.rowptr, T.split, T.col, T.val, T.kappa, T.rexp, nullptr};
  const SmallTeam team{CL ? (int)(blockIdx.x % size) : 0, CL ? size : 1};
  const int n = T.n, tid = threadIdx.x, ns = (n + team.size - 1) / team.size, r0 = team.rank * ns;
  double2* A = smem;
  double2* cA = A + m * m;
  double2* V = cA + m;
  double2* p = V + (size_t)m * ns;
  double2* psi = p + ns;
  const double2* src = x + T.psi_off + scol[w];
  for (int r = tid; r < n; r += SMALL_THREADS) psi[r] = src[(size_t)r * T.ldp];
  __syncthreads();
  int turn = 0;
  const bool herm = T.kappa != nullptr;
  small_krylov<CL>(J, lanczos != 0, herm, herm ? *T.kappa : 0.0, m, A, cA, V, p, psi, red, ort, turn, team, &ex);
  __syncthreads();
  if (team.rank == 0) {
    for (int k = tid; k < m * m; k += SMALL_THREADS) Ahess[(size_t)w * m * m + k] = A[k];
    if (tid < m) cvec[(size_t)w * m + tid] = cA[tid];
  }
  double2* dst = Q + T.q_off + (w % SPC_LANES);
  for (int k = tid; k < T.m * ns; k += SMALL_THREADS) {
    const int j = k / ns, r = r0 + k - j * ns;
    if (r < n) dst[((size_t)j * n + r) * SPC_LANES] = V[k];
  }
  if (CL) cooperative_groups::this_cluster().sync();  // no CTA leaves before the others' last access
}

// max |sum_t P_t - I| over the me x me block of the four Grams (NaN wins):
// the orthonormality of a Lanczos basis (the Grams sum to Q^H Q). Called by
// all threads; every thread gets the maximum.
__device__ __forceinline__ double small_ortho_err(int me, int m, const double2* P, double* terms, double* cstat) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t mm = (size_t)m * m;
  double mx = 0.0;
  for (int id = tid; id < me * me; id += SMALL_THREADS) {
    const int i = id % me, j = id / me;
    const size_t x = (size_t)i + (size_t)j * m;
    const double2 g = cadd(cadd(P[x], P[mm + x]), cadd(P[2 * mm + x], P[3 * mm + x]));
    const double e = fmax(fabs(g.x - (i == j ? 1.0 : 0.0)), fabs(g.y));
    mx = (e > mx || e != e) ? e : mx;
  }
  for (int d = 16; d > 0; d >>= 1) {
    const double v = __shfl_xor_sync(0xffffffffu, mx, d);
    mx = (v > mx || v != v) ? v : mx;
  }
  if (lane == 0) terms[warp] = mx;
  __syncthreads();
  if (warp == 0) {
    double v = lane < SMALL_WARPS ? terms[lane] : 0.0;
    for (int d = 16; d > 0; d >>= 1) {
      const double u = __shfl_xor_sync(0xffffffffu, v, d);
      v = (u > v || u != u) ? u : v;
    }
    if (lane == 0) cstat[0] = v;
  }
  __syncthreads();
  const double mall = cstat[0];
  __syncthreads();
  return mall;
}

// Grid: one CTA of SMALL_THREADS per sample (global sample s = blockIdx.x).
// work + soff[s]: the sample's basis (m x n), work vector (n) and state (n);
// with vec_smem they live in shared memory instead (every job's (m+2) n
// complex fits there), which cuts the latency of the row sweeps.
// Dynamic shared memory: A, E (m^2 each), P (4 m^2), c and c' (m each),
// max(5 m^2, small_gram_elems) of expm / projector scratch, all complex, then
// the vectors when vec_smem.
// CTAS: CTAs in an SM that the registers allow. Two (128 registers) need spills that
// a lone CTA does not: 120 samples, m = 8, 40 steps of 1 ns, dim 144 0.94 -> 0.86,
// dim 216 1.05 -> 0.91 ms; 304 samples at dim 432, m = 24 (one CTA fits) 2.57 -> 2.42.
template <int CTAS>
__global__ void __launch_bounds__(SMALL_THREADS, CTAS)
    k_small_prop(const SmallJob* __restrict__ jobs, const int* __restrict__ sjob, const int* __restrict__ scol,
                 const int64_t* __restrict__ soff, double2* __restrict__ work, Theta th, int m, int T, double dt,
                 double t_end, double tol, int lanczos, int vec_smem, double* __restrict__ obs,
                 long long* __restrict__ nsteps, unsigned long long* __restrict__ counts, int* __restrict__ err) {
  extern __shared__ double2 smem[];
  __shared__ double rowsum[SPC_MAX_M];
  __shared__ int band[4];
  __shared__ SmallRed red;
  __shared__ SmallOrtho ort;
  __shared__ double2 part[4][32];
  __shared__ double terms[16];
  __shared__ double cstat[2];
  __shared__ double loop_t;
  __shared__ int loop_k, loop_done;
  __shared__ long long loop_steps;

  const int s = blockIdx.x;
  const SmallJob J = jobs[sjob[s]];
  const int n = J.n, Z = J.Z, me = J.me;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t mm = (size_t)m * m;
  double2* A = smem;
  double2* E = A + mm;
  double2* P = E + mm;
  double2* cA = P + 4 * mm;
  double2* cB = cA + m;
  double2* X = cB + m;
  double2* Q = vec_smem ? X + max(5 * mm, small_gram_elems(m)) : work + soff[s];
  double2* p = Q + (size_t)m * n;
  double2* psi = p + n;
  const bool herm = J.kappa != nullptr;
  const double kap = herm ? *J.kappa : 0.0;
  const double2* zk = J.zk + (size_t)scol[s] * Z;
  double* o = obs + (size_t)s * 4 * T;

  // psi_0 = theta (x) z (kron_vector)
  for (int r = tid; r < n; r += SMALL_THREADS) psi[r] = cmul(th.v[r / Z], zk[r % Z]);
  __syncthreads();
  double t = 0.0;
  int k = 1;  // outputs 0 hold the initial populations (k_obs_init)
  long long steps = 0;
  int turn = 0;
  unsigned long long nb = 0, nf = 0;
  bool done = !(0.0 < t_end);
  while (!done) {
    bool lz = lanczos != 0 && herm;
    for (int attempt = 0; attempt < 2; ++attempt) {
      small_krylov(J, lz, herm, kap, m, A, cA, Q, p, psi, red, ort, turn);
      __syncthreads();
      small_projectors(m, me, n, Z, ort.top, Q, P, X);
      if (!lz) break;
      // a Lanczos basis must be orthonormal: max |sum_t P_t - I| <= ORTHO_TOL
      const double mall = small_ortho_err(me, m, P, terms, cstat);
      if (mall <= ORTHO_TOL) break;
      nf++;
      lz = false;  // rebuild this basis with full MGS
    }
    nb++;
    expm_one<false>(me, m, A, E, dt, X, rowsum, band, lz, tid, SMALL_THREADS);
    __syncthreads();
    double2* W = X;  // 4 x npair weights in the spent expm scratch
    dt_weights(m, me, P, W, tid, SMALL_THREADS);
    __syncthreads();
    if (warp < 4) {
      double2 c = lane < me ? cA[lane] : cz();
      if (dt_steps(m, me, E, W, c, t, k, steps, T, dt, t_end, tol, o, part, terms)) {
        if (tid == 0) atomicExch(err, 1);
        done = true;
      }
      if (warp == 0 && lane < me) cA[lane] = c;  // for psi = Q c
      if (tid == 0) {
        loop_t = t;
        loop_k = k;
        loop_steps = steps;
        loop_done = done ? 1 : 0;
      }
    }
    __syncthreads();  // warps 4-7 wait here
    t = loop_t;
    k = loop_k;
    steps = loop_steps;
    done = loop_done != 0;
    if (!done) done = !(t < t_end);
    if (!done) small_psi(me, n, Q, cA, psi);
    // c lives in cA; the next build rewrites it after a barrier
    __syncthreads();
  }
  if (tid == 0) {
    atomicAdd((unsigned long long*)nsteps, (unsigned long long)steps);
    atomicAdd(&counts[0], nb);
    atomicAdd(&counts[1], nf);
  }
}

// ---------------------------------------------------------------------------
// Pair form: a cluster of two CTAs per sample, for calls whose clusters are
// all resident at once (at most half as many samples as SMs: the dim-288
// workload runs 64 samples on 152 SMs, so one CTA per sample leaves 88 SMs
// idle). The main CTA (cluster rank 0) keeps
// the sample's serial path: the Krylov builds, the expm, the recurrence
// c <- E c of the dt loop with its stop test, and psi = Q c. The helper CTA
// (rank 1) takes the work off that path:
//  * the four projector Grams, staged from the main CTA's basis through
//    distributed shared memory, and the Lanczos orthonormality check, while
//    the main CTA runs the expm of the same basis;
//  * the populations Re(c^H P_X c) of every dt step, from the coordinates c
//    that the main CTA's dt loop stores into the helper's shared memory in
//    segments of at most hmax steps (two buffers): the helper evaluates a
//    segment while the main CTA runs the next one, psi = Q c and the next
//    Krylov build.
// The main CTA's dt step is then c' = E c on four warps and the stop test on a
// fifth, beside the next step.
// Control flow is uniform across the cluster: a flag that ends a loop is
// written to both CTAs' shared memory before a cluster barrier and read after
// it, and every thread of both CTAs reaches every cluster barrier. The
// arithmetic is k_small_prop's except for the order in which the populations
// add their pair terms (each lane's pairs in order, then a shuffle tree), so
// populations agree with it to rounding and the rebuild schedule is the same.
struct PairCtrl {
  int ok;       // the basis passed the orthonormality check (written by the helper)
  int over;     // the last segment ran out of output slots (main CTA)
  int cnt[2];   // per history buffer (written by the main CTA): steps in the segment,
  int k0[2];    // output index of its first step,
  int more[2];  // whether the build continues past it,
  int done[2];  // whether the sample's propagation has ended
};

// Populations of cnt consecutive dt steps from their Krylov coordinates
// (hist[st * m + i]), with the build's Hermitian weights W (4 x npair) and
// pair table: step st on warp st mod SMALL_WARPS, the lanes over the pairs
// (each lane adds its pairs' terms in order), then k_small_prop's
// reduce-scatter; lanes 0, 8, 16, 24 write the four populations of output
// index k0 + st. Called by all threads of the helper CTA.
__device__ __forceinline__ void small_pair_forms(int cnt, int k0, int m, int npair, const double2* hist,
                                                 const double2* W, const int2* pij, double* o, int T) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int st = warp; st < cnt; st += SMALL_WARPS) {
    const double2* cv = hist + (size_t)st * m;
    double f0 = 0.0, f1 = 0.0, f2 = 0.0, f3 = 0.0;
    for (int pp = lane; pp < npair; pp += 32) {
      const int2 ij = pij[pp];
      const double2 ci = cv[ij.x], cj = cv[ij.y];
      const double gx = fma(ci.x, cj.x, ci.y * cj.y), gy = fma(ci.x, cj.y, -ci.y * cj.x);
      const double2 w0 = W[pp], w1 = W[npair + pp], w2 = W[2 * npair + pp], w3 = W[3 * npair + pp];
      f0 = fma(w0.x, gx, fma(w0.y, gy, f0));
      f1 = fma(w1.x, gx, fma(w1.y, gy, f1));
      f2 = fma(w2.x, gx, fma(w2.y, gy, f2));
      f3 = fma(w3.x, gx, fma(w3.y, gy, f3));
    }
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    double ka = h16 ? f2 : f0, kb = h16 ? f3 : f1;
    ka += __shfl_xor_sync(0xffffffffu, h16 ? f0 : f2, 16);
    kb += __shfl_xor_sync(0xffffffffu, h16 ? f1 : f3, 16);
    double v = h8 ? kb : ka;
    v += __shfl_xor_sync(0xffffffffu, h8 ? ka : kb, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if ((lane & 7) == 0) {
      const int ty = lane >> 3;
      const int slot = ty == 0 ? 2 : (ty == 1 ? 0 : (ty == 2 ? 1 : 3));  // proj type -> obs slot
      o[(size_t)slot * T + k0 + st] = v;
    }
  }
}

// Dynamic shared memory of k_small_pair (complex elements). Main CTA: A, E
// (m^2 each), c (m), expm scratch (5 m^2), then the vectors when vec_smem.
// Helper CTA: P (4 m^2), projector staging (small_gram_elems), weights
// (4 m(m+1)/2), pair table (m(m+1)/2 int2), history (2 hmax m).
__host__ __device__ __forceinline__ size_t pair_main_elems(int m, int n, bool vec_smem) {
  const size_t mm = (size_t)m * m;
  return 7 * mm + (size_t)m + (vec_smem ? (size_t)(m + 2) * n : 0);
}
__host__ __device__ __forceinline__ size_t pair_help_elems(int m, int hmax) {
  const size_t mm = (size_t)m * m, np = (size_t)m * (m + 1) / 2;
  return 4 * mm + small_gram_elems(m) + 4 * np + (np + 1) / 2 + 2 * (size_t)hmax * m;
}

// Grid: two CTAs per sample (global sample s = blockIdx.x / 2), clusters of
// two; arguments as k_small_prop's, plus hmax (steps per history buffer).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SMALL_THREADS, 1)
    k_small_pair(const SmallJob* __restrict__ jobs, const int* __restrict__ sjob, const int* __restrict__ scol,
                 const int64_t* __restrict__ soff, double2* __restrict__ work, Theta th, int m, int T, double dt,
                 int nstep, double tol, int lanczos, int vec_smem, int hmax, double* __restrict__ obs,
                 long long* __restrict__ nsteps, unsigned long long* __restrict__ counts, int* __restrict__ err) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double2 smem[];
  __shared__ double rowsum[SPC_MAX_M];
  __shared__ int band[4];
  __shared__ SmallRed red;
  __shared__ SmallOrtho ort;
  __shared__ double part[4][2 * SMALL_MAX_M];
  __shared__ double terms[16];
  __shared__ double cstat[2];
  __shared__ int holds;
  __shared__ PairCtrl ctrl;

  const int rank = (int)cluster.block_rank();
  const int s = blockIdx.x >> 1;
  const SmallJob J = jobs[sjob[s]];
  const int n = J.n, Z = J.Z, me = J.me;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t mm = (size_t)m * m;
  const int npair = me * (me + 1) / 2;
  // main CTA's layout
  double2* A = smem;
  double2* E = A + mm;
  double2* cA = E + mm;
  double2* X = cA + m;
  double2* Q = vec_smem ? X + 5 * mm : work + soff[s];
  double2* p = Q + (size_t)m * n;
  double2* psi = p + n;
  // helper CTA's layout
  const size_t np_max = (size_t)m * (m + 1) / 2;
  double2* P = smem;
  double2* V = P + 4 * mm;
  double2* W = V + small_gram_elems(m);
  int2* pij = reinterpret_cast<int2*>(W + 4 * np_max);
  double2* H = W + 4 * np_max + (np_max + 1) / 2;
  // the other CTA's shared memory
  PairCtrl* ctrl_main = cluster.map_shared_rank(&ctrl, 0);
  PairCtrl* ctrl_help = cluster.map_shared_rank(&ctrl, 1);
  const SmallOrtho* ort_main = cluster.map_shared_rank(&ort, 0);
  double2* H_help = cluster.map_shared_rank(H, 1);
  const double2* Q_main = vec_smem ? cluster.map_shared_rank(Q, 0) : Q;
  const bool herm = J.kappa != nullptr;
  const double kap = herm ? *J.kappa : 0.0;
  double* o = obs + (size_t)s * 4 * T;

  if (rank == 0) {
    // psi_0 = theta (x) z (kron_vector)
    const double2* zk = J.zk + (size_t)scol[s] * Z;
    for (int r = tid; r < n; r += SMALL_THREADS) psi[r] = cmul(th.v[r / Z], zk[r % Z]);
  }
  __syncthreads();
  // The dt loop's layout: thread (part q, component x) of warps 0-3 has columns
  // [q ncol, (q + 1) ncol) of row x / 2
  const int nq = min(4, 64 / me), ncol = (me + nq - 1) / nq;
  const int dq = tid / (2 * me), dx = tid - dq * 2 * me;
  const bool dimag = (dx & 1) != 0;
  int k = 1;  // outputs 0 hold the initial populations (k_obs_init); steps done: k - 1
  int turn = 0;
  unsigned long long nb = 0, nf = 0;
  bool done = nstep == 0;
  while (!done) {
    bool lz = lanczos != 0 && herm;
    const int k_build = k;
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (rank == 0) small_krylov(J, lz, herm, kap, m, A, cA, Q, p, psi, red, ort, turn);
      cluster.sync();  // basis, A and c complete
      if (rank == 0) {
        expm_one<false>(me, m, A, E, dt, X, rowsum, band, lz, tid, SMALL_THREADS);
        __syncthreads();
      } else {
        small_projectors(m, me, n, Z, ort_main->top, Q_main, P, V);
        // a Lanczos basis must be orthonormal: max |sum_t P_t - I| <= ORTHO_TOL
        const bool okv = !lz || small_ortho_err(me, m, P, terms, cstat) <= ORTHO_TOL;
        if (tid == 0) {
          ctrl.ok = okv ? 1 : 0;
          ctrl_main->ok = okv ? 1 : 0;
        }
        dt_weights(m, me, P, W, tid, SMALL_THREADS);
        for (int idx = tid; idx < npair; idx += SMALL_THREADS) pij[idx] = dt_pair(me, idx);
        __syncthreads();
      }
      // dt loop (:348-364) in segments of at most hmax steps. The first segment
      // runs while the helper forms the Grams and the check of the same basis: a
      // basis that fails it is rebuilt, and the segment's steps count for nothing.
      // c lives in cA. A step is bound by the FP64 pipes of four schedulers and by
      // latency, so it is laid out for few FP64 instructions in a row: c' = E c by
      // components, 2 ncol multiply-adds a thread on coefficients in registers,
      // the parts added by one thread a component; steps are counted (nstep, the
      // host's count of the reference's t < t_end loop) instead of adding t; and
      // warp 4 stores c' into the helper's history and applies the stop test while
      // warps 0-3 already form the next step, which counts for nothing after the
      // last. Before (lane = row, every warp adding the parts, testing and
      // carrying t) a step at m = 20 took 3060 clocks, now 1860: 64 samples at
      // dim 288, 5000 steps 22.1 -> 19.0 ms; dim 48, m = 10, 500 steps 1.88 -> 1.64 ms.
      bool ok = true;
      int buf = 0;
      for (;;) {
        if (rank == 0) {
          if (warp < 5) {
            double2 ec[SMALL_MAX_M / 2];
#pragma unroll
            for (int u = 0; u < SMALL_MAX_M / 2; ++u) {
              const int j = dq * ncol + u;
              ec[u] = dq < nq && u < ncol && j < me ? E[(dx >> 1) + j * m] : cz();
              ec[u].y = flip(ec[u].y, !dimag);
            }
            double2* hist = H_help + (size_t)buf * hmax * m;
            const int k0 = k;
            int cnt = 0;
            bool go = true, overflow = false;
            for (;;) {
              const bool last = cnt == hmax || k > nstep;
              const bool full = !last && k >= T;  // output full (guard; every chain thread takes it)
              if (warp == 4) {
                if (cnt > 0) {
                  const double2 c = lane < me ? cA[lane] : cz();
                  if (lane < me) hist[(size_t)(cnt - 1) * m + lane] = c;
                  const bool in = krylov_holds(c, me, tol);
                  if (lane == 0) holds = in ? 1 : 0;
                }
              } else if (!last && !full && dq < nq) {
                double a = 0.0;
#pragma unroll
                for (int u = 0; u < SMALL_MAX_M / 2; ++u) {
                  if (u >= ncol) break;
                  const double2 c = cA[min(dq * ncol + u, me - 1)];
                  a = fma(ec[u].x, dimag ? c.y : c.x, a);
                  a = fma(ec[u].y, dimag ? c.x : c.y, a);
                }
                part[dq][dx] = a;
              }
              small_bar5();
              if (cnt > 0) go = holds != 0;
              overflow = go && full;
              if (!go || last || full) break;
              if (tid < 2 * me) {
                double a = part[0][tid];
                if (nq > 1) a += part[1][tid];
                if (nq > 2) a += nq > 3 ? part[2][tid] + part[3][tid] : part[2][tid];
                reinterpret_cast<double*>(cA)[tid] = a;
              }
              small_bar5();
              k = k + 1;
              cnt++;
            }
            const bool more = !overflow && cnt == hmax && go && k <= nstep;
            const bool dn = overflow || (!more && k > nstep);
            if (tid == 0) {
              ctrl.over = overflow ? 1 : 0;
              ctrl.more[buf] = more ? 1 : 0;
              ctrl.done[buf] = dn ? 1 : 0;
              ctrl_help->cnt[buf] = cnt;
              ctrl_help->k0[buf] = k0;
              ctrl_help->more[buf] = more ? 1 : 0;
              ctrl_help->done[buf] = dn ? 1 : 0;
            }
          }
          __syncthreads();
        }
        // history segment, flags and (first segment) the check visible to both;
        // the flags of buffer buf are next written two segments on, after a
        // cluster barrier that every thread reaches only once it has read them
        cluster.sync();
        ok = ctrl.ok != 0;
        const bool more = ok && ctrl.more[buf] != 0;
        done = ok && ctrl.done[buf] != 0;
        if (ok && rank == 0 && tid == 0 && ctrl.over) atomicExch(err, 1);
        if (ok && rank == 1)
          small_pair_forms(ctrl.cnt[buf], ctrl.k0[buf], m, npair, H + (size_t)buf * hmax * m, W, pij, o, T);
        if (!more) break;
        buf ^= 1;
      }
      if (ok) break;
      // every thread has read the flags before the next segment writes them
      cluster.sync();
      nf++;
      lz = false;  // rebuild this basis with full MGS
      k = k_build;
    }
    nb++;
    if (rank == 0 && !done) small_psi(me, n, Q, cA, psi);
    __syncthreads();
  }
  // keep the helper's shared memory alive until the main CTA's last remote
  // access has completed
  cluster.sync();
  if (rank == 0 && tid == 0) {
    atomicAdd((unsigned long long*)nsteps, (unsigned long long)(k - 1));
    atomicAdd(&counts[0], nb);
    atomicAdd(&counts[1], nf);
  }
}

// Dynamic shared memory of k_small_prop for Krylov dimension m (bytes),
// without the vectors.
static size_t small_smem_bytes(int m) {
  const size_t mm = (size_t)m * m;
  return sizeof(double2) * (6 * mm + 2 * (size_t)m + std::max<size_t>(5 * mm, small_gram_elems(m)));
}

// Whether a call runs on k_small_prop (sets smem). Rows, m, shared memory
// and device memory must fit; in SPC_SAMPLE_AUTO mode also every job's build
// must be small (an estimate of its FP64 FMAs: SpMM, passes, projectors,
// expm) and the samples at most two waves of resident CTAs.
static bool small_path_fits(Handle* h, const std::vector<JobSpec>& jobs, int m, int T, size_t& smem) {
  if (m > SMALL_MAX_M || jobs.empty()) return false;
  int64_t G = 0;
  double bytes = 0.0, wmax = 0.0;
  for (const JobSpec& j : jobs) {
    if (j.n > SMALL_NMAX || j.n < 4 || j.M < 1) return false;
    G += j.M;
    bytes += 16.0 * (double)(m + 2) * j.n * j.M;
    const double me = std::min(m, j.n), n = j.n;
    // MGS rounds (rates unequal, or MGS requested) add ~m^2 n/2 complex FMAs
    const bool mgs = !(h->krylov_method == 1 || h->krylov_method == 2) || !j.herm_shift;
    wmax = std::max(wmax, 4.0 * me * (double)j.nnz + 16.0 * me * n + 2.0 * n * me * me + 48.0 * me * me * me +
                              (mgs ? 2.0 * me * me * n : 0.0));
  }
  if (G > INT32_MAX) return false;
  bytes += 32.0 * T * (double)G + 16.0 * (double)G;
  smem = small_smem_bytes(m);
  if (smem + SMALL_STATIC > h->smem_optin) return false;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
  double held = 0.0;
  for (const Handle::Buf* b : {&h->Q, &h->obs, &h->tt, &h->kk, &h->done}) held += (double)b->bytes;
  double budget = (double)free_b + held - (512.0 * (1 << 20) + 0.02 * (double)total_b);
  if (h->mem_limit) budget = std::min(budget, (double)h->mem_limit);
  if (bytes > budget) return false;
  if (h->sample_path == SPC_SAMPLE_ON || h->sample_path == SPC_SAMPLE_SINGLE) return true;
  if (allow_smem(k_small_prop<2>, h->smem_optin - SMALL_STATIC) != cudaSuccess) return false;
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_small_prop<2>, SMALL_THREADS, smem) != cudaSuccess) return false;
  return wmax <= 2.5e6 && G <= 2LL * h->sm_count * std::max(1, b);
}

// propagate_batch on k_small_prop: one launch for every sample of every job,
// then the per-job average (k_average).
static int propagate_small(Handle* h, const double* theta, const double* init_pop, const std::vector<JobSpec>& jobs,
                           double dt, double t_end, int m, double tol, int T, size_t smem) {
  auto t_start = std::chrono::steady_clock::now();
  cudaStream_t st = h->stream;
  const int nj = (int)jobs.size();
  int G = 0;
  for (const JobSpec& j : jobs) G += j.M;
  std::vector<SmallJob> sj(nj);
  std::vector<JobOut> jo(nj);
  std::vector<int> sjob(G), scol(G);
  std::vector<int64_t> soff(G);
  bool lanczos = h->krylov_method == 1 || h->krylov_method == 2;
  int64_t wt = 0;
  for (int k = 0, g = 0; k < nj; ++k) {
    const JobSpec& j = jobs[k];
    lanczos = lanczos && j.herm_shift;
    sj[k] = SmallJob{j.n, j.n / 4, std::min(m, j.n), j.rowptr, j.split, j.col, j.val,
                     j.herm_shift ? j.kappa : nullptr, j.rexp, j.zk};
    jo[k] = JobOut{g, j.M, j.out};
    for (int s = 0; s < j.M; ++s, ++g) {
      sjob[g] = k;
      scol[g] = s;
      soff[g] = wt;
      wt += (int64_t)(m + 2) * j.n;
    }
  }
  // plan: jobs | sample -> job | sample -> column | sample -> work offset
  const size_t o_sjob = sizeof(SmallJob) * nj;
  const size_t o_scol = o_sjob + sizeof(int) * G;
  const size_t o_soff = (o_scol + sizeof(int) * G + 7) / 8 * 8;
  const size_t plan_bytes = o_soff + sizeof(int64_t) * G;
  if (h->ensure(h->Q, sizeof(double2) * wt) || h->ensure(h->obs, sizeof(double) * 4 * (size_t)T * G) ||
      h->ensure(h->tt, sizeof(double) * G) || h->ensure(h->kk, sizeof(int) * G) ||
      h->ensure(h->done, sizeof(int) * G) || h->ensure(h->err, 32) || h->ensure(h->plan, plan_bytes) ||
      h->ensure(h->jobtab, sizeof(JobOut) * nj + 64))
    return SPC_ERR_ALLOC;
  std::vector<char> hp(plan_bytes);
  std::memcpy(hp.data(), sj.data(), sizeof(SmallJob) * nj);
  std::memcpy(hp.data() + o_sjob, sjob.data(), sizeof(int) * G);
  std::memcpy(hp.data() + o_scol, scol.data(), sizeof(int) * G);
  std::memcpy(hp.data() + o_soff, soff.data(), sizeof(int64_t) * G);
  char* plan = (char*)h->plan.p;
  int64_t launches0 = h->launches;
  CK(cudaMemcpyAsync(plan, hp.data(), plan_bytes, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(h->jobtab.p, jo.data(), sizeof(JobOut) * nj, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(h->err.p, 0, 32, st));
  double* d_obs = (double*)h->obs.p;
  // slots past a sample's last step stay zero, as the reference's arrays
  CK(cudaMemsetAsync(d_obs, 0, sizeof(double) * 4 * (size_t)T * G, st));
  k_obs_init<<<(G + 127) / 128, 128, 0, st>>>(G, T, init_pop[0], init_pop[1], init_pop[2], init_pop[3], d_obs,
                                               (double*)h->tt.p, (int*)h->kk.p, (int*)h->done.p);
  h->count_launch();
  Theta th;
  for (int e = 0; e < 4; ++e) th.v[e] = make_double2(theta[2 * e], theta[2 * e + 1]);
  // the vectors in shared memory when every job's fit beside the matrices
  int nmax = 0;
  for (const JobSpec& j : jobs) nmax = std::max(nmax, j.n);
  const size_t budget = h->smem_optin > SMALL_STATIC ? h->smem_optin - SMALL_STATIC : 0;  // less the static shared memory
  int* d_err = (int*)h->err.p;
  long long* d_nsteps = (long long*)((char*)h->err.p + 8);
  unsigned long long* d_counts = (unsigned long long*)((char*)h->err.p + 16);
  // pair form (two CTAs per sample) when the samples fill at most half the
  // SMs and its shared memory fits: history buffers of up to 64 steps
  bool pair = h->sample_path != SPC_SAMPLE_SINGLE && 2 * (int64_t)G <= h->sm_count;
  CK(cudaGetLastError());  // a failed query below is cleared, not an earlier error
  int hmax = 64;
  size_t psmem = 0;
  bool pvec = false;
  if (pair) {
    while (hmax > 8 && sizeof(double2) * pair_help_elems(m, hmax) > budget) hmax /= 2;
    const size_t help = sizeof(double2) * pair_help_elems(m, hmax);
    pvec = sizeof(double2) * pair_main_elems(m, nmax, true) <= budget;
    psmem = std::max(help, sizeof(double2) * pair_main_elems(m, nmax, pvec));
    pair = psmem <= budget &&
           allow_smem(k_small_pair, budget) == cudaSuccess;
    if (pair) {
      // every cluster resident at once (SMs pair up within a GPC, so this can
      // be fewer than half the SMs)
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * G);
      cfg.blockDim = dim3(SMALL_THREADS);
      cfg.dynamicSmemBytes = psmem;
      cfg.stream = st;
      int ncl = 0;
      pair = cudaOccupancyMaxActiveClusters(&ncl, k_small_pair, &cfg) == cudaSuccess && ncl >= G;
    }
    if (!pair) (void)cudaGetLastError();  // fall back to one CTA per sample
  }
  int pe = h->prof.begin(st);
  if (pair) {
    // steps of the reference's loop (t += dt while t < t_end), past T the guard's
    int nstep = 0;
    for (double t = 0.0; t < t_end && nstep < T; t = t + dt) ++nstep;
    k_small_pair<<<2 * G, SMALL_THREADS, psmem, st>>>((const SmallJob*)plan, (const int*)(plan + o_sjob),
                                                      (const int*)(plan + o_scol), (const int64_t*)(plan + o_soff),
                                                      (double2*)h->Q.p, th, m, T, dt, nstep, tol, lanczos ? 1 : 0,
                                                      pvec ? 1 : 0, hmax, d_obs, d_nsteps, d_counts, d_err);
  } else {
    // With more samples than SMs two CTAs share one where their shared memory lets
    // them, and their vectors stay in global memory (L2): two waves of lone CTAs
    // take 6.0 ms where these take 4.5 (201 samples at dim 288, MGS, m = 20).
    // Otherwise (fewer samples, or m past 20) the CTA has the SM's registers, and
    // shared memory for its vectors if they fit.
    const size_t vbytes = sizeof(double2) * (size_t)(m + 2) * nmax;
    int ctas = 1;
    if (G > h->sm_count) {
      CK(allow_smem(k_small_prop<2>, budget));
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, k_small_prop<2>, SMALL_THREADS, smem));
    }
    const bool vec_smem = ctas < 2 && smem + vbytes + SMALL_STATIC <= h->smem_optin;
    if (vec_smem) smem += vbytes;
    const auto prop = ctas < 2 ? k_small_prop<1> : k_small_prop<2>;
    CK(allow_smem(prop, budget));
    prop<<<G, SMALL_THREADS, smem, st>>>((const SmallJob*)plan, (const int*)(plan + o_sjob),
                                                 (const int*)(plan + o_scol), (const int64_t*)(plan + o_soff),
                                                 (double2*)h->Q.p, th, m, T, dt, t_end, tol, lanczos ? 1 : 0,
                                                 vec_smem ? 1 : 0, d_obs,
                                                 d_nsteps, d_counts, d_err);
  }
  h->prof.end(st, pe, PK_SAMPLE, 0.0, 0.0);
  h->count_launch();
  for (int j0 = 0; j0 < nj; j0 += 65535) {
    const int cnt = std::min(65535, nj - j0);
    k_average<<<dim3((4 * T + 255) / 256, cnt), 256, 0, st>>>((const JobOut*)h->jobtab.p, j0, T, d_obs);
    h->count_launch();
  }
  CK(cudaGetLastError());
  unsigned char eh[32];
  CK(cudaMemcpyAsync(eh, h->err.p, 32, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  h->prof.collect();
  int err0 = 0;
  long long nsteps = 0;
  unsigned long long counts[2] = {0, 0};
  std::memcpy(&err0, eh, 4);
  std::memcpy(&nsteps, eh + 8, 8);
  std::memcpy(counts, eh + 16, 16);
  h->stats.krylov_builds = (int64_t)counts[0];
  h->stats.lanczos_fallbacks = (int64_t)counts[1];
  h->stats.rounds = 1;
  h->stats.sample_steps = nsteps;
  h->stats.kernel_launches = h->launches - launches0;
  h->stats.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
  if (err0 == 1) return set_error(SPC_ERR_NUMERIC, "time index overflow: the dt loop ran past %d output slots", T);
  return SPC_OK;
}
