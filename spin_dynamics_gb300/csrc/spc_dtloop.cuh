// The dt loop (src/qm_dynamics.f90:348-364) of one sample on four warps, for
// Krylov dimensions up to 32. Included by spc_propagate.cu inside namespace spc.

// Stop test of the dt loop, |c_{me-1}|^2 <= tol |c|^2, for the coordinates in a
// warp's lanes (zero past me). In single precision where that decides it (two
// sides apart by more than its rounding): five FP64 adds with their shuffles
// take 545 clocks, more than half of a step's products.
__device__ __forceinline__ bool krylov_holds(double2 c, int me, double tol) {
  const float x = cut_float(c.x), y = cut_float(c.y);
  const float own = x * x + y * y;
  float s = own;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float last = __shfl_sync(0xffffffffu, own, me - 1), lim = (float)tol * s;
  if (lim > 1e-30f && lim < 1e30f && fabsf(last - lim) > 1e-4f * lim) return last <= lim;
  const double n2 = warp_sum(fma(c.x, c.x, c.y * c.y));
  const double l2 = __shfl_sync(0xffffffffu, c.x * c.x + c.y * c.y, me - 1);
  return l2 <= tol * n2;
}

// Barrier of warps 0-3 (the dt loop's warps; a CTA's others wait at its next
// __syncthreads).
__device__ __forceinline__ void small_bar4() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ void small_bar5() { asm volatile("bar.sync 2, 160;" ::: "memory"); }  // of warps 0-4

// pair number idx of (i, j >= i) in row order
__device__ __forceinline__ int2 dt_pair(int me, int idx) {
  int i = 0;
  while (idx >= me - i) {
    idx -= me - i;
    ++i;
  }
  return make_int2(i, i + idx);
}
// Hermitian weights W_t = (s Re P_t, -s Im P_t) of the pairs i <= j (s = 1 on the
// diagonal, 2 above it) of the four projectors P (m x m each)
__device__ __forceinline__ void dt_weights(int m, int me, const double2* P, double2* W, int tid, int nt) {
  const int npair = me * (me + 1) / 2;
  for (int idx = tid; idx < npair; idx += nt) {
    const int2 ij = dt_pair(me, idx);
    const double s = ij.x == ij.y ? 1.0 : 2.0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double2 v = P[(size_t)t * m * m + ij.x + (size_t)ij.y * m];
      W[t * npair + idx] = make_double2(s * v.x, -s * v.y);
    }
  }
}

// c <- E c; P_X(t) = Re(c^H P_X c) to o (S, T0, Tp, Tm rows of T); until the
// last Krylov coordinate grows past tol or the window ends. Warps 0-3 (all 128
// threads), c in the lanes of each. One warp per scheduler: GB300's FP64 pipe sits
// in each scheduler and a warp instruction holds it for the same time whatever
// its active lanes, so the step is laid out to issue few FP64 warp instructions:
//  * c' = E c with lane = row and warp w over the columns j = w mod 4 (c_j by
//    shuffle); every warp adds the four partials in warp order, so each holds c'
//    in its lanes and no further barrier is needed;
//  * the four forms over the pairs i <= j with g_ij = conj(c_i) c_j shared by the
//    types: 12 FP64 operations a pair, where four products P_X c take 16 per
//    matrix element;
//  * each warp's four sums by a reduce-scatter over its lanes (6 adds instead of
//    20), then the warps' sums added in warp order.
// part and terms are shared memory. Returns whether the output is full (guard).
#define DT_ROUNDS 5  // pair rounds over 128 threads: 32 * 33 / 2 <= 5 * 128
__device__ __forceinline__ bool dt_steps(int m, int me, const double2* E, const double2* W, double2& c, double& t, int& k,
                                         long long& steps, int T, double dt, double t_end, double tol, double* o,
                                         double2 (*part)[32], double* terms) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int npair = me * (me + 1) / 2;
  int2 pr[DT_ROUNDS];
#pragma unroll
  for (int r = 0; r < DT_ROUNDS; ++r) {
    const int idx = r * 128 + tid;
    pr[r] = idx < npair ? dt_pair(me, idx) : make_int2(-1, 0);
  }
  bool go = true;
  while (go && t < t_end) {
    if (k >= T) return true;  // every thread takes it
    double2 a = cz();
    for (int j = warp; j < me; j += 4) {
      const double2 cj = make_double2(__shfl_sync(0xffffffffu, c.x, j), __shfl_sync(0xffffffffu, c.y, j));
      if (lane < me) a = cfma(E[lane + j * m], cj, a);
    }
    part[warp][lane] = a;
    small_bar4();
    double2 cn = cz();
    if (lane < me) cn = cadd(cadd(cadd(part[0][lane], part[1][lane]), part[2][lane]), part[3][lane]);
    double f0 = 0.0, f1 = 0.0, f2 = 0.0, f3 = 0.0;
#pragma unroll
    for (int r = 0; r < DT_ROUNDS; ++r) {
      if (r * 128 + warp * 32 >= npair) break;  // no pair of this warp left
      const int i = max(pr[r].x, 0), j = pr[r].y;
      const double cix = __shfl_sync(0xffffffffu, cn.x, i), ciy = __shfl_sync(0xffffffffu, cn.y, i);
      const double cjx = __shfl_sync(0xffffffffu, cn.x, j), cjy = __shfl_sync(0xffffffffu, cn.y, j);
      if (pr[r].x >= 0) {
        const double gx = fma(cix, cjx, ciy * cjy), gy = fma(cix, cjy, -ciy * cjx);
        const int pp = r * 128 + tid;
        const double2 w0 = W[pp], w1 = W[npair + pp], w2 = W[2 * npair + pp], w3 = W[3 * npair + pp];
        f0 = fma(w0.x, gx, fma(w0.y, gy, f0));
        f1 = fma(w1.x, gx, fma(w1.y, gy, f1));
        f2 = fma(w2.x, gx, fma(w2.y, gy, f2));
        f3 = fma(w3.x, gx, fma(w3.y, gy, f3));
      }
    }
    // reduce-scatter: lanes 8t..8t+7 end with the warp's sum of form t
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    double ka = h16 ? f2 : f0, kb = h16 ? f3 : f1;
    ka += __shfl_xor_sync(0xffffffffu, h16 ? f0 : f2, 16);
    kb += __shfl_xor_sync(0xffffffffu, h16 ? f1 : f3, 16);
    double v = h8 ? kb : ka;
    v += __shfl_xor_sync(0xffffffffu, h8 ? ka : kb, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if ((lane & 7) == 0) terms[4 * warp + (lane >> 3)] = v;
    small_bar4();
    if (tid < 4) {
      const int slot = tid == 0 ? 2 : (tid == 1 ? 0 : (tid == 2 ? 1 : 3));  // proj type -> obs slot
      o[(size_t)slot * T + k] = ((terms[tid] + terms[4 + tid]) + terms[8 + tid]) + terms[12 + tid];
    }
    go = krylov_holds(cn, me, tol);
    c = cn;
    t = t + dt;
    k = k + 1;
    steps++;
  }
  return false;
}

// The dt loop of a round's slots on dt_steps, one 128-thread CTA per sample;
// dynamic shared memory E (m^2) and the weights (2 m (m + 1)), complex. Against a
// warp per sample that forms the four products P_X c from global memory (k_dtloop)
// it issues half the FP64 instructions on four times the schedulers: dim 2304,
// 384 samples, m = 16, 120 steps 2.4 -> 0.84 ms; dim 55296, 512 samples, m = 30,
// 54 steps 3.2 -> 0.72 ms.
__host__ __device__ __forceinline__ size_t dt_smem_bytes(int m) {
  return sizeof(double2) * ((size_t)m * m + 2 * (size_t)m * (m + 1));
}
__global__ void __launch_bounds__(128)
    k_dtloop_cta(int m, int T, const TileInfo* __restrict__ tiles, const int* __restrict__ map,
                 const int* __restrict__ skip, const double2* __restrict__ Aexp, const double2* __restrict__ proj,
                 double2* __restrict__ cvec, double* __restrict__ tt, int* __restrict__ kk, int* __restrict__ done,
                 double* __restrict__ obs, double dt, double t_end, double tol, long long* __restrict__ nsteps,
                 int* __restrict__ err) {
  extern __shared__ double2 dsm[];
  __shared__ double2 part[4][32];
  __shared__ double terms[16];
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  if (map[w] < 0 || skip[w]) return;
  const int s = map[w], me = tiles[w / SPC_LANES].m;
  const size_t mm = (size_t)m * m;
  double2* E = dsm;
  double2* W = dsm + mm;
  for (int i = tid; i < (int)mm; i += 128) E[i] = Aexp[(size_t)w * mm + i];
  dt_weights(m, me, proj + (size_t)w * 4 * mm, W, tid, 128);
  double2 c = lane < me ? cvec[(size_t)w * m + lane] : cz();
  double t = tt[s];
  int k = kk[s];
  long long steps = 0;
  __syncthreads();
  if (dt_steps(m, me, E, W, c, t, k, steps, T, dt, t_end, tol, obs + (size_t)s * 4 * T, part, terms) && tid == 0)
    atomicExch(err, 1);
  if (tid < me) cvec[(size_t)w * m + tid] = c;
  if (tid == 0) {
    tt[s] = t;
    kk[s] = k;
    done[s] = t < t_end ? 0 : 1;
    atomicAdd((unsigned long long*)nsteps, (unsigned long long)steps);
  }
}
