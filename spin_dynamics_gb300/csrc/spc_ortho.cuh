// Orthogonalisation passes of the Krylov basis (get_krylov,
// src/qm_dynamics.f90:445-465). Included by spc_propagate.cu inside namespace
// spc.
//
// Sums over a tile's rows. GB300 adds two doubles per clock and SM, so a last
// CTA that adds the partial sums of several hundred others (32 samples each)
// takes 10 us and more. Here every CTA adds its sums to per-sample integers
// with 64-bit atomics: a double is an integer multiple of 2^(e - 110), e the
// exponent of a bound on the sum, held as two words (the bits from 2^50 up,
// the 50 below) that no carry couples. Integer sums do not depend on their
// order, so results repeat bit for bit, and their only rounding is the last
// one. The kernel that needs a sum reads it in its prologue. Three sets of
// accumulators rotate: a kernel adds to one, reads the one before and clears
// the one after. A square norm has a third word, 50 bits further down: a vector
// may be small against ||H|| (a state in a part of H far below the bound), and
// its norm has a double's bits down to 2^-53 of the bound.
#define ACC_VECS 15             // complex sums per sample (8 dots + 7 basis products)
#define ACC_MAX (4 * ACC_VECS)  // largest component's high word
#define ACC_BAD (4 * ACC_VECS + 1)
#define ACC_ROWS 64
typedef unsigned long long acc_t;

struct AccArgs {
  acc_t* acc;  // [3][tiles][ACC_ROWS][32]
  int ntiles, in, out, clear;
};
__device__ __forceinline__ acc_t* acc_tile(const AccArgs& A, int set, int tile) {
  return A.acc + ((size_t)set * A.ntiles + tile) * ACC_ROWS * SPC_LANES;
}
// x to the accumulator pair at p (stride 32; NORM: the upper or the lower pair of
// three words), |sum| <= 2^e; NaN, infinities and values past the bound mark the
// sample
template <bool NORM = false>
__device__ __forceinline__ void acc_add(acc_t* p, acc_t* bad, double x, int e) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)(b >> 52) & 0x7ff;
  if (ex == 0) return;
  if (ex - 1023 > e + 1) {
    *bad = 1;
    return;
  }
  const acc_t man = (b & 0xfffffffffffffll) | (1ull << 52);
  int sh = ex - 965 - e;  // <= 59
  if (NORM && sh < 0) {
    sh += 50;
    p += SPC_LANES;
  }
  acc_t lo, hi;  // man * 2^sh as hi 2^50 + lo
  if (sh >= 0) {
    lo = (man << sh) & ((1ull << 50) - 1);
    hi = sh >= 50 ? man << (sh - 50) : man >> (50 - sh);
  } else {
    const acc_t v = sh < -62 ? 0 : ((man >> (-sh - 1)) + 1) >> 1;
    lo = v & ((1ull << 50) - 1);
    hi = v >> 50;
  }
  if (b < 0) {
    lo = 0 - lo;
    hi = 0 - hi;
  }
  atomicAdd(p, hi);
  atomicAdd(p + SPC_LANES, lo);
}
__device__ __forceinline__ double acc_get(const acc_t* p, int e) {
  return ldexp(fma((double)(long long)p[0], 1125899906842624.0, (double)(long long)p[SPC_LANES]), e - 110);
}
// The sum of three words; the third adds less than 2^-54 of it from 2^16 units of
// the first on.
__device__ __forceinline__ double acc_get_norm(const acc_t* p, int e) {
  const double word = 1125899906842624.0;
  const long long hi = (long long)p[0], mid = (long long)p[SPC_LANES];
  double s = fma((double)hi, word, (double)mid);
  if (hi < 65536) {
    s = fma((double)hi, word * word, fma((double)mid, word, (double)(long long)p[2 * SPC_LANES]));
    e -= 50;
  }
  return ldexp(s, e - 110);
}
__device__ __forceinline__ void acc_clear(const AccArgs& A, int tile, int tid, int nth) {
  acc_t* p = acc_tile(A, A.clear, tile);
  for (int k = tid; k < ACC_ROWS * SPC_LANES; k += nth) p[k] = 0;
}
// exponents of the bounds: dots of a basis vector with p, p's square norm,
// products of two basis vectors
__device__ __forceinline__ int acc_dot_exp(const TileInfo& T) { return T.rexp; }
__device__ __forceinline__ int acc_norm_exp(const TileInfo& T) { return 2 * T.rexp; }
#define ACC_GRAM_EXP 4

// (float)v, cut off instead of rounded, from the words of v: the conversion
// instruction holds the FP64 pipe as a multiply-add does.
__device__ __forceinline__ float cut_float(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int e = (int)(hi >> 20 & 0x7ff) - 896;
  const unsigned mag = e <= 0 ? 0u : e >= 255 ? 0x7f800000u : (unsigned)e << 23 | (hi & 0xfffff) << 3 | lo >> 29;
  return __uint_as_float((hi & 0x80000000u) | mag);
}

// The leading 20 bits of a double below 2^127 as a float (0 below 2^-126), and a
// float as a double.
__device__ __forceinline__ float head_float(double v) {
  const unsigned h = (unsigned)__double2hiint(v);
  const unsigned u = max(h & 0x7fffffffu, 896u << 20) - (896u << 20);
  return __uint_as_float((u << 3) | (h & 0x80000000u));
}
__device__ __forceinline__ double wide_float(float f) {
  const unsigned b = __float_as_uint(f), u = b & 0x7fffffffu;
  const unsigned h = u < 0x00800000u ? 0u : (u >> 3) + (896u << 20);
  return __hiloint2double((int)(h | (b & 0x80000000u)), u < 0x00800000u ? 0 : (int)(b << 29));
}
// The same with infinities and NaN kept.
__device__ __forceinline__ double wide_any(float f) {
  const double v = wide_float(f);
  const bool special = (__float_as_uint(f) & 0x7f800000u) == 0x7f800000u;
  return __hiloint2double(__double2hiint(v) + (special ? 896 << 20 : 0), __double2loint(v));
}
// Whether coefficients of a Hamiltonian with ||H|| <= 2^rexp stay in the range of
// single precision, with room for their products: what they lose below 2^-126 is
// under 2^-86 of the bound.
__device__ __forceinline__ bool single_range(int rexp) { return rexp >= -40 && rexp <= 100; }
#define ORTHO_SMALL 44  // bits of a coefficient below the last beta

struct OrthoArgs {
  PassArgs p;
  AccArgs a;
  int ja, jd;      // first vector to subtract, first to project on
  double2* gram;   // [tile][basis vector][8][32]: <Q_j, Q_k> of the vectors k < j of j's block
  float far;       // size past which a product <Q_j, Q_k>, k < j - 1, calls for the recurrence
};
#define ORTHO_NB 8

// One pass over the rows of a work item: p -= sum_{v < NA} h_v Q_{ja+v}, then
// ND > 0: the sums <Q_{jd+v}, p>, v < ND;  ND = 0: ||p||^2 and p's largest
// component. Modified Gram-Schmidt projects on the basis in blocks of
// ORTHO_NB: with d_v = <Q_v, p> on the p that enters the block,
//   h_v = <Q_v, p - sum_{k < v} h_k Q_k> = d_v - sum_{k < v} <Q_v, Q_k> h_k,
// the coefficient of the one-vector pass in exact arithmetic (as the blocked
// forms of Swirydowicz, Langou, Ananthan, Yang and Thomas, "Low synchronization
// Gram-Schmidt and generalized minimal residual algorithms", Numer. Linear
// Algebra Appl. 28 (2021), e2343). The products of basis vectors are formed once,
// by the pass that first projects on the newer one (GRAM: Q_{jd+ND-1} is new).
// What bounds it: FP64 issue, 8 FMAs per vector and row as the one-vector pass;
// that pass took a launch, a read and a write of p and a serial last sum for each
// vector. Per Krylov step at m = 24, dim 9216, 64 samples (MGS): 12.5 passes of
// 29 us before, 3 of 31-82 us now; dim 55296, 32 samples, m = 30: 56.5 -> 27 ms a
// build. Blocks of eight: the newest block's pass holds 15 complex sums and 8
// vectors in 128 registers (with unequal rates it spills 68 bytes). Lanczos at dim 2304, 77 samples: the norm pass 15.3
// -> 10.1 us, k_spmm_blk with its projection 27.9 -> 19.5 us without the last sum.
// Small coefficients: where H is Hermitian up to a shift every h_v but the last
// two is of rounding size. A vector whose coefficients are below 2^-44 of the
// last beta (the coefficient of Q_{i-1}, so no more than ||p||) in all of a
// tile's samples is subtracted in single precision: eight of them, cut to 23
// bits, times q's leading 20 leave an error below 2^-60 of ||p||, 1/128 of one
// FP64 rounding of it. (A line at 2^-44 of the bound on ||H|| took everything
// for small where the state is in a part of H far below the bound.) 64 FP32
// multiply-adds issue in the time of one FP64, and the conversions are done on
// the words, since the conversion instruction also runs on the FP64 pipe. Up to
// two other vectors are subtracted beside them in FP64; a block with more
// (unequal rates) takes FP64 throughout. The block's pass and the norm pass
// at dim 2304, 384 samples, m = 16: 97 -> 68 and 35 -> 31 us; dim 55296, 32
// samples, m = 30: 200 -> 129 and 69 -> 59 us. A branch for each vector instead
// made the norm pass slower (40 and 80 us).
// HERM (every tile Hermitian up to a shift): the products of the new vector with
// the ones before its neighbour in FP32. They multiply coefficients h_k, k < i - 1,
// which are of the size of the basis' defect of orthogonality d times ||H||; an
// error of 1e-6 of the products adds 1e-6 d ||H|| and less. With them the products
// cost one FP64 sum instead of up to seven: dim 2304, 384 samples, m = 16, a newest
// block's pass 48 -> 42 us alone and 68 -> 54 us after a block; dim 55296, 32 samples,
// m = 30: 103 -> 96 and 129 -> 114 us.
// REAL: Lanczos on the Hermitian part; NA = 1 with ND = 1 takes beta_{i-1}
// (coef), with ND = 0 alpha_i.
template <int NA, int ND, bool GRAM, bool REAL, bool HERM = false>
__global__ void __launch_bounds__(256, 2) k_ortho(OrthoArgs o) {
  constexpr int NG = GRAM && ND > 1 ? ND - 1 : 0, NS = ND + NG;
  constexpr int NF = HERM && NG > 1 ? NG - 1 : 0;  // products in FP32
  constexpr int NR = ND == 0 ? 1 : (NS < 4 ? NS : 4);  // sums reduced at a time
  __shared__ double2 h[NA > 0 ? NA : 1][SPC_LANES];
  __shared__ double2 red[NR][SPC_WARPS][SPC_LANES];
  __shared__ unsigned mx[SPC_WARPS][SPC_LANES];
  __shared__ float2 hs[NA > 0 && !REAL ? NA : 1][SPC_LANES];
  __shared__ int large[NA > 0 && !REAL ? NA : 1];
  const PassArgs& a = o.p;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
  const int2 it = a.items[blockIdx.x];
  const TileInfo& T = a.tiles[it.x];
  const int i = a.col_i;
  if (i >= T.m) return;  // past this job's Krylov dimension
  const int w = it.x * SPC_LANES + tx;
  const bool act = a.map[w] >= 0;
  const bool first = it.y == 0;  // the CTA that records the tile's coefficients
  // the last column ends with its coefficients: no next vector
  const bool tail = ND == 0 && i == T.m - 1;
  if (tail && !first) return;
  if (first) acc_clear(o.a, it.x, tid, 256);
  unsigned lgm = 0;  // the vectors with large coefficients
  if (NA > 0) {
    const size_t mm = (size_t)a.m * a.m;
    const acc_t* in = acc_tile(o.a, o.a.in, it.x) + tx;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    if (REAL) {
      if (ty == 0) {
        double c;
        if (ND == 1) {
          c = act ? a.coef[w].x : 0.0;
        } else {
          c = in[ACC_BAD * SPC_LANES] ? nan : acc_get(in, acc_dot_exp(T));
          if (first && act)
            a.Ahess[(size_t)w * mm + i + (size_t)i * a.m] = make_double2(c, -*T.kappa);
        }
        h[0][tx] = make_double2(c, 0.0);
      }
      __syncthreads();
    } else {
      // d_v by warp v, then the corrections; the last block's newest vector has
      // its basis products in the accumulators
      const bool last = o.ja + NA == i + 1;
      const int jv = o.ja + ty;
      double2 d = cz();
      float2 gk[ORTHO_NB - 1];
      bool big = !single_range(T.rexp);
      unsigned eb = 0;  // the last beta's exponent
      if (i > 0) eb = abs_high(a.coef[w]) >> 20;
      double2* G = o.gram + ((size_t)it.x * a.m + jv) * ORTHO_NB * SPC_LANES + tx;
      if (ty < NA) {
        d = make_double2(acc_get(in + 4 * ty * SPC_LANES, acc_dot_exp(T)),
                         acc_get(in + (4 * ty + 2) * SPC_LANES, acc_dot_exp(T)));
        if (in[ACC_BAD * SPC_LANES]) d = make_double2(nan, nan);
        h[ty][tx] = d;
#pragma unroll
        for (int k = 0; k < NA - 1; ++k) {
          gk[k] = make_float2(0.f, 0.f);
          if (k < ty) {
            double2 gv;
            if (last && ty == NA - 1) {
              // <Q_k, Q_new>, stored as <Q_new, Q_k>
              gv = make_double2(acc_get(in + 4 * (NA + k) * SPC_LANES, ACC_GRAM_EXP),
                                -acc_get(in + (4 * (NA + k) + 2) * SPC_LANES, ACC_GRAM_EXP));
              if (first) G[k * SPC_LANES] = gv;
            } else {
              gv = G[k * SPC_LANES];
            }
            gk[k] = make_float2(cut_float(gv.x), cut_float(gv.y));
            big |= act && !(fabsf(gk[k].x) + fabsf(gk[k].y) < (k == ty - 1 ? 4e-9f : o.far));
          }
        }
      }
      // an orthonormal basis (products of rounding size): the corrections are
      // below 4e-9 of the coefficients (1e-5 of small ones between far vectors
      // where HERM), and first order and single precision leave at most 7e-15
      // (7 products, two factors cut to 23 bits) of the largest. The coefficient
      // recorded is the one subtracted, so H Q = Q A holds to rounding all the
      // same, and what is missing adds to a defect of orthogonality of the
      // products' own size. A basis past a breakdown takes the recurrence in
      // full, as do units past single precision.
      if (!__syncthreads_or(big ? 1 : 0)) {
        float2 c = make_float2(0.f, 0.f);
        if (ty < NA) {
#pragma unroll
          for (int k = 0; k < NA - 1; ++k) {
            const float hx = cut_float(h[k][tx].x), hy = cut_float(h[k][tx].y);
            c.x += gk[k].x * hx - gk[k].y * hy;
            c.y += gk[k].x * hy + gk[k].y * hx;
          }
          d = make_double2(d.x - wide_any(c.x), d.y - wide_any(c.y));
        }
        __syncthreads();
        if (ty < NA) h[ty][tx] = d;
      } else {
        for (int k = 0; k + 1 < NA; ++k) {
          __syncthreads();  // h_k is final
          if (ty > k && ty < NA) {
            double2 gv;
            if (last && ty == NA - 1)
              gv = make_double2(acc_get(in + 4 * (NA + k) * SPC_LANES, ACC_GRAM_EXP),
                                -acc_get(in + (4 * (NA + k) + 2) * SPC_LANES, ACC_GRAM_EXP));
            else
              gv = G[k * SPC_LANES];
            d = cfms(gv, h[k][tx], d);
            h[ty][tx] = d;
          }
        }
      }
      if (first && act && ty < NA) a.Ahess[(size_t)w * mm + jv + (size_t)i * a.m] = d;
      if (ty < NA) {
        // |h| < 2^-ORTHO_SMALL beta by the exponents; NaN and infinities are large
        // as are all where products would leave the range of single precision
        // (and a column without a beta)
        const bool lg = __any_sync(0xffffffffu, act && (eb < 1023 - 60 || eb > 1023 + 100 ||
                                                        (abs_high(d) >> 20) + ORTHO_SMALL >= eb));
        hs[ty][tx] = lg ? make_float2(0.f, 0.f) : make_float2(cut_float(d.x), cut_float(d.y));
        if (tx == 0) large[ty] = lg ? 1 : 0;
      }
      __syncthreads();
#pragma unroll
      for (int v = 0; v < NA; ++v) lgm |= (unsigned)large[v] << v;
    }
  }
  if (tail) return;
  const int nl = __popc(lgm), v0 = nl > 0 ? __ffs(lgm) - 1 : 0, v1 = nl > 1 ? 31 - __clz(lgm) : 0;
  const int n = act ? T.n : 0;
  const int stride = T.nio * SPC_WARPS;
  const size_t vs = (size_t)T.n * SPC_LANES;
  const double2* Qa = a.Q + T.q_off + (size_t)o.ja * vs + tx;
  const double2* Qd = a.Q + T.q_off + (size_t)o.jd * vs + tx;
  double2* P = a.P + T.p_off + tx;
  double2 acc[NS > 0 ? NS : 1];
#pragma unroll
  for (int v = 0; v < (NS > 0 ? NS : 1); ++v) acc[v] = cz();
  float2 accf[NF > 0 ? NF : 1];
#pragma unroll
  for (int v = 0; v < (NF > 0 ? NF : 1); ++v) accf[v] = make_float2(0.f, 0.f);
  unsigned top = 0;
  for (int r = it.y * SPC_WARPS + ty; r < n; r += stride) {
    const size_t off = (size_t)r * SPC_LANES;
    double2 p = P[off];
    double2 qd[ND > 0 ? ND : 1];
#pragma unroll
    for (int v = 0; v < ND; ++v) qd[v] = Qd[v * vs + off];
    if (NA > 0 && REAL) {
      const double2 q = Qa[off];
      const double c = h[0][tx].x;
      p.x = fma(-c, q.x, p.x);
      p.y = fma(-c, q.y, p.y);
    } else if (NA > 0 && nl > 2) {
#pragma unroll
      for (int v = 0; v < NA; ++v) p = cfms(h[v][tx], Qa[v * vs + off], p);
    } else if (NA > 0) {
      float sx = 0.f, sy = 0.f;
#pragma unroll
      for (int v = 0; v < NA; ++v) {
        const double2 x = Qa[v * vs + off];
        const float qx = head_float(x.x), qy = head_float(x.y);
        const float2 c = hs[v][tx];
        sx = fmaf(c.x, qx, fmaf(-c.y, qy, sx));
        sy = fmaf(c.x, qy, fmaf(c.y, qx, sy));
      }
      if (nl > 0) p = cfms(h[v0][tx], Qa[v0 * vs + off], p);  // in L1 by now
      if (nl > 1) p = cfms(h[v1][tx], Qa[v1 * vs + off], p);
      p.x -= wide_float(sx);
      p.y -= wide_float(sy);
    }
    if (NA > 0) P[off] = p;
    if (ND == 0) {
      acc[0].x = fma(p.x, p.x, acc[0].x);
      acc[0].x = fma(p.y, p.y, acc[0].x);
      top = max(top, abs_high(p));
    }
#pragma unroll
    for (int v = 0; v < ND; ++v) {
      if (REAL) {
        acc[v].x = fma(qd[v].x, p.x, acc[v].x);
        acc[v].x = fma(qd[v].y, p.y, acc[v].x);
      } else {
        acc[v] = cjfma(qd[v], p, acc[v]);
      }
    }
#pragma unroll
    for (int v = NF; v < NG; ++v) acc[ND + v] = cjfma(qd[v], qd[ND > 0 ? ND - 1 : 0], acc[ND + v]);
    if (NF > 0) {
      const float nx = head_float(qd[ND > 0 ? ND - 1 : 0].x), ny = head_float(qd[ND > 0 ? ND - 1 : 0].y);
#pragma unroll
      for (int v = 0; v < NF; ++v) {
        const float qx = head_float(qd[v].x), qy = head_float(qd[v].y);
        accf[v].x = fmaf(qx, nx, fmaf(qy, ny, accf[v].x));
        accf[v].y = fmaf(qx, ny, fmaf(-qy, nx, accf[v].y));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NF; ++v) acc[ND + v] = make_double2(wide_float(accf[v].x), wide_float(accf[v].y));
  // the CTA's sums over its warps, then to the accumulators: warp y takes sum
  // y / 2's real or imaginary part
  acc_t* out = acc_tile(o.a, o.a.out, it.x) + tx;
#pragma unroll
  for (int v0 = 0; v0 < (ND == 0 ? 1 : NS); v0 += NR) {
    if (v0 > 0) __syncthreads();
#pragma unroll
    for (int u = 0; u < NR; ++u)
      if (v0 + u < (ND == 0 ? 1 : NS)) red[u][ty][tx] = acc[v0 + u];
    if (ND == 0) mx[ty][tx] = top;
    __syncthreads();
    const int u = ty >> 1, im = ty & 1, v = v0 + u;
    if (act && u < NR && v < (ND == 0 ? 1 : NS) && !(im && (REAL || ND == 0))) {
      double s = im ? red[u][0][tx].y : red[u][0][tx].x;
#pragma unroll
      for (int y = 1; y < SPC_WARPS; ++y) s += im ? red[u][y][tx].y : red[u][y][tx].x;
      const int e = ND == 0 ? acc_norm_exp(T) : (v < ND ? acc_dot_exp(T) : ACC_GRAM_EXP);
      acc_add<ND == 0>(out + (4 * v + 2 * im) * SPC_LANES, out + ACC_BAD * SPC_LANES, s, e);
      if (ND == 0) {
#pragma unroll
        for (int y = 1; y < SPC_WARPS; ++y) top = max(top, mx[y][tx]);
        atomicMax(out + ACC_MAX * SPC_LANES, (acc_t)top);
      }
    }
  }
}

// After the norm pass: 1/||p||, the exponent bound of p/||p|| and, recorded by
// the tile's first CTA, the Hessenberg's subdiagonal, the next Lanczos
// coefficient, the exponent and the basis' maximum. Called by 32 lanes.
__device__ __forceinline__ double ortho_norm(const PassArgs& a, const AccArgs& A, const TileInfo& T, int tile, int lane,
                                             bool record, int* ex) {
  const int w = tile * SPC_LANES + lane;
  const acc_t* in = acc_tile(A, A.in, tile) + lane;
  double b = sqrt(acc_get_norm(in, acc_norm_exp(T)));
  if (in[ACC_BAD * SPC_LANES]) b = __longlong_as_double(0x7ff8000000000000ll);
  // exact breakdown (p == 0): the next basis vector is 0 instead of 0/0
  const double rb = b > 0.0 ? 1.0 / b : (b == 0.0 ? 0.0 : b);
  const unsigned top = (unsigned)in[ACC_MAX * SPC_LANES];
  const double q = top == 0u ? 0.0 : __hiloint2double((int)(top + 1u), 0) * rb;
  const unsigned hq = (unsigned)__double2hiint(q) & 0x7fffffffu;
  *ex = (int)(hq >> 20);
  if (record && a.map[w] >= 0) {
    const size_t mm = (size_t)a.m * a.m;
    const int i = a.col_i;
    a.Ahess[(size_t)w * mm + (i + 1) + (size_t)i * a.m] = make_double2(b, 0.0);
    if (a.lanczos) {
      // Hermitian tridiagonal: A(i, i+1) = beta_i, the coefficient of Q_i in
      // the next step's three-term recurrence
      a.Ahess[(size_t)w * mm + i + (size_t)(i + 1) * a.m] = make_double2(b, 0.0);
    }
    a.coef[w] = make_double2(b, 0.0);
    a.xexp[w] = *ex;
    a.qmax[w] = max(a.qmax[w], hq);
  }
  return rb;
}

typedef void (*OrthoFn)(OrthoArgs);
// The pass of a block: `nd` dots after subtracting nothing or a full block (nd
// = 8 on an older block; the newest block also forms its basis products), or
// the norm after the last block's `na` vectors.
template <bool HERM>
static OrthoFn ortho_fn(int na, int nd, bool newest) {
  static const OrthoFn old[2] = {k_ortho<0, 8, false, false>, k_ortho<8, 8, false, false>};
  static const OrthoFn lone[8] = {
      k_ortho<0, 1, true, false, HERM>, k_ortho<0, 2, true, false, HERM>, k_ortho<0, 3, true, false, HERM>,
      k_ortho<0, 4, true, false, HERM>, k_ortho<0, 5, true, false, HERM>, k_ortho<0, 6, true, false, HERM>,
      k_ortho<0, 7, true, false, HERM>, k_ortho<0, 8, true, false, HERM>};
  static const OrthoFn next[8] = {
      k_ortho<8, 1, true, false, HERM>, k_ortho<8, 2, true, false, HERM>, k_ortho<8, 3, true, false, HERM>,
      k_ortho<8, 4, true, false, HERM>, k_ortho<8, 5, true, false, HERM>, k_ortho<8, 6, true, false, HERM>,
      k_ortho<8, 7, true, false, HERM>, k_ortho<8, 8, true, false, HERM>};
  static const OrthoFn norm[8] = {k_ortho<1, 0, false, false>, k_ortho<2, 0, false, false>, k_ortho<3, 0, false, false>,
                                  k_ortho<4, 0, false, false>, k_ortho<5, 0, false, false>, k_ortho<6, 0, false, false>,
                                  k_ortho<7, 0, false, false>, k_ortho<8, 0, false, false>};
  if (nd == 0) return norm[na - 1];
  if (!newest) return old[na > 0];
  return na > 0 ? next[nd - 1] : lone[nd - 1];
}
