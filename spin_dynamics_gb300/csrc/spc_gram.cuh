// Projector Grams on the FP16 tensor cores in exact digit arithmetic
// (spc_digits.cuh). Included by spc_propagate.cu inside namespace spc.

__device__ __forceinline__ unsigned twice(unsigned x) {
  const __half2 h = *reinterpret_cast<const __half2*>(&x);
  const __half2 v = __hadd2(h, h);
  return *reinterpret_cast<const unsigned*>(&v);
}

// The Krylov-space projectors (k_proj's Grams, same `part` layout) for m <= 32.
// k_gram: CTA = (sample, type, split of the nuclear rows). Staged per chunk of GRAM_R
// rows: the type's vectors V (q1, q2 - q3, q2 + q3 or q4, formed exactly in
// integers) as digit pairs (re, im), 32 bits each, [digit][vector][row]. With
// k = (row, part) both operands of V^H V are the same words: the A fragment
// of 16 vectors is the B fragments of its two 8-column halves; the imaginary
// part takes B = (im, -re).
// A warp holds one 16 x 16 block of the real or imaginary part (MT = 2: 8
// blocks; MT = 1: 2 blocks, four warps each over every fourth k-step). Digit
// pairs (i, j) and (j, i) give transposed blocks, so only i <= j is formed,
// with A_i doubled for i < j: T = sum_(i<j) 2 A_i B_j + sum_i A_i B_i, 20
// products instead of 36 (i + j <= 7), and G = (T + T^T) / 2 (Re),
// (T - T^T) / 2 (Im). A k-step adds at most 8 * 16 * 2^14 = 2^21 to a level:
// after 8 steps the FP32 sums are closed into 64-bit integers in shared memory.
// V is in units of 2^(E - 60), E the exponent of the basis' largest component.
// Row stride GRAM_R + 4 words (36, or 20 with 16 rows): the 8 vectors x 4 rows
// of a fragment load fall into 32 different banks.
// The next chunk's components are copied to shared memory while a chunk's
// products run: without that a warp waited on global loads in 2.8 of 8.4 clocks.
// Measured, all four Grams of 512 samples at dim 55296, m = 30: 18.7 ms (21.6
// without the copies) against 71.4 ms for k_proj (which holds the FP64 pipe at
// 92 %); 64 samples at dim 9216, m = 24: 0.40 (0.45) against 1.17 ms; 384
// samples at dim 2304, m = 16: 0.23 (0.28) against 0.59 ms. The products take a
// third of the time, the loads (one 32-byte sector a component, the type's
// vectors read once more for S and T0) and their conversion to digits the rest.
#define GRAM_R 32
__host__ __device__ __forceinline__ size_t gram_smem_bytes(int mt, int rows = GRAM_R) {
  return sizeof(unsigned) * DIGITS * 16 * mt * (rows + 4) + sizeof(longlong2) * 8 * 256;
}
// Sums of one type over the rows [n0, n1): T of every block, in units of the
// digit products, to Tm ([2][MP][MP + 1] doubles in V's place). get(j, row, e) is
// the address of the component of basis vector j < me at nuclear row `row`,
// electron state e. AHEAD: the next chunk's components are copied to raw while
// the products run (a thread copies what it converts). The CTA's 256 threads;
// ends with a barrier.
template <int MT, int R, bool AHEAD, typename Get>
__device__ __forceinline__ void gram_sums(int type, int m, int me, int emax, int64_t n0, int64_t n1, longlong2* acc64,
                                          unsigned* V, double2* raw, Get get) {
  constexpr int MP = 16 * MT, LD = R + 4;
  const int tid = threadIdx.y * 32 + threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  // this warp's block: part (0 Re, 1 Im), rows 16 mi, columns 16 ni, k-steps
  const int im = warp & 1;
  const int mi = MT == 2 ? (warp >> 1) & 1 : 0, ni = MT == 2 ? warp >> 2 : 0;
  const int k0 = MT == 2 ? 0 : warp >> 1, kstep = MT == 2 ? 1 : 4;
  const bool two = 16 * ni + 8 < m;  // the second 8 columns hold basis vectors
  float acc[2][DIGITS][4];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int l = 0; l < DIGITS; ++l)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[t][l][r] = 0.f;
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (r < 4 || two) acc64[r * 256 + tid] = make_longlong2(0, 0);
  auto close = [&]() {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (t > 0 && !two) break;
        long long s[DIGITS];
#pragma unroll
        for (int l = 0; l < DIGITS; ++l) {
          s[l] = __float2int_rn(acc[t][l][r]);
          acc[t][l][r] = 0.f;
        }
        longlong2 a = acc64[(4 * t + r) * 256 + tid];
        a.x += (s[0] << 24) + (s[1] << 16) + (s[2] << 8) + s[3];
        a.y += (s[4] << 24) + (s[5] << 16) + (s[6] << 8) + s[7];
        acc64[(4 * t + r) * 256 + tid] = a;
      }
  };
  const int e0 = type == 0 ? 0 : (type == 3 ? 3 : 1);
  const bool sum2 = type == 1 || type == 2;
  auto copy = [&](int64_t c0) {
    const int len = (int)min((int64_t)R, n1 - c0);
#pragma unroll 4
    for (int idx = tid; idx < MP * R; idx += 256) {
      const int j = idx / R, nn = idx % R;
      if (j < me && nn < len) {
        copy16<false>(raw + idx, get(j, c0 + nn, e0));
        if (sum2) copy16<false>(raw + MP * R + idx, get(j, c0 + nn, 2));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (AHEAD && n0 < n1) copy(n0);
  int steps = 0;
  for (int64_t c0 = n0; c0 < n1; c0 += R) {
    const int len = (int)min((int64_t)R, n1 - c0);
    if (AHEAD) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll 4
    for (int idx = tid; idx < MP * R; idx += 256) {
      const int j = idx / R, nn = idx % R;
      long long vr = 0, vi = 0;
      if (j < me && nn < len) {
        const double2 a = AHEAD ? raw[idx] : *get(j, c0 + nn, e0);
        vr = to_fixed<8>(a.x, emax);
        vi = to_fixed<8>(a.y, emax);
        if (sum2) {
          const double2 b = AHEAD ? raw[MP * R + idx] : *get(j, c0 + nn, 2);
          const long long br = to_fixed<8>(b.x, emax), bi = to_fixed<8>(b.y, emax);
          vr = type == 1 ? vr - br : vr + br;
          vi = type == 1 ? vi - bi : vi + bi;
        }
      }
      const unsigned long long ur = (unsigned long long)vr + DIGIT_BIAS, ui = (unsigned long long)vi + DIGIT_BIAS;
      const unsigned rl = (unsigned)ur, rh = (unsigned)(ur >> 32), il = (unsigned)ui, ih = (unsigned)(ui >> 32);
      unsigned* dst = V + j * LD + nn;
#pragma unroll
      for (int d = 0; d < DIGITS; ++d)
        dst[d * MP * LD] = d < 4 ? digit_pair(rh, ih, 3 - d) : digit_pair(rl, il, 7 - d);
    }
    if (AHEAD && c0 + R < n1) copy(c0 + R);
    __syncthreads();
    for (int ks = k0; ks * 8 < len; ks += kstep) {
      const unsigned* Vk = V + ks * 8 + q;
      unsigned B[2][DIGITS][2];
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (t == 0 || two)
#pragma unroll
          for (int d = 0; d < DIGITS; ++d)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const unsigned x = Vk[(d * MP + 16 * ni + 8 * t + g) * LD + 4 * h];
              B[t][d][h] = im ? __byte_perm(x, x, 0x1032) ^ 0x80000000u : x;
            }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        unsigned A[4];
        const unsigned* Va = Vk + (i * MP + 16 * mi + g) * LD;
        A[0] = Va[0];
        A[1] = Va[8 * LD];
        A[2] = Va[4];
        A[3] = Va[8 * LD + 4];
        mma_digits(acc[0][2 * i], A, B[0][i][0], B[0][i][1]);
        if (two) mma_digits(acc[1][2 * i], A, B[1][i][0], B[1][i][1]);
#pragma unroll
        for (int r = 0; r < 4; ++r) A[r] = twice(A[r]);
#pragma unroll
        for (int j = i + 1; j <= 7 - i; ++j) {
          mma_digits(acc[0][i + j], A, B[0][j][0], B[0][j][1]);
          if (two) mma_digits(acc[1][i + j], A, B[1][j][0], B[1][j][1]);
        }
      }
      if (++steps == 8) {
        close();
        steps = 0;
      }
    }
    __syncthreads();
  }
  close();
  __syncthreads();
  double* Tm = reinterpret_cast<double*>(V);
  constexpr int TL = MP + 1;
  if (MT == 2 || k0 == 0) {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (t > 0 && !two) break;
        longlong2 a = acc64[(4 * t + r) * 256 + tid];
        if (MT == 1)
          for (int o = 1; o < 4; ++o) {
            const longlong2 b = acc64[(4 * t + r) * 256 + tid + 64 * o];
            a.x += b.x;
            a.y += b.y;
          }
        const int row = 16 * mi + g + (r >> 1) * 8, colm = 16 * ni + 8 * t + 2 * q + (r & 1);
        Tm[(im * MP + row) * TL + colm] = fma((double)a.x, 4294967296.0, (double)a.y);
      }
  }
  __syncthreads();
}
// G_ij, i <= j, from the sums; unit: V in 2^(E - 60), products closed at 256^7,
// T twice the Gram. `bad` (an infinite or undefined basis) gives NaN.
__device__ __forceinline__ double gram_unit(unsigned top) {
  return top >= 0x7ff00000u ? __longlong_as_double(0x7ff8000000000000ll)
                            : ldexp(1.0, 2 * ((int)(top >> 20) - 1023) - 120 + 56 - 1);
}
template <int MT>
__device__ __forceinline__ double2 gram_entry(const double* Tm, int i, int j, double unit) {
  constexpr int MP = 16 * MT, TL = MP + 1;
  return make_double2((Tm[i * TL + j] + Tm[j * TL + i]) * unit,
                      (Tm[(MP + i) * TL + j] - Tm[(MP + j) * TL + i]) * unit);
}

__host__ __device__ __forceinline__ size_t gram_raw_bytes(int mt) { return sizeof(double2) * 2 * 16 * mt * GRAM_R; }
template <int MT>
__global__ void __launch_bounds__(256, 2)
    k_gram(const TileInfo* __restrict__ tiles, const int* __restrict__ slots, int m, int ncombo,
           const double2* __restrict__ Q, const unsigned* __restrict__ qmax, int nsplit, int64_t rps,
           double2* __restrict__ part, int nslots) {
  constexpr int MP = 16 * MT;
  extern __shared__ __align__(16) unsigned char gsm[];
  longlong2* acc64 = reinterpret_cast<longlong2*>(gsm);               // [8][256]
  unsigned* V = reinterpret_cast<unsigned*>(acc64 + 8 * 256);         // [DIGITS][MP][GRAM_R + 4]
  const int type = blockIdx.x & 3;
  const int w = slots ? slots[blockIdx.x >> 2] : blockIdx.x >> 2;  // null: every slot has a sample
  const TileInfo& Ti = tiles[w / SPC_LANES];
  const int64_t Z = Ti.n / 4;
  const int nsp = proj_splits(nsplit, rps, Z);
  const int split = blockIdx.y;
  if (split >= nsp) return;
  const int64_t per = (Z + nsp - 1) / nsp;
  const int64_t n0 = (int64_t)split * per, n1 = min(Z, n0 + per);
  const unsigned top = qmax[w];
  const size_t vs = (size_t)Ti.n * SPC_LANES;
  const double2* Qt = Q + Ti.q_off + (w % SPC_LANES);
  double2* raw = reinterpret_cast<double2*>(gsm + gram_smem_bytes(MT));
  gram_sums<MT, GRAM_R, true>(type, m, Ti.m, (int)(top >> 20), n0, n1, acc64, V, raw, [&](int j, int64_t row, int e) {
    return &Qt[(size_t)j * vs + (size_t)(e * Z + row) * SPC_LANES];
  });
  const double* Tm = reinterpret_cast<const double*>(V);
  const double unit = gram_unit(top);
  const int nc = ncombo / 4;
  double2* out = part + ((size_t)split * nslots + w) * ncombo + type * nc;
  for (int idx = threadIdx.x; idx < MP * MP; idx += 256) {
    const int i = idx / MP, j = idx % MP;
    if (i <= j && j < m) out[i * m - i * (i - 1) / 2 + (j - i)] = gram_entry<MT>(Tm, i, j, unit);
  }
}
