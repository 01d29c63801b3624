// SpMM of the general builder's Hamiltonians on the FP16 tensor cores, in
// exact digit arithmetic (spc_digits.cuh). Included by spc_propagate.cu
// inside namespace spc.
//
// For a nuclear index n the four rows (e, n) of H couple to the four rows of
// n itself and of the indices n' that differ in one nucleus by one step: 4 x 4
// complex blocks over the electron pair, 8 x 8 real ones. Y^T = X^T H^T is
// then a product with 16 samples on the M side, the 8 real outputs of n on the
// N side and two blocks (2 x 8 real inputs) per k-step. The off-diagonal blocks
// depend on (nucleus, state, direction) only and stay in L1 (1 KB each as
// fragments); the diagonal block is stored per n.
//
// H enters in units of 2^(eoff - 53), eoff the exponent of its largest
// off-diagonal component (raised where a diagonal component would pass eight
// digits), with digits k = 0..7 (k = 0 only in the diagonal blocks) in
// [-128, 127]; X in units of 2^(E - 61), E the exponent of the sample's largest
// component, with digits d = 0..7, the first in [-128, 127], the others plain
// bytes 0..255: a byte alone in an FP16 word is the subnormal byte * 2^-24, so
// one byte permute makes an operand. Products with k + d <= 8 are formed. A
// row has at most 4 real terms per neighbour and 8 for itself, so a level
// l <= 6 stays within 2^7 * 255 * (6 (4 nbr + 8) + 8) < 2^24 for up to
// BLK_MAXNBR neighbours and is exact; so are the last two but for sums that a
// rounding unit of 2^-57 of the result reaches only when nearly every digit of
// a row has its largest value and one sign.

static_assert(128 * 255 * (6 * (4 * BLK_MAXNBR + 8) + 8) < 1 << 24, "sums of digit products stay exact");
static_assert(BLK_MAXNBR + 1 <= 32, "a list has an entry for each lane at most");
#define BLK_THREADS 128
#define BLK_AHEAD 2  // k-steps copied ahead (and the least length of a list)
#define BLK_IDX (BLK_THREADS / 64)  // nuclear indices of a CTA at a time

// One system's blocks: host description and place in its store.
struct BlkDesc {
  int Z, nn, bk, eoff;           // nuclear rows, nuclei, list length per n (even), unit exponent
  int nuc0, tab0;                // first nucleus, unused table entry 0 (zero block)
  const int* rowptr;
  const int* col;
  const double2* val;
  uint4* self;                   // Z x 64: digits 0-3 of the 32 lanes, then 4-7
  uint4* tab;                    // ntab x 64
  int2* nbr;                     // Z x bk: (index, table entry); entry 0: (n, k-steps)
};
struct BlkNuc {
  int g, tab;                    // multiplicity, first table entry: tab + 2 m + (1 for m + 1)
  int64_t stride;
};

// Digits 0..7 of h in units of 2^(eoff - 53) for the B fragment of the block
// rows (e, part) = lane / 4, inputs e' = lane % 4: (h_r, -h_i) or (h_i, h_r).
__device__ __forceinline__ void blk_words(double2 h, int part, int eoff, uint4* dst) {
  const double a = part ? h.y : h.x, b = part ? h.x : -h.y;
  const unsigned long long ua = (unsigned long long)__double2ll_rn(scalbn(a, 53 - eoff)) + DIGIT_BIAS;
  const unsigned long long ub = (unsigned long long)__double2ll_rn(scalbn(b, 53 - eoff)) + DIGIT_BIAS;
  unsigned w[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    w[k] = k < 4 ? digit_pair((unsigned)(ua >> 32), (unsigned)(ub >> 32), 3 - k)
                 : digit_pair((unsigned)ua, (unsigned)ub, 7 - k);
  dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
  dst[32] = make_uint4(w[4], w[5], w[6], w[7]);
}
// H[row, c] of a row of the execution copy (0 where not stored)
__device__ __forceinline__ double2 blk_entry(const BlkDesc& D, int64_t row, int c) {
  double2 h = cz();
  for (int k = D.rowptr[row]; k < D.rowptr[row + 1]; ++k)
    if (D.col[k] == c) h = cadd(h, D.val[k]);
  return h;
}
// Diagonal blocks: one warp per nuclear index; grid (x, systems).
__global__ void __launch_bounds__(256) k_blk_self(const BlkDesc* __restrict__ descs) {
  const BlkDesc D = descs[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int n = blockIdx.x * 8 + (threadIdx.x >> 5); n < D.Z; n += gridDim.x * 8) {
    const int e = lane >> 3, part = (lane >> 2) & 1, q = lane & 3;
    blk_words(blk_entry(D, (int64_t)e * D.Z + n, q * D.Z + n), part, D.eoff, D.self + (size_t)n * 64 + lane);
  }
}
// Neighbour lists (one thread per nuclear index) and, by the first CTA of
// each system, the table of off-diagonal blocks.
__global__ void __launch_bounds__(256) k_blk_lists(const BlkDesc* __restrict__ descs, const BlkNuc* __restrict__ nucs) {
  const BlkDesc D = descs[blockIdx.y];
  const BlkNuc* nuc = nucs + D.nuc0;
  for (int n = blockIdx.x * 256 + threadIdx.x; n < D.Z; n += gridDim.x * 256) {
    int2* L = D.nbr + (size_t)n * D.bk;
    int c = 1;
    for (int j = D.nn - 1; j >= 0; --j) {
      const int m = (int)((n / nuc[j].stride) % nuc[j].g);
      if (m > 0) L[c++] = make_int2((int)(n - nuc[j].stride), nuc[j].tab + 2 * m);
      if (m < nuc[j].g - 1) L[c++] = make_int2((int)(n + nuc[j].stride), nuc[j].tab + 2 * m + 1);
    }
    while (c < 2 * BLK_AHEAD - 1) L[c++] = make_int2(n, 0);  // zero blocks: k_spmm_blk's lists have its depth
    if (c & 1) L[c++] = make_int2(n, 0);
    L[0] = make_int2(n, c / 2);
  }
  if (blockIdx.x != 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    D.tab[lane] = make_uint4(0, 0, 0, 0);
    D.tab[lane + 32] = make_uint4(0, 0, 0, 0);
  }
  const int e = lane >> 3, part = (lane >> 2) & 1, q = lane & 3;
  for (int j = 0; j < D.nn; ++j)
    for (int t = warp; t < 2 * nuc[j].g; t += 8) {
      const int m = t >> 1, mp = (t & 1) ? m + 1 : m - 1;
      const bool in = mp >= 0 && mp < nuc[j].g;
      const int64_t n = m * nuc[j].stride, np = mp * nuc[j].stride;
      const double2 h = in ? blk_entry(D, (int64_t)e * D.Z + n, (int)((int64_t)q * D.Z + np)) : cz();
      blk_words(h, part, D.eoff, D.tab + (size_t)(nuc[j].tab + t) * 64 + lane);
    }
}

// The eight digits of both parts as bytes (the first + 128): word w holds
// (re_2w, im_2w, re_2w+1, im_2w+1).
__device__ __forceinline__ uint4 pack_digits(double2 x, int emax) {
  const unsigned long long r = (unsigned long long)to_fixed<9>(x.x, emax) ^ (1ull << 63);
  const unsigned long long i = (unsigned long long)to_fixed<9>(x.y, emax) ^ (1ull << 63);
  const unsigned rh = (unsigned)(r >> 32), rl = (unsigned)r, ih = (unsigned)(i >> 32), il = (unsigned)i;
  return make_uint4(__byte_perm(rh, ih, 0x6273), __byte_perm(rh, ih, 0x4051), __byte_perm(rl, il, 0x6273),
                    __byte_perm(rl, il, 0x4051));
}
// FP16 pair of digit d, times 2^-24, from the packed digits
__device__ __forceinline__ unsigned unpack_digit(uint4 v, int d) {
  const unsigned word = d < 2 ? v.x : (d < 4 ? v.y : (d < 6 ? v.z : v.w));
  if (d > 0) return __byte_perm(word, 0u, (d & 1) ? 0x4342 : 0x4140);
  const unsigned h = __byte_perm(word, 0x64646464u, 0x4140);  // 1024 + byte
  const __half2 f = __hfma2(*reinterpret_cast<const __half2*>(&h), __half2half2(__ushort_as_half(0x0001)),
                            __half2half2(__ushort_as_half(0x8480)));  // * 2^-24 - 1152 * 2^-24
  return *reinterpret_cast<const unsigned*>(&f);
}

// hi 2^32 + lo as a double, one rounding: the top 62 bits converted once, the
// exponent added as an integer (an FP64 instruction holds a scheduler's pipe
// for 64 clocks, an integer one for 2).
__device__ __forceinline__ double close_sum(long long hi, long long lo) {
  const long long t = hi + (lo >> 32);
  const int s = max(0, 34 - __clzll(t ^ (t >> 63)));  // bits of t beyond 30
  const double d = (double)((t << (32 - s)) | (long long)((unsigned)lo >> s));
  return __hiloint2double(__double2hiint(d) + (s << 20), __double2loint(d));  // s > 0 only where d is large
}
// d * 2^e in integers: 0 below the normal range; e >= DIGIT_NAN gives NaN
#define DIGIT_NAN 8192
__device__ __forceinline__ double times_pow2(double d, int e) {
  const int h = __double2hiint(d), ex = (h >> 20) & 0x7ff, f = ex + e;
  const int lo = __double2loint(d);
  if (f >= 0x7ff) return ex == 0 && e < DIGIT_NAN ? 0.0 : __hiloint2double(e >= DIGIT_NAN ? 0x7ff80000 : 0x7ff00000, 0);
  return ex == 0 || f <= 0 ? 0.0 : __hiloint2double(h + (e << 20), lo);
}
// 16 bytes from global to this thread's shared memory, asynchronously; L1 holds
// the source line only with KEEP.
template <bool KEEP>
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (KEEP)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// P_t = H Q_t[i] for the tiles' items: one warp per (nuclear index, 16
// samples), a CTA takes BLK_IDX consecutive indices at a time. DX holds the
// current vector's packed digits, the four electron rows of an index together:
// [n][32 samples][4]. A lane's operand is then row q = lane % 4 of sample
// lane / 4 and the next: a quarter warp reads 128 consecutive bytes. The
// results change lanes before they are stored, so that eight lanes hold eight
// samples of one row.
// Every operand is first copied to the shared memory of the lane that uses it,
// BLK_AHEAD k-steps ahead and across the end of an index (lane t holds entry t
// of the current and the next index' list): read where they are used, a
// step's list entry and rows cost two L2 latencies that five warps per
// scheduler do not cover.
// LZ false (MGS rounds): a Hermitian-part copy gets -i kappa x added, as
// k_spmm. LZ true: the kernel also does the first projection of the same Lanczos
// step (k_ortho<1, 1, false, true>) on the rows it holds, P = H Q_i - beta_{i-1}
// Q_{i-1} and the sum alpha_i = Re <Q_i, P>.
//
// Measured: dim 55296, 512 samples, 1.62 ms with the Lanczos projection against
// 4.60 ms for k_spmm and 0.27 ms for the pass; dim 9216, 64 samples, MGS: 36
// against 91 us; dim 2304, 77 samples: 28 against 44 + 14 us. The tensor pipe
// is busy 52 % of the time (its floor is 0.85 ms at dim 55296): 1.7 k
// instructions per warp and index, 270 of them products, issue every 2.4
// clocks with the four warps per scheduler that 128 registers leave. Five or
// six warps at fewer registers, or rows copied three steps ahead, measure the
// same within 3 %.
template <bool LZ>
__global__ void __launch_bounds__(BLK_THREADS, 4)
    k_spmm_blk(PassArgs a, AccArgs A, const int2* __restrict__ items, const uint4* __restrict__ DX) {
  __shared__ uint4 s_x[BLK_AHEAD + 1][4][BLK_THREADS];
  __shared__ double2 s_q[LZ ? 4 : 2][BLK_THREADS];
  __shared__ int s_exp[SPC_LANES];
  __shared__ double s_beta[SPC_LANES], s_dot[2][BLK_THREADS];
  const int i = a.col_i;
  const int2 it = items[blockIdx.x];
  const TileInfo& T = a.tiles[it.x];
  if (i >= T.m) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int Z = T.n / 4;
  const int s0 = 16 * (warp & 1);
  const int per = ((Z + BLK_IDX - 1) / BLK_IDX + T.nib - 1) / T.nib;
  const int nend = min(Z, (it.y + 1) * per * BLK_IDX);
  const int* map = a.map + it.x * SPC_LANES;
  if (warp == 0) {
    const int w = it.x * SPC_LANES + lane;
    const int ex = a.xexp[w];
    s_exp[lane] = ex >= 0x7ff ? DIGIT_NAN : ex - 1023 + T.bexp;
    s_beta[lane] = LZ && i > 0 ? a.coef[w].x : 0.0;
  }
  s_dot[0][tid] = s_dot[1][tid] = 0.0;
  if (LZ && it.y == 0) acc_clear(A, it.x, tid, BLK_THREADS);
  __syncthreads();
  const uint4* X = DX + T.p_off + (s0 + g) * 4 + q;
  const uint4* bself = T.bself + lane;
  const uint4* btab = T.btab + lane;
  const bool shift = !LZ && a.shift && T.kappa != nullptr;
  // store side: this lane's row re and samples s0 + gs, + 8
  const int re = lane >> 3, gs = lane & 7;
  const size_t row0 = (size_t)re * Z * SPC_LANES + s0 + gs;
  const double2* Qi = a.Q + T.q_off + (size_t)i * T.n * SPC_LANES + row0;
  const int bk = T.bk;
  const int2* lists = T.bnbr + min(lane, bk - 1);
  int n = it.y * per * BLK_IDX + (warp >> 1);
  int2 cur = make_int2(0, 0), nxt = make_int2(0, 0);
  if (n < nend) cur = lists[(size_t)n * bk];
  if (n + BLK_IDX < nend) nxt = lists[(size_t)(n + BLK_IDX) * bk];
  // copies run BLK_AHEAD steps before the products: `at` is the next step to
  // copy, of the current index' list or (ahead) of the next one's
  int at = 0, slot_in = 0, slot_out = 0;
  bool ahead = false;
  auto copy_step = [&]() {
    const int total = __shfl_sync(0xffffffffu, ahead ? nxt.y : cur.y, 0);
    if (at >= total && !ahead) {
      ahead = true;
      at = 0;
    }
    const int from = ahead ? nxt.x : cur.x;
    const int have = __shfl_sync(0xffffffffu, ahead ? nxt.y : cur.y, 0);
    const int r0 = __shfl_sync(0xffffffffu, from, 2 * at), r1 = __shfl_sync(0xffffffffu, from, 2 * at + 1);
    if (at < have) {
      const uint4* xa = X + (size_t)r0 * 128;
      const uint4* xb = X + (size_t)r1 * 128;
      copy16<true>(&s_x[slot_in][0][tid], xa);
      copy16<true>(&s_x[slot_in][1][tid], xa + 32);
      copy16<true>(&s_x[slot_in][2][tid], xb);
      copy16<true>(&s_x[slot_in][3][tid], xb + 32);
      ++at;
      slot_in = slot_in == BLK_AHEAD ? 0 : slot_in + 1;
    }
  };
#pragma unroll
  for (int s = 0; s < BLK_AHEAD; ++s) {
    copy_step();
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (; n < nend; n += BLK_IDX) {
    const size_t o = (size_t)n * SPC_LANES;
    const int steps = __shfl_sync(0xffffffffu, cur.y, 0);
    if (LZ || shift) {  // the rows of this index for the end of it
      copy16<false>(&s_q[0][tid], Qi + o);
      copy16<false>(&s_q[1][tid], Qi + o + 8);
      if (LZ && i > 0) {
        copy16<false>(&s_q[LZ ? 2 : 0][tid], Qi + o - (size_t)T.n * SPC_LANES);
        copy16<false>(&s_q[LZ ? 3 : 0][tid], Qi + o - (size_t)T.n * SPC_LANES + 8);
      }
    }
    float acc[9][4];
#pragma unroll
    for (int l = 0; l < 9; ++l)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[l][r] = 0.f;
    // one k-step with the blocks at b0p and b1p
    auto step = [&](const uint4* b0p, const uint4* b1p, auto diag) {
      const uint4 p0 = b0p[0], p1 = b0p[32], p2 = b1p[0], p3 = b1p[32];
      copy_step();
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group %0;" ::"n"(BLK_AHEAD) : "memory");
      const uint4 x0 = s_x[slot_out][0][tid], x1 = s_x[slot_out][1][tid], x2 = s_x[slot_out][2][tid],
                  x3 = s_x[slot_out][3][tid];
      slot_out = slot_out == BLK_AHEAD ? 0 : slot_out + 1;
      const unsigned b0[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
      const unsigned b1[8] = {p2.x, p2.y, p2.z, p2.w, p3.x, p3.y, p3.z, p3.w};
#pragma unroll
      for (int d = 0; d < DIGITS; ++d) {
        const unsigned A[4] = {unpack_digit(x0, d), unpack_digit(x1, d), unpack_digit(x2, d), unpack_digit(x3, d)};
#pragma unroll
        for (int k = decltype(diag)::value ? 0 : 1; k < 8 && k + d < 9; ++k) mma_digits(acc[k + d], A, b0[k], b1[k]);
      }
    };
    step(bself + (size_t)n * 64, btab + (size_t)__shfl_sync(0xffffffffu, cur.y, 1) * 64, std::true_type());
    for (int s = 1; s < steps; ++s)
      step(btab + (size_t)__shfl_sync(0xffffffffu, cur.y, 2 * s) * 64,
           btab + (size_t)__shfl_sync(0xffffffffu, cur.y, 2 * s + 1) * 64, std::false_type());
    // the next index becomes the current one
    cur = nxt;
    if (n + 2 * BLK_IDX < nend)
      nxt = lists[(size_t)(n + 2 * BLK_IDX) * bk];
    else
      nxt = make_int2(0, 0);
    ahead = false;  // every list is at least BLK_AHEAD steps long: the copies are in this index by now
    double y[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int v[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = __float2int_rn(acc[k][r] * 16777216.f);
      const long long hi = (long long)v[4] + (long long)v[3] * 256 + (long long)v[2] * 65536 + (long long)v[1] * 16777216 +
                           ((long long)v[0] << 32);
      const long long lo = (long long)v[8] + (long long)v[7] * 256 + (long long)v[6] * 65536 + (long long)v[5] * 16777216;
      y[r] = close_sum(hi, lo);
    }
    // (sample g, row q) moves to lane 8 q + g
    const int from = gs * 4 + re;
#pragma unroll
    for (int r = 0; r < 4; ++r) y[r] = __shfl_sync(0xffffffffu, y[r], from);
    if ((LZ || shift) && steps < BLK_AHEAD + 1) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = s0 + gs + 8 * h;
      if (map[c] < 0) continue;
      const int u = s_exp[c];
      double2 yv = make_double2(times_pow2(y[2 * h], u), times_pow2(y[2 * h + 1], u));
      if (LZ) {
        if (i > 0) {
          const double b = s_beta[c];
          const double2 q0 = s_q[LZ ? 2 + h : 0][tid];
          yv.x = fma(-b, q0.x, yv.x);
          yv.y = fma(-b, q0.y, yv.y);
        }
        const double2 x = s_q[h][tid];
        s_dot[h][tid] = fma(x.y, yv.y, fma(x.x, yv.x, s_dot[h][tid]));
      } else if (shift) {
        const double kp = *T.kappa;
        const double2 xr = s_q[h][tid];
        yv.x = fma(kp, xr.y, yv.x);
        yv.y = fma(-kp, xr.x, yv.y);
      }
      a.P[T.p_off + row0 + o + 8 * h] = yv;
    }
  }
  if (!LZ) return;
  // the CTA's sum of sample c = 16 half + 8 h + gs: the four rows and the warps
  // of its half
  __syncthreads();
  if (warp == 0 && map[lane] >= 0) {
    double s = 0.0;
#pragma unroll
    for (int v = 0; v < BLK_IDX; ++v)
#pragma unroll
      for (int r = 0; r < 4; ++r) s += s_dot[(lane >> 3) & 1][(2 * v + (lane >> 4)) * 32 + 8 * r + (lane & 7)];
    acc_t* out = acc_tile(A, A.out, it.x) + lane;
    acc_add(out, out + ACC_BAD * SPC_LANES, s, acc_dot_exp(T));
  }
}

// Bytes of a store's buffers (self, tab, nbr, desc) with the fragments of the systems in
// `use`: 1 KB a nuclear index and a table entry.
struct BlockSizes {
  size_t self = 0, tab = 0, nbr = 0, desc = 0;
};
static BlockSizes block_sizes(const Handle::BlockStore& S, const std::vector<char>& use) {
  BlockSizes z;
  size_t nuc = 1, systems = 0;
  for (size_t k = 0; k < S.sys.size(); ++k) {
    if (!use[k]) continue;
    const BlockSys& b = S.sys[k];
    int64_t entries = 1;
    for (int g : b.g) entries += 2 * g;
    z.self += 1024 * (size_t)b.Z;
    z.tab += 1024 * (size_t)entries;
    z.nbr += sizeof(int2) * (size_t)(b.Z * b.bk);
    nuc += b.g.size();
    ++systems;
  }
  z.desc = sizeof(BlkDesc) * systems + sizeof(BlkNuc) * nuc;
  return z;
}
// What the store's buffers come to once they hold `use` (buffers only grow).
static size_t block_bytes_after(const Handle::BlockStore& S, const std::vector<char>& use) {
  if (S.has(use)) return S.bytes();
  const BlockSizes z = block_sizes(S, use);
  return std::max(S.self.bytes, z.self) + std::max(S.tab.bytes, z.tab) + std::max(S.nbr.bytes, z.nbr) +
         std::max(S.desc.bytes, z.desc);
}

// Fragments of the systems in `use`, built by the first propagation that runs on
// them, two launches in all. Holds nothing where it fails.
static int prepare_blocks(Handle* h, Handle::BlockStore& S, const std::vector<char>& use,
                          const std::vector<const int*>& rowptr, const std::vector<const int*>& col,
                          const std::vector<const double2*>& val) {
  // a call that failed after building returned without waiting for its stream
  if (S.stream != h->stream && S.built && cudaStreamWaitEvent(h->stream, S.built, 0) != cudaSuccess)
    return set_error(SPC_ERR_CUDA, "waiting for the blocks failed: %s", cudaGetErrorString(cudaGetLastError()));
  if (S.has(use)) return SPC_OK;
  const BlockSizes z = block_sizes(S, use);
  if (h->ensure(S.self, z.self) || h->ensure(S.tab, z.tab) || h->ensure(S.nbr, z.nbr) || h->ensure(S.desc, z.desc)) {
    S.release();
    return SPC_ERR_ALLOC;
  }
  std::vector<BlkDesc> d;
  std::vector<BlkNuc> nu;
  int64_t selfs = 0, tabs = 0, nbrs = 0;
  int zmax = 1;
  for (size_t k = 0; k < S.sys.size(); ++k) {
    if (!use[k]) continue;
    BlockSys& b = S.sys[k];
    b.self_off = selfs;
    b.tab_off = tabs;
    b.nbr_off = nbrs;
    BlkDesc x{};
    x.Z = (int)b.Z;
    x.nn = (int)b.g.size();
    x.bk = b.bk;
    x.eoff = b.eoff;
    x.nuc0 = (int)nu.size();
    x.rowptr = rowptr[k];
    x.col = col[k];
    x.val = val[k];
    x.self = (uint4*)S.self.p + 64 * selfs;
    x.tab = (uint4*)S.tab.p + 64 * tabs;
    x.nbr = (int2*)S.nbr.p + nbrs;
    int t = 1;
    for (size_t j = 0; j < b.g.size(); ++j) {
      nu.push_back(BlkNuc{b.g[j], t, b.stride[j]});
      t += 2 * b.g[j];
    }
    d.push_back(x);
    selfs += b.Z;
    tabs += t;
    nbrs += b.Z * b.bk;
    zmax = std::max(zmax, (int)b.Z);
  }
  S.placed.assign(S.sys.size(), 0);
  const size_t nb = sizeof(BlkDesc) * d.size();
  cudaError_t e = cudaMemcpyAsync(S.desc.p, d.data(), nb, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess && !nu.empty())
    e = cudaMemcpyAsync((char*)S.desc.p + nb, nu.data(), sizeof(BlkNuc) * nu.size(), cudaMemcpyHostToDevice, h->stream);
  const int gx = std::max(1, std::min((zmax + 7) / 8, h->sm_count * 8));
  for (size_t y0 = 0; e == cudaSuccess && y0 < d.size(); y0 += 65535) {
    const int ny = (int)std::min<size_t>(65535, d.size() - y0);
    k_blk_self<<<dim3(gx, ny), 256, 0, h->stream>>>((const BlkDesc*)S.desc.p + y0);
    k_blk_lists<<<dim3((gx + 31) / 32, ny), 256, 0, h->stream>>>((const BlkDesc*)S.desc.p + y0,
                                                                 (const BlkNuc*)((char*)S.desc.p + nb));
    h->count_launch(2);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && !S.built) e = cudaEventCreateWithFlags(&S.built, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventRecord(S.built, h->stream);
  S.stream = h->stream;
  if (e != cudaSuccess)
    return set_error(SPC_ERR_CUDA, "block fragments of the Hamiltonian failed: %s", cudaGetErrorString(e));
  S.placed = use;
  return SPC_OK;
}
