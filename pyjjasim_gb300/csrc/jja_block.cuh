// Products of dense FP64 blocks with many right-hand sides on the tensor cores (included by jja_gb300.cu).
//
// out[R_u, :] += B_u in[C_u, :] for a list of blocks B_u of at most 128 x 64 entries, by the digit
// products of jja_sine.cuh with the roles exchanged: the block's 6 digits are the MMA's M side (128
// rows), the data's 7 digits lie side by side on its N side (up to 64 problems), so one MMA forms the
// products of a block digit with up to four data digits, into adjacent accumulators.
//
// Face solves of circuits that no fast transform fits are a few such launches instead of the 14-28
// dependent ones of two triangular sweeps (jja_plan_set_blocks):
//   small circuits: x = K^-1 b, one launch with the whole inverse;
//   larger ones: the elimination tree is cut into subtrees ("leaves", l) of a few hundred faces and
//   the separator faces above them (s). With G_l = K_ll^-1 K_ls and S the separators' Schur complement
//     launch 1: b_s -= G_l^T b_l  and  x_l = K_ll^-1 b_l      (all leaves)
//     launch 2: x_s = S^-1 b_s
//     launch 3: x_l -= G_l x_s.
// The blocks come from the plan's own factor by sweeps over parts of its tree with columns of the
// identity (jja_plan_set_blocks). Each row of a block has its own scale.
//
// The products of the blocks side by side are added atomically, in any order: runs repeat to rounding, not bit for
// bit, as with the sweeps' split dot products.
//
// Measured (GB300, us per step with the sweeps -> with these products): honeycomb 24x24 x 61 problems
// 99 -> 24, triangular 64x48 with spread resistances x 96 240 -> 134, one such array 89 -> 33. A unit
// (128 x 64 block, 64 problems) takes about 12k cycles on its SM: 1.5k reading and splitting the data,
// 3.5k the products (the multipliers' rate), 7k joining the digits and adding to the result, while
// the next block's 96 KB arrive. The joining (the ALU pipe) bounds launches of many units, the
// latency of one unit and the launch those of few.

namespace {

constexpr int kBlockRows = 128, kBlockCols = 64;
constexpr int kBlockThreads = 512;
constexpr int kBlocksMax = 1 << 15;       // blocks of a plan: 3 GB of digits
constexpr int kBlockMatBytes = kMatDigits * kBlockRows * kBlockCols * 2;   // 96 KB of digits per block

struct BlockUnit {
  int in_off, in_cnt;      // into the list of input rows, at most kBlockCols of them
  int out_off, out_cnt;    // into the list of output rows, at most kBlockRows
  int mat;                 // block of digits
  int from;                // 0: in = b, out = x; 1: in = b, out = b; 2: in = x, out = x
};

struct BlockList {
  const BlockUnit* units = nullptr;
  const int32_t* in_rows = nullptr;
  const int32_t* out_rows = nullptr;
  const unsigned char* mats = nullptr;   // per block: digit, 8-column group, row, column
  const int* e_row = nullptr;            // per block and row of it: |entry| < 2^e
  int n = 0, spin = kMmaSpinLimit;
};

__host__ __device__ __forceinline__ uint32_t block_tmem_cols(int wp) { return wp <= 16 ? 128 : (wp <= 32 ? 256 : 512); }

size_t block_smem_bytes(int wp) {
  return (size_t)kBlockMatBytes + (size_t)kDatDigits * wp * kBlockCols * 2 + (size_t)(kBlockCols / 8 + 1) * wp * sizeof(uint32_t) + 64;
}

// 4 columns of each of the 7 accumulators are read by tmem_load_digits. Grid: x walks the units, y
// the tiles of wp problems of [w0, w0 + wn). The next unit's digits are fetched while this one's
// products are joined.
template <int wp>
__global__ void __launch_bounds__(kBlockThreads, 1) k_block_apply(BlockList L, double* b, double* x, int W, int w0,
                                                                 int wn, int* __restrict__ err) {
  pdl_begin();
  extern __shared__ __align__(128) unsigned char blk_sh[];
  constexpr int groups = kBlockCols / 8;
  constexpr int dat_bytes = kDatDigits * wp * kBlockCols * 2;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  unsigned char* mat = blk_sh;
  unsigned char* dat = blk_sh + kBlockMatBytes;
  uint32_t* colmax = reinterpret_cast<uint32_t*>(dat + dat_bytes);   // groups x wp
  int* colexp = reinterpret_cast<int*>(colmax + groups * wp);        // wp
  uint64_t* mbar = reinterpret_cast<uint64_t*>(colexp + wp);         // [0] MMA batches, [1] block copies
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int w_lo = w0 + blockIdx.y * wp, live_w = min(wp, w0 + wn - w_lo);
  // this thread's data: problem w_lo + dw, columns 8 kg .. 8 kg + 7 (lanes along the problems)
  const int dw = tid % wp, kg = tid / wp;
  double A[8];
  // (a launch never writes the rows that it reads)
  auto load = [&](const BlockUnit& U) {
    const double* in = U.from == 2 ? x : b;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = kg * 8 + e;
      A[e] = (kg < groups && dw < live_w && j < U.in_cnt)
                 ? in[(int64_t)__ldg(L.in_rows + U.in_off + j) * W + w_lo + dw] : 0.0;
    }
  };
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                 "r"(block_tmem_cols(wp)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  int u = blockIdx.x;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar + 1)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    *gave_up = 0;
    if (u < L.n) bulk_load(smem_addr(mat), L.mats + (size_t)L.units[u].mat * kBlockMatBytes, kBlockMatBytes, smem_addr(mbar + 1));
  }
  int copies = u < L.n ? 1 : 0, batches = 0;   // of blocks, started by thread 0; of products, by warp 0
  BlockUnit U{};
  if (u < L.n) {
    U = L.units[u];
    load(U);
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (!*gave_up && !mbar_wait(smem_addr(bar), parity, L.spin)) {
      *gave_up = 1;
      atomicExch(err, 1);
    }
  };
  for (; u < L.n; u += gridDim.x) {
    uint32_t top = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) top = max(top, (uint32_t)__double2hiint(A[e]) * 2u);
    if (kg < groups) colmax[kg * wp + dw] = top;
    __syncthreads();
    if (*gave_up) break;   // the same for all: no wait lies between the last barrier and this one
    if (kg < groups) {
#pragma unroll
      for (int k = 0; k < groups; ++k) top = max(top, colmax[k * wp + dw]);
      const int emax = max((int)(top >> 21), 64);
      if (kg == 0) colexp[dw] = emax;
      int64_t X[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) X[e] = fixed_of(A[e], emax) * 2;   // the digits' range is 2^62
      uint4 dig[kDatDigits];
      digits_of(X, dig);
#pragma unroll
      for (int i = 0; i < kDatDigits; ++i)
        *reinterpret_cast<uint4*>(dat + ((size_t)(kg * kDatDigits + i) * wp + dw) * 16) = dig[i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tmem_fence_before();   // this thread's accumulator loads of the previous unit are complete
    __syncthreads();
    if (warp == 0) {
      wait(mbar + 1, phase);   // the block's digits
      __syncwarp();
      tmem_fence_after();
      constexpr uint32_t lbo_a = kBlockRows * 16, lbo_b = kDatDigits * wp * 16;
      const uint64_t a0 = mma_desc(smem_addr(mat), lbo_a, 128), b0 = mma_desc(smem_addr(dat), lbo_b, 128);
      const bool go = !__any_sync(0xffffffffu, *gave_up);
      batches += go;
      if (elect_one() && go) {
        // block digit i times the data digits [j0, j0 + nj): accumulators i + j0 ...
        auto mma = [&](int i, int j0, int nj, int ks) {
          mma_f16(tmem + (uint32_t)((i + j0) * wp), a0 + (uint32_t)((i * groups + 2 * ks) * lbo_a >> 4),
                  b0 + (uint32_t)((2 * ks * lbo_b + j0 * wp * 16) >> 4), mma_idesc(nj * wp), (i | ks) ? 1u : 0u);
        };
#pragma unroll
        for (int ks = 0; ks < kBlockCols / 16; ++ks)
#pragma unroll
          for (int i = 0; i < kMatDigits; ++i) {   // digit 0 comes first and starts every accumulator
            constexpr int widest = 256 / wp;       // N is at most 256
#pragma unroll
            for (int j0 = 0; j0 < kDatDigits - i; j0 += widest)
              mma(i, j0, kDatDigits - i - j0 < widest ? kDatDigits - i - j0 : widest, ks);
          }
        mma_commit(smem_addr(mbar));
      }
      __syncwarp();
    }
    const BlockUnit now = U;
    const int row = tid & (kBlockRows - 1);   // of the join; where it goes is read ahead of the wait
    const bool live = row < now.out_cnt;
    double* dst = (now.from == 1 ? b : x) + (live ? (int64_t)__ldg(L.out_rows + now.out_off + row) * W : 0) + w_lo;
    const int e_row = __ldg(L.e_row + now.mat * kBlockRows + row);
    if (u + (int)gridDim.x < L.n) {
      U = L.units[u + gridDim.x];
      load(U);
    }
    wait(mbar, phase);
    __syncwarp();
    tmem_fence_after();
    const bool ok = !__any_sync(0xffffffffu, *gave_up);
    if (tid == 0 && u + (int)gridDim.x < L.n && ok) {   // every product has read the block
      bulk_load(smem_addr(mat), L.mats + (size_t)U.mat * kBlockMatBytes, kBlockMatBytes, smem_addr(mbar + 1));
      ++copies;
    }
    phase ^= 1u;
    // join (see k_sine_lines); warp quadrant = 32 rows, quarter of the problems per group of 4 warps
    const uint32_t lane_base = tmem + ((uint32_t)((tid >> 5) & 3) << 21);
#pragma unroll 1
    for (int blk = 0; blk < wp / 16; ++blk) {
      const int n0 = (tid >> 7) * (wp / 4) + blk * 4;
      if (n0 >= live_w || !ok) break;   // the same for the whole warp
      float P[kDatDigits][4];
      tmem_load_digits(lane_base + (uint32_t)n0, (uint32_t)wp, P);
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        int64_t R = __float2int_rn(fmaf(P[6][o], 0x1p-16f, fmaf(P[5][o], 0x1p-7f, P[4][o] * 4.0f)));
        R += (int64_t)__float2int_rn(P[3][o]) * (1 << 11);
        R += (int64_t)__float2int_rn(P[2][o]) * (1 << 20);
        R += (int64_t)__float2int_rn(P[1][o]) * (1 << 29);
        R += (int64_t)((uint64_t)(uint32_t)(__float2int_rn(P[0][o]) * 64) << 32);
        if (live && n0 + o < live_w) {
          const int emax = colexp[n0 + o];
          atomicAdd(dst + n0 + o, emax == 0x7ff ? __longlong_as_double((long long)kNaNBits)
                                                : double_of_fixed(R, emax - 1022 - 1 + e_row));
        }
      }
    }
  }
  if (tid == 0 && *gave_up) mbar_drain(mbar, copies, batches);
  tmem_fence_before();
  __syncthreads();
  if (tid < 32) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(block_tmem_cols(wp)));
  }
}

using BlockKernel = void (*)(BlockList, double*, double*, int, int, int, int*);
BlockKernel block_kernel(int wp) {
  return wp == 16 ? k_block_apply<16> : wp == 32 ? k_block_apply<32> : wp == 48 ? k_block_apply<48> : k_block_apply<64>;
}

// problems per tile: the width whose rounds of units over the SMs cost least, a unit costing about
// 3 + 0.14 wp thousand cycles (reading and splitting, products, joining)
int block_width(int n_units, int wn) {
  int best = 64;
  double cost = 1e300;
  for (int wp : {16, 32, 48, 64}) {
    const int64_t rounds = ((int64_t)n_units * ((wn + wp - 1) / wp) + kNumSMs - 1) / kNumSMs;
    const double c = (double)rounds * (3.0 + 0.14 * std::min(wp, wn));
    if (c < cost * 0.999) {
      cost = c;
      best = wp;
    }
  }
  return best;
}

// ---- setup -----------------------------------------------------------------------------------------

// b = columns c0 .. c0 + 63 of the identity on the listed rows (row i of the list has its one in column
// pos[i] - c0), zero elsewhere; b is zeroed before
__global__ void k_unit_columns(double* __restrict__ b, const int32_t* __restrict__ rows,
                               const int32_t* __restrict__ pos, int n, int c0) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (pos[i] >= c0 && pos[i] < c0 + kBlockCols) b[(int64_t)rows[i] * kBlockCols + pos[i] - c0] = 1.0;
}

// where a block's entries lie in the setup's store: entry (r, j) at base + r s_r + j s_c
struct BlockSource {
  int64_t base, s_r, s_c;
  int rows, cols;
};

// The listed rows (null: all n) of E - K (x + dx), E the columns c0 .. c0 + 63 of the identity as in
// k_unit_columns (pos null: zero), in twice the working precision (exact products, two-sums): residuals for
// refining the blocks, and couplings. K by rows in the factor's order.
struct MatrixRows {
  const int64_t* ptr = nullptr;
  const int32_t* idx = nullptr;
  const double* val = nullptr;
};
__global__ void __launch_bounds__(256) k_residual(MatrixRows K, const int32_t* __restrict__ rows,
                                                  const int32_t* __restrict__ pos, int n, int c0,
                                                  const double* __restrict__ x, const double* __restrict__ dx,
                                                  double* __restrict__ out) {
  const int64_t total = (int64_t)n * kBlockCols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / kBlockCols), j = (int)(e % kBlockCols), r = rows ? rows[i] : i;
    double hi = pos && pos[i] == c0 + j ? 1.0 : 0.0, lo = 0.0;
    for (int64_t k = K.ptr[r]; k < K.ptr[r + 1]; ++k) {
      const double a = -K.val[k], v = x[(int64_t)K.idx[k] * kBlockCols + j];
      const double p = a * v, s = hi + p, t = s - hi;
      lo += ((hi - (s - t)) + (p - t)) + fma(a, v, -p);
      if (dx) lo = fma(a, dx[(int64_t)K.idx[k] * kBlockCols + j], lo);
      hi = s;
    }
    out[(int64_t)r * kBlockCols + j] = hi + lo;
  }
}

// rows of 64 solved columns (x + dx, dx may be null) into the store: dst + i s_i + j for list rows i, columns j < cnt
struct StoreRows {
  int64_t dst;       // of the list's first row, column c0
  int64_t s_i;       // between rows; columns are s_j apart
  int64_t s_j;
  int first, count;  // rows of the list
  int cols;          // columns in range (cnt - c0 <= 64)
};
__global__ void k_store_rows(const double* __restrict__ x, const double* __restrict__ dx,
                             const int32_t* __restrict__ rows, const StoreRows* __restrict__ jobs,
                             double* __restrict__ store) {
  const StoreRows J = jobs[blockIdx.x];
  for (int i = threadIdx.x; i < J.count * kBlockCols; i += blockDim.x) {
    const int r = i / kBlockCols, j = i % kBlockCols;
    const int64_t at = (int64_t)rows[J.first + r] * kBlockCols + j;
    if (j < J.cols) store[J.dst + r * J.s_i + j * J.s_j] = dx ? x[at] + dx[at] : x[at];
  }
}

// digits of the blocks, each row scaled by its own largest magnitude; one thread block per block, a warp
// per row. (One scale for a block's 128 rows held the rows of small entries to fewer bits: with resistances
// of a lognormal spread of 3 the phases moved 15 times further from the exact ones.)
__global__ void __launch_bounds__(256) k_block_digits(const double* __restrict__ store,
                                                      const BlockSource* __restrict__ src,
                                                      unsigned char* __restrict__ mats, int* __restrict__ e_row) {
  const BlockSource B = src[blockIdx.x];
  const int lane = threadIdx.x & 31;
  __half* m = reinterpret_cast<__half*>(mats + (size_t)blockIdx.x * kBlockMatBytes);
  for (int r = threadIdx.x >> 5; r < kBlockRows; r += blockDim.x >> 5) {
    double v[kBlockCols / 32];
    uint32_t top = 0;
#pragma unroll
    for (int q = 0; q < kBlockCols / 32; ++q) {
      const int j = lane + 32 * q;
      v[q] = r < B.rows && j < B.cols ? store[B.base + r * B.s_r + j * B.s_c] : 0.0;
      top = max(top, (uint32_t)__double2hiint(v[q]) * 2u);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    const int e = max((int)(top >> 21), 64) - 1022;
    if (lane == 0) e_row[(size_t)blockIdx.x * kBlockRows + r] = e;
#pragma unroll
    for (int q = 0; q < kBlockCols / 32; ++q) {
      const int j = lane + 32 * q;
      uint64_t t = (uint64_t)llrint(scalbn(v[q], 53 - e));   // 2^53 of the scale
#pragma unroll
      for (int d = 0; d < kMatDigits; ++d) t += 256ull << (9 * d);
#pragma unroll
      for (int d = 0; d < kMatDigits; ++d) {
        const int f9 = (int)((t >> (9 * (kMatDigits - 1 - d))) & (d ? 511 : 1023)) - 256;
        m[(((size_t)d * (kBlockCols / 8) + j / 8) * kBlockRows + r) * 8 + j % 8] = __float2half((float)f9);
      }
    }
  }
}

}  // namespace
