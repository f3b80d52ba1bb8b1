// Sine-transform solve of uniform square arrays on the tensor cores (included by jja_gb300.cu).
//
// With equal R, C and a uniform self-inductance K = kappa (4 I - adjacency) on the grid of faces.
// A solve is three kernels: the sine transform (DST-I) of every grid line along one axis, a
// tridiagonal solve along the other axis per (mode, problem), and the sine transform back.
//   x = S (tridiagonal_k)^-1 S b / (kappa (m + 1) / 2),   S_kj = sin(pi k j / (m + 1)).
//
// The transforms are contractions with a constant matrix. GB300's FP64 pipe does 2 FMA per clock
// and SM, its tensor cores 4096 (FP16 in, FP32 out), so the product is formed in pieces: both
// factors are held in fixed point (the matrix in 54 bits against 1, the data in 63 bits against
// the largest magnitude of its line) and cut into 6 and 7 signed digits of 9 bits; FP16 holds a
// digit exactly, the products of the digits i and j with i + j = g <= 6 are summed by tcgen05.mma
// into the FP32 accumulator g (integers, below 2^24 for g <= 3; above that a rounding lies under
// 2^-53 of the largest term; the products left out lie below 2^-60), and the seven integers are
// joined in 64-bit fixed point and rounded once to FP64: the error is that of the stored result
// and of the matrix entries, smaller than an FP64 dot product's. Splitting and joining run on the
// integer pipe. (The scheme is the error-free splitting of Ozaki, Ogita, Oishi and Rump,
// Numerical Algorithms 59, 2012, with fixed-point digits. 6 data digits, 21 products instead of
// 27, were measured to leave residuals 4-6 times those of FP64 triangular sweeps.)
//
// Even and odd modes see x_j + x_{N-j} and x_j - x_{N-j} (N = m + 1), which halves the products:
// two contractions of length <= 64 for lines of up to 128 faces.
//
// Measured (GB300, the face solve of a step; the sweeps they replace -> these kernels): 128x128 x
// 512 problems 850 -> 195 us (70 us per transform, 56 us for the chains: 43 us of FP64 work), 101x60 x
// 24 178 -> 31 us; an adjoint run on 64x64 x 64 121 -> 46 ms (critical currents that the
// plan has not seen: 181 -> 52); 1024x1024 x 8 (8 strips) 1976 -> 510 us:
// 77 us per transform, 108 and 159 us for the two passes over the chains (72 and 100 us of FP64 work),
// 30 us for the edges, 44 us for the separators. A tile (128 columns of 127 faces) takes about 30k
// cycles: reading and splitting 6k, twice the products 3.8k (3.5k of MMA issue at the multipliers' rate)
// and the joining 7k. Overlapping the products with the joins (chunks of modes, two sets of accumulators) was
// measured and gained nothing: at 16 warps the digit work itself waits on its own latencies.
// What bounds it: the shifts and logic of splitting and joining (the ALU pipe runs half a warp
// instruction per clock and scheduler), serialised with the products because one tile's digits and
// accumulators fill the SM's shared memory and TMEM.

namespace {

constexpr int kMatDigits = 6;                  // 9-bit digits of a matrix entry
constexpr int kDatDigits = 7;                  // ... of a data value; also the number of accumulators
constexpr int kSineMaxPoints = 128;            // longest transform (folded length 64)
constexpr int kSineMaxSide = 4096;             // of the grid (the separators' dense sine matrix: 200 MB of digits)
constexpr int kSineColumns = 128;              // (line, problem) columns per tile: the MMA's M
constexpr int kSineThreads = 512;
// TMEM columns of the 7 accumulators of kp columns each (a power of two is allocated)
__host__ __device__ __forceinline__ uint32_t sine_tmem_cols(int kp) { return kp <= 16 ? 128 : (kp <= 32 ? 256 : 512); }
constexpr int kMmaSpinLimit = 1 << 24;   // try_wait polls; far beyond any MMA batch (~3 us)

// one transform direction: m points a line, `lines` lines, element (line, t, w) at
// line * s_c + t * s_t + w; half lengths padded to kp (a multiple of 16)
struct SineArgs {
  int m, kp, lines;
  int64_t s_t, s_c;
  int64_t off, s_strip;   // first line, and between strips of the grid (see SineStrips)
  FastDiv per_strip;      // lines of one strip
  int parts;            // blocks a tile of columns is shared by: 1, 2 (odd, even modes) or 2 x mode chunks
  const unsigned char* mat;   // digits of the odd and even half matrices in the MMA operand layout
  int e_shift;          // result exponent offset (the power-of-two part of the scale)
  int spin = kMmaSpinLimit;
};

struct SineTri {
  int n, top;           // points a chain, points of the upper half
  int lines;            // chains: strips x modes
  FastDiv modes;        // modes per strip
  int64_t s_n, s_c;     // strides along a chain and between modes
  int64_t off, s_strip;
  const double* c;      // c[i * modes + mode]: reciprocal pivots, from either end
  const double* g;      // per mode: the join at the middle (top, then bottom)
  // values on the separators beside the strips (null: none): sep[(i * seps + s) * W + w], added to the
  // right-hand side as edge[mode] times the sum (modes 1, 3, ...) or difference of both sides'
  const double* sep;
  const double* edge;
  int seps, strip0;     // separators of the grid, first strip of this launch
  // chains in segments (k_sine_chain): `segs` warps of `seg_len` points each (the last one shorter), one
  // point between neighbours; segs = 0: two halves (k_sine_tri)
  int segs, seg_len;
  const double* spike;  // spike[i * modes + mode]: response at point i to the point before the segment
  const double* spike_last;
  const double* seg_piv;   // reciprocal pivots across the points between segments
  const double* seg_cpl;   // per mode: coupling through a whole segment
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory operand descriptor, K-major without swizzle: 8 x 16-byte core matrices, `lbo`
// bytes apart along K and `sbo` bytes apart along M or N
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// FP16 x FP16 -> FP32, both operands K-major, M = 128
__device__ __forceinline__ uint32_t mma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

// one lane of a converged warp (the MMA issue then keeps its descriptors in uniform registers)
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}

// bounded wait for the mbarrier's phase; false when the bound ran out. A kernel whose wait ran out reports it,
// starts no further copies or products, and waits again (drain) for those in flight before it gives its memory back.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int limit) {
  for (int i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}

// 4 columns of each of the 7 accumulators (`stride` columns apart) for this thread's lane. One
// statement with the wait, so no use of the values can be scheduled before they have arrived.
__device__ __forceinline__ void tmem_load_digits(uint32_t addr, uint32_t stride, float (*v)[4]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%28];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%29];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%30];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12, %13, %14, %15}, [%31];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16, %17, %18, %19}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20, %21, %22, %23}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24, %25, %26, %27}, [%34];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(v[0][0]), "=f"(v[0][1]), "=f"(v[0][2]), "=f"(v[0][3]), "=f"(v[1][0]), "=f"(v[1][1]),
        "=f"(v[1][2]), "=f"(v[1][3]), "=f"(v[2][0]), "=f"(v[2][1]), "=f"(v[2][2]), "=f"(v[2][3]),
        "=f"(v[3][0]), "=f"(v[3][1]), "=f"(v[3][2]), "=f"(v[3][3]), "=f"(v[4][0]), "=f"(v[4][1]),
        "=f"(v[4][2]), "=f"(v[4][3]), "=f"(v[5][0]), "=f"(v[5][1]), "=f"(v[5][2]), "=f"(v[5][3]),
        "=f"(v[6][0]), "=f"(v[6][1]), "=f"(v[6][2]), "=f"(v[6][3])
      : "r"(addr), "r"(addr + stride), "r"(addr + 2 * stride), "r"(addr + 3 * stride), "r"(addr + 4 * stride),
        "r"(addr + 5 * stride), "r"(addr + 6 * stride)
      : "memory");
}

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// x 2^(61 - E) as an integer (truncated; one unit low when negative), E = emax - 1022 for the
// line's largest biased exponent emax >= 64 (|x| < 2^E, so the result is below 2^61 in magnitude).
// The implicit bit is set for subnormals and zero too: their shift leaves nothing of it. GB300's
// ALU pipe (shifts, logic, adds) has half the FMA pipe's rate, so left shifts are multiplications.
__device__ __forceinline__ int64_t fixed_of(double x, int emax) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu);
  const uint64_t M = (uint64_t)lo * 256u + ((uint64_t)(((hi & 0xfffffu) | 0x100000u) * 256u) << 32);
  return (int64_t)(M >> min(emax - e, 63)) ^ (int64_t)((int32_t)hi >> 31);
}

// R 2^(e - 53) as a double, |R| < 2^62, rounded half up in magnitude; zero below the normal range
__device__ __forceinline__ double double_of_fixed(int64_t R, int e) {
  const int32_t neg = (int32_t)(R >> 63);
  const uint64_t a = (uint64_t)((R ^ (int64_t)neg) - neg);
  uint32_t h = (uint32_t)(a >> 32), l = (uint32_t)a;
  int top = e + (1023 + 63 - 53 - 1);   // biased exponent - 1 of a leading bit at position 63
  if (h == 0) {                         // rare: far below the line's scale
    h = l >> 2;
    l = l << 30;
    top -= 30;
  }
  const int sh = __clz((int)h) - 1;     // the leading bit to position 62: the rounding cannot overflow
  uint64_t n = ((uint64_t)__funnelshift_l(l, h, sh) << 32) | (l << sh);
  n = (n + 0x200u) >> 10;
  const int ex = top - 1 - sh;
  uint32_t rh = (uint32_t)(n >> 32) + (uint32_t)ex * (1u << 20), rl = (uint32_t)n;
  if ((uint32_t)ex > 2044u || h == 0) {   // rare: zero, underflow, overflow
    rh = ex > 2044 && h != 0 ? 0x7ff00000u : 0u;
    rl = 0u;
  }
  return __hiloint2double((int)(rh | ((uint32_t)neg & 0x80000000u)), (int)rl);
}

// the balanced digits of 8 fixed-point numbers (|X| <= 2^62), as FP16: out[i] holds digit i of the
// 8 numbers. X + 256 (1 + 2^9 + ... + 2^54) has the digits + 256 as plain 9-bit fields; a field
// placed in the mantissa of 1024.0 is 1024 + digit + 256 exactly.
__device__ __forceinline__ void digits_of(const int64_t* X, uint4* out) {
  constexpr uint64_t kOffset = 256ull * ((1ull << 54) + (1ull << 45) + (1ull << 36) + (1ull << 27) + (1ull << 18) +
                                         (1ull << 9) + 1ull);
  const __half2 bias = __halves2half2(__ushort_as_half((unsigned short)0x6500), __ushort_as_half((unsigned short)0x6500));   // 1280
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint64_t t0 = (uint64_t)X[2 * p] + kOffset, t1 = (uint64_t)X[2 * p + 1] + kOffset;
    const uint32_t l0 = (uint32_t)t0, h0 = (uint32_t)(t0 >> 32), l1 = (uint32_t)t1, h1 = (uint32_t)(t1 >> 32);
    const uint32_t lo[kDatDigits] = {h0 >> 22, h0 >> 13, h0 >> 4, __funnelshift_r(l0, h0, 27), l0 >> 18, l0 >> 9, l0};
    // the second number's field moved to bit 16
    const uint32_t up[kDatDigits] = {h1 >> 6, h1 << 3, h1 << 12, __funnelshift_r(l1, h1, 11), l1 >> 2, l1 << 7, l1 << 16};
#pragma unroll
    for (int i = 0; i < kDatDigits; ++i) {
      const uint32_t both = (lo[i] & 0xffffu) | (up[i] & 0xffff0000u);
      const uint32_t packed = (both & (i ? 0x01ff01ffu : 0x03ff03ffu)) | 0x64006400u;
      const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&packed), bias);
      reinterpret_cast<uint32_t*>(&out[i])[p] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
}

// before a kernel whose wait ran out ends: the last of its copies (counted on mbar[1]) and batches of products (mbar[0])
__device__ __forceinline__ void mbar_drain(uint64_t* mbar, int copies, int batches) {
  if (copies) mbar_wait(smem_addr(mbar + 1), (uint32_t)(copies - 1) & 1u, kMmaSpinLimit);
  if (batches) mbar_wait(smem_addr(mbar), (uint32_t)(batches - 1) & 1u, kMmaSpinLimit);
}

// `bytes` (a multiple of 16) from global to shared memory, counted on the mbarrier
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar) : "memory");
}

// Sine transform of every line for problems [w0, w0 + wn), in != out. Tiles of 128 (line, problem)
// columns on a persistent grid, one block per SM; with few tiles a tile is shared by `parts`
// blocks, each joining the odd or the even modes, or a chunk of them, and the tiles of a last wave
// that fills at most half of the blocks are shared by two (508 tiles on 152 blocks: 3.5 instead of
// 4 tiles' time). Shared memory: the matrix
// digits (2 halves x 6 digits x kp x kp, one bulk copy), the data digits of one half
// (7 x 128 x kp), scales and barriers.
template <int kp>
__global__ void __launch_bounds__(kSineThreads, 1) k_sine_lines(SineArgs d, const double* __restrict__ in,
                                                               double* __restrict__ out, int w0, int wn,
                                                               FastDiv by_wn, int* __restrict__ err) {
  pdl_begin();
  extern __shared__ __align__(128) unsigned char sine_sh[];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), m = d.m, half = m >> 1;
  constexpr uint32_t mat_bytes = kMatDigits * kp * kp * 2;   // one half's digits
  constexpr int dat_bytes = kDatDigits * kp * kSineColumns * 2;
  unsigned char* mat = sine_sh;
  unsigned char* dat = sine_sh + 2 * mat_bytes;
  uint32_t* colmax = reinterpret_cast<uint32_t*>(dat + dat_bytes);    // 4 x 128
  uint64_t* mbar = reinterpret_cast<uint64_t*>(colmax + 4 * kSineColumns);   // [0] MMA batches, [1] the matrix copy
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // this block's share of its tiles: halves [p_lo, p_hi), modes [n_lo, n_lo + nc) of each
  const int part = blockIdx.x % d.parts, chunks = d.parts > 2 ? d.parts / 2 : 1;
  int p_lo = d.parts > 1 ? part & 1 : 0, p_hi = d.parts > 1 ? p_lo + 1 : 2;
  const int nc = kp / chunks, n_lo = (part >> 1) * nc;
  const int64_t ncols = (int64_t)d.lines * wn;
  const int tiles = (int)((ncols + kSineColumns - 1) / kSineColumns);
  const int col = tid & (kSineColumns - 1), q4 = tid >> 7;   // column of the tile, quarter of the k groups
  constexpr int groups = kp / 8;                             // 8-point groups of a half
  int tile = blockIdx.x / d.parts;
  const int tile_step = gridDim.x / d.parts;
  // the first tile of a last wave in halves (parts = 1), or no such tile
  const int left = tiles % (int)gridDim.x;
  const int halves_from = d.parts == 1 && 2 * left <= (int)gridDim.x ? tiles - left : INT_MAX;
  // the pairs x_j, x_{N-j} of this thread's k groups (doubles, then fixed point)
  int64_t A[2][8], B[2][8];
  auto load = [&](int tl) {
    const int64_t c = (int64_t)tl * kSineColumns + col;
    const bool live = c < ncols;
    const int64_t line = live ? by_wn(c) : 0, strip = d.per_strip(line);
    const double* src = in + d.off + strip * d.s_strip + (line - strip * d.per_strip.d) * d.s_c + (live ? w0 + (c - line * wn) : 0);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int j = (q4 + 4 * r) * 8 + e;
        double a = 0.0, b = 0.0;
        if (live && j < m - half) a = src[(int64_t)j * d.s_t];
        if (live && j < half) b = src[(int64_t)(m - 1 - j) * d.s_t];   // none for the middle of an odd line
        A[r][e] = __double_as_longlong(a);
        B[r][e] = __double_as_longlong(b);
      }
  };
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                 "r"(sine_tmem_cols(kp)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar + 1)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    *gave_up = 0;
    bulk_load(smem_addr(mat + p_lo * mat_bytes), d.mat + (size_t)p_lo * mat_bytes, (uint32_t)(p_hi - p_lo) * mat_bytes,
              smem_addr(mbar + 1));
  }
  if (tile < tiles) load(tile);
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (!*gave_up && !mbar_wait(smem_addr(bar), parity, d.spin)) {
      *gave_up = 1;
      atomicExch(err, 1);
    }
  };
  int batches = 0;                   // of products, started by warp 0
  if (tid == 0) wait(mbar + 1, 0);   // only the MMA issuer reads the matrix
  __syncwarp();
  while (tile < tiles) {
    const bool last = tile >= halves_from;
    int next = last ? tiles : tile + tile_step;
    if (!last && next >= halves_from) next = halves_from + ((int)blockIdx.x >> 1);
    if (last) {
      p_lo = blockIdx.x & 1;
      p_hi = p_lo + 1;
    }
    const int64_t c = (int64_t)tile * kSineColumns + col;
    const bool live = c < ncols;
    const int64_t line = live ? by_wn(c) : 0, strip = d.per_strip(line);
    double* dst = out + d.off + strip * d.s_strip + (line - strip * d.per_strip.d) * d.s_c + (live ? w0 + (c - line * wn) : 0);
    uint32_t top = 0;   // the line's largest magnitude (high words without the sign)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e)
        top = max(top, max((uint32_t)(A[r][e] >> 32) * 2u, (uint32_t)(B[r][e] >> 32) * 2u));
    colmax[q4 * kSineColumns + col] = top;
    __syncthreads();
    if (*gave_up) break;   // the same for all: no wait lies between the last barrier and this one
#pragma unroll
    for (int q = 0; q < 4; ++q) top = max(top, colmax[q * kSineColumns + col]);
    const int emax = max((int)(top >> 21), 64);
    const bool bad = emax == 0x7ff;      // a NaN or inf in the line: NaN in every mode of it
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        A[r][e] = fixed_of(__longlong_as_double(A[r][e]), emax);
        B[r][e] = fixed_of(__longlong_as_double(B[r][e]), emax);
      }
#pragma unroll 1
    for (int parity = p_lo; parity < p_hi; ++parity) {   // 0: modes 1, 3, 5, ... (sums), 1: 2, 4, ... (differences)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int kg = q4 + 4 * r;
        if (kg < groups) {
          int64_t X[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) X[e] = parity ? A[r][e] - B[r][e] : A[r][e] + B[r][e];
          uint4 dig[kDatDigits];
          digits_of(X, dig);
#pragma unroll
          for (int i = 0; i < kDatDigits; ++i)
            *reinterpret_cast<uint4*>(dat + ((size_t)(i * groups + kg) * kSineColumns + col) * 16) = dig[i];
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tmem_fence_before();       // this thread's accumulator loads of the previous half are complete
      __syncthreads();
      if (warp == 0) {
        // data digit j times the matrix digits [i0, i0 + ni) side by side (they are adjacent in the
        // operand's N, and so are their accumulators i + j in TMEM): wide MMAs read the data
        // digits once for up to four products, which leaves them bound by the multipliers
        tmem_fence_after();
        constexpr uint32_t lbo_a = kSineColumns * 16, lbo_b = kMatDigits * kp * 16;
        const uint64_t a0 = mma_desc(smem_addr(dat), lbo_a, 128);
        const uint64_t b0 = mma_desc(smem_addr(mat) + (uint32_t)parity * mat_bytes, lbo_b, 128);
        const bool go = !__any_sync(0xffffffffu, *gave_up);
        batches += go;
        if (elect_one() && go) {
          auto mma = [&](int j, int i0, int ni, int ks, bool add) {
            mma_f16(tmem + (uint32_t)((i0 + j) * kp), a0 + (uint32_t)((j * groups + 2 * ks) * lbo_a >> 4),
                    b0 + (uint32_t)((2 * ks * lbo_b + i0 * kp * 16) >> 4), mma_idesc(ni * kp), add ? 1u : 0u);
          };
#pragma unroll
          for (int ks = 0; ks < kp / 16; ++ks) {
            mma(6, 0, 1, ks, ks > 0);   // the first products of every accumulator start it
            mma(0, 0, 4, ks, ks > 0);
            mma(0, 4, 2, ks, ks > 0);
            mma(1, 0, 4, ks, true);
            mma(1, 4, 2, ks, true);
            mma(2, 0, 4, ks, true);
            mma(2, 4, 1, ks, true);
            mma(3, 0, 4, ks, true);
            mma(4, 0, 3, ks, true);
            mma(5, 0, 2, ks, true);
          }
          mma_commit(smem_addr(mbar));
        }
        __syncwarp();
      }
      // the next tile's values arrive during the last half's products
      if (parity + 1 == p_hi && next < tiles) load(next);
      wait(mbar, phase);
      phase ^= 1u;
      __syncwarp();
      tmem_fence_after();
      // join the seven integers of every (column, mode): P0 2^38 + P1 2^29 + ... + P6 2^-16, units
      // 2^-54 of the line's scale. Warp quadrant = 32 columns, q4 = a quarter of the modes
      const uint32_t lane_base = tmem + ((uint32_t)((tid >> 5) & 3) << 21);
      const int count = parity ? half : m - half;
      if (__any_sync(0xffffffffu, *gave_up)) continue;
      for (int blk = 0; blk < (nc >> 4); ++blk) {
        const int n0 = q4 * (nc >> 2) + blk * 4;
        float P[kDatDigits][4];
        tmem_load_digits(lane_base + (uint32_t)(n_lo + n0), (uint32_t)kp, P);
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          // the last three in FP32: an error of 2^-24 P4, a fraction of R's unit
          int64_t R = __float2int_rn(fmaf(P[6][o], 0x1p-16f, fmaf(P[5][o], 0x1p-7f, P[4][o] * 4.0f)));
          R += (int64_t)__float2int_rn(P[3][o]) * (1 << 11);
          R += (int64_t)__float2int_rn(P[2][o]) * (1 << 20);
          R += (int64_t)__float2int_rn(P[1][o]) * (1 << 29);
          R += (int64_t)((uint64_t)(uint32_t)(__float2int_rn(P[0][o]) * 64) << 32);
          const int k = n_lo + n0 + o;
          if (live && k < count)
            dst[(int64_t)(2 * k + parity) * d.s_t] =
                bad ? __longlong_as_double((long long)kNaNBits) : double_of_fixed(R, emax - 1022 + d.e_shift);
        }
      }
    }
    tile = next;
  }
  if (tid == 0 && *gave_up) mbar_drain(mbar, 1, batches);
  tmem_fence_before();
  __syncthreads();
  if (tid < 32) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(sine_tmem_cols(kp)));
  }
}

using SineKernel = void (*)(SineArgs, const double*, double*, int, int, FastDiv, int*);
SineKernel sine_kernel(int kp) {
  return kp == 16 ? k_sine_lines<16> : kp == 32 ? k_sine_lines<32> : kp == 48 ? k_sine_lines<48> : k_sine_lines<64>;
}

// blocks per tile: as many parts as keep the launch within one block per SM (a single tile's
// latency is the digits of its columns, the products, and the joining of its modes, which the
// parts divide)
int sine_parts(int kp, int64_t tiles) {
  int parts = 1;
  for (int q : {2, 4, 8})
    if (tiles * q <= kNumSMs && kp % (16 * std::max(1, q / 2)) == 0) parts = q;
  return parts;
}

size_t sine_smem_bytes(int kp) {
  return (size_t)kp * 2 * (2 * kMatDigits * kp + kDatDigits * kSineColumns) + 4 * kSineColumns * sizeof(int) + 64;
}

// Tridiagonal solve per (mode, problem), in -> out (which may be the same array):
// (lambda_mode + 2) x_i - x_{i-1} - x_{i+1} = v_i, eliminated from both ends towards the middle by two
// threads (half the chain each), joined there, and substituted back outwards. 3 FP64 operations per
// element, 5 with values on the separators.
constexpr int kTriColumns = 64;
template <bool kSep>
__global__ void __launch_bounds__(2 * kTriColumns) k_sine_tri(SineTri t, const double* in, double* out, int W, int w0,
                                                             int wn, FastDiv by_wn) {
  pdl_begin();
  __shared__ double join_z[2][kTriColumns];
  const int side = threadIdx.x / kTriColumns, lc = threadIdx.x - side * kTriColumns;   // 0: from the first point
  const int64_t c = (int64_t)blockIdx.x * kTriColumns + lc, ncols = (int64_t)t.lines * wn;
  const bool live = c < ncols;
  const int64_t line = live ? by_wn(c) : 0;
  const int strip = (int)t.modes(line), modes = (int)t.modes.d, mode = (int)line - strip * modes;
  const int w = w0 + (live ? (int)(c - line * wn) : 0);
  const int cnt = side ? t.n - t.top : t.top;
  const int64_t step = side ? -t.s_n : t.s_n;
  const int64_t base = t.off + strip * t.s_strip + (int64_t)mode * t.s_c + w + (side ? (int64_t)(t.n - 1) * t.s_n : 0);
  const double* src = in + base;
  double* dst = out + base;
  const double* ct = t.c + mode;
  // the separators before and after the strip
  const int s1 = t.strip0 + strip;
  const double* sep_l = kSep && s1 > 0 ? t.sep + ((int64_t)(side ? t.n - 1 : 0) * t.seps + s1 - 1) * W + w : nullptr;
  const double* sep_r = kSep && s1 < t.seps ? t.sep + ((int64_t)(side ? t.n - 1 : 0) * t.seps + s1) * W + w : nullptr;
  const int64_t sep_step = (side ? -1 : 1) * (int64_t)t.seps * W;
  const double edge = kSep ? __ldg(t.edge + mode) : 0.0;
  auto rhs = [&](int i) -> double {
    const double v = src[(int64_t)i * step];
    if (!kSep) return v;
    double s = sep_l ? __ldg(sep_l + i * sep_step) : 0.0;
    if (sep_r) s += signed_by(__ldg(sep_r + i * sep_step), mode & 1);
    return fma(edge, s, v);
  };
  double z = 0.0, cp = 0.0;
  if (live) {
    // z_i = v_i + c_{i-1} z_{i-1}; c_i z_i is kept for the way back
    int i = 0;
    for (; i + 8 <= cnt; i += 8) {
      double x[8], cc[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = rhs(i + u);
        cc[u] = __ldg(ct + (int64_t)(i + u) * modes);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        z = fma(cp, z, x[u]);
        cp = cc[u];
        dst[(int64_t)(i + u) * step] = cp * z;
      }
    }
    for (; i < cnt; ++i) {
      z = fma(cp, z, rhs(i));
      cp = __ldg(ct + (int64_t)i * modes);
      dst[(int64_t)i * step] = cp * z;
    }
  }
  join_z[side][lc] = cp * z;    // z / pivot of the half's last point
  __syncthreads();
  if (!live || cnt == 0) return;
  // x at the two middle points: x_b = (z_b + c_t z_t) c_b / (1 - c_t c_b), and the same mirrored
  const double other = join_z[side ^ 1][lc];
  double x = (z + other) * __ldg(t.g + (int64_t)side * modes + mode);
  dst[(int64_t)(cnt - 1) * step] = x;
  int i = cnt - 2;
  for (; i >= 7; i -= 8) {
    double y[8], cc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      y[u] = dst[(int64_t)(i - u) * step];
      cc[u] = __ldg(ct + (int64_t)(i - u) * modes);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x = fma(cc[u], x, y[u]);
      dst[(int64_t)(i - u) * step] = x;
    }
  }
  for (; i >= 0; --i) {
    x = fma(__ldg(ct + (int64_t)i * modes), x, dst[(int64_t)i * step]);
    dst[(int64_t)i * step] = x;
  }
}

// The same with a chain's points split over `segs` warps (lane = column): each eliminates its segment
// with zero outside values and forms the solution at its ends (one elimination and one dot product),
// one warp solves for the points between the segments, and each substitutes back with them:
// 5 FP64 operations per element instead of 3, chains of n / segs instead of n / 2 dependent ones.
constexpr int kMaxSegs = 16;
template <bool kSep>
__global__ void __launch_bounds__(32 * kMaxSegs) k_sine_chain(SineTri t, const double* in, double* out, int W, int w0,
                                                             int wn, FastDiv by_wn) {
  pdl_begin();
  __shared__ double u1[kMaxSegs][32], uL[kMaxSegs][32], mid[kMaxSegs][32];
  const int seg = threadIdx.x >> 5, lane = threadIdx.x & 31, segs = t.segs, len_full = t.seg_len;
  const int64_t c = (int64_t)blockIdx.x * 32 + lane, ncols = (int64_t)t.lines * wn;
  const bool live = c < ncols;
  const int64_t line = live ? by_wn(c) : 0;
  const int strip = (int)t.modes(line), modes = (int)t.modes.d, mode = (int)line - strip * modes;
  const int w = w0 + (live ? (int)(c - line * wn) : 0);
  const int pos0 = seg * (len_full + 1), len = min(len_full, t.n - pos0);
  const bool last = seg == segs - 1;
  const int64_t base = t.off + strip * t.s_strip + (int64_t)mode * t.s_c + w + (int64_t)pos0 * t.s_n;
  const double* src = in + base;
  double* dst = out + base;
  const double* ct = t.c + mode;
  const double* sp = (last ? t.spike_last : t.spike) + mode;
  const int s1 = t.strip0 + strip;
  const double* sep_l = kSep && s1 > 0 ? t.sep + ((int64_t)pos0 * t.seps + s1 - 1) * W + w : nullptr;
  const double* sep_r = kSep && s1 < t.seps ? t.sep + ((int64_t)pos0 * t.seps + s1) * W + w : nullptr;
  const int64_t sep_step = (int64_t)t.seps * W;
  const double edge = kSep ? __ldg(t.edge + mode) : 0.0;
  auto rhs = [&](int i) -> double {
    const double v = src[(int64_t)i * t.s_n];
    if (!kSep) return v;
    double s = sep_l ? __ldg(sep_l + i * sep_step) : 0.0;
    if (sep_r) s += signed_by(__ldg(sep_r + i * sep_step), mode & 1);
    return fma(edge, s, v);
  };
  double z = 0.0, first = 0.0, cp = 0.0;
  if (live) {
    const double between = last ? 0.0 : rhs(len_full);
    int i = 0;
    for (; i + 8 <= len; i += 8) {
      double x[8], cc[8], ll[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = rhs(i + u);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        cc[u] = __ldg(ct + (int64_t)(i + u) * modes);
        ll[u] = __ldg(sp + (int64_t)(i + u) * modes);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        z = fma(cp, z, x[u]);
        cp = cc[u];
        first = fma(ll[u], x[u], first);
        dst[(int64_t)(i + u) * t.s_n] = z;
      }
    }
    for (; i < len; ++i) {
      const double x = rhs(i);
      z = fma(cp, z, x);
      cp = __ldg(ct + (int64_t)i * modes);
      first = fma(__ldg(sp + (int64_t)i * modes), x, first);
      dst[(int64_t)i * t.s_n] = z;
    }
    mid[seg][lane] = between;
  }
  u1[seg][lane] = first;
  uL[seg][lane] = cp * z;
  __syncthreads();
  if (seg == 0 && live) {
    const double cpl = __ldg(t.seg_cpl + mode);
    double y = 0.0;
    for (int s = 0; s + 1 < segs; ++s) {
      y = fma(cpl, y, mid[s][lane] + uL[s][lane] + u1[s + 1][lane]) * __ldg(t.seg_piv + (int64_t)s * modes + mode);
      mid[s][lane] = y;
    }
    for (int s = segs - 3; s >= 0; --s) {
      y = fma(cpl * __ldg(t.seg_piv + (int64_t)s * modes + mode), y, mid[s][lane]);
      mid[s][lane] = y;
    }
  }
  __syncthreads();
  if (!live) return;
  const double gl = seg ? mid[seg - 1][lane] : 0.0, gr = last ? 0.0 : mid[seg][lane];
  if (!last) dst[(int64_t)len_full * t.s_n] = gr;
  double x = gr;
  int i = len - 1;
  for (; i >= 7; i -= 8) {
    double y[8], cc[8], ll[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) y[u] = dst[(int64_t)(i - u) * t.s_n];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      cc[u] = __ldg(ct + (int64_t)(i - u) * modes);
      ll[u] = __ldg(sp + (int64_t)(i - u) * modes);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x = (y[u] + x) * cc[u];
      dst[(int64_t)(i - u) * t.s_n] = fma(ll[u], gl, x);
    }
  }
  for (; i >= 0; --i) {
    x = (dst[(int64_t)i * t.s_n] + x) * __ldg(ct + (int64_t)i * modes);
    dst[(int64_t)i * t.s_n] = fma(__ldg(sp + (int64_t)i * modes), gl, x);
  }
}

// segments per chain: about 24 warps per SM, at least 8 points each; none for many columns, where the
// two-sided elimination's fewer operations count
int chain_segments(int n, int64_t columns) {
  const int64_t want = 24LL * kNumSMs * 32 / std::max<int64_t>(1, columns);
  const int segs = (int)std::min<int64_t>(std::min(kMaxSegs, (n + 1) / 9), want);
  return segs >= 3 ? segs : 0;
}

// ------------------------------------------------------------------------------------------
// Arrays whose sides both exceed 128 faces: the longer side is cut into strips of up to 128 grid lines
// with one grid line (a separator) between neighbours. Per strip the solver above; the separators'
// values g follow from their own equations, which the sine transform along the chains diagonalises:
// for every transverse mode q a tridiagonal system over the separators,
//   (2 + l_q - a_i - a_{i+1}) g_i - c_i g_{i-1} - c_{i+1} g_{i+1} = b_i / kappa + u0_i(last) + u0_{i+1}(first)
// with a_i, c_i the corner entries of the inverse of strip i's tridiag(-1, 2 + l_q, -1) and u0 the
// strips' solutions for zero separators. So: transform the strips, solve the chains, form u0 at the
// strips' edges, transform the separators (a product with the dense sine matrix, jja_block.cuh), solve
// across them, transform back, solve the chains again with the separators' values, transform back.
// ------------------------------------------------------------------------------------------
struct SineStrips {
  int n = 0, seps = 0;                // points a chain, separators
  int64_t s_n = 0, s_x = 0;           // strides along a chain and between grid lines
  const int32_t* sep_x = nullptr;     // grid line of every separator
  double inv_kappa = 0.0;
  const double* piv = nullptr;        // (n x seps): reciprocal pivots per transverse mode
  const double* cpl = nullptr;        // (n x seps): coupling c of strip s + 1 (between separators s and s + 1)
  double* edge = nullptr;             // n x strips x 2 x W: u0 at the first and last line of every strip
  double* rhs = nullptr;              // n x seps x W
  double* hat = nullptr;
  double* g = nullptr;
};

// u0 at the edges of the strips of one width: sums of es[mode] z over odd and even modes. A warp sums a
// (point, strip) over the contiguous modes x problems when the problems divide its lanes or the
// lanes divide the problems; else a block does, problems x slices of the modes. Grid: (points,
// strips, tiles of the problems). The lanes' sums take no branch on the parity: with one, both sides'
// FP64 instructions took the pipe (1024x1024 x 8: 44 -> 30 us).
__global__ void __launch_bounds__(256) k_sine_edges(const double* __restrict__ z, const double* __restrict__ es, int modes,
                                                    int64_t off, int64_t s_strip, int64_t s_n, int64_t s_c, int strip0,
                                                    int strips, int n, int W, double* __restrict__ edge) {
  pdl_begin();
  const int strip = blockIdx.y;
  const bool lanes = 32 % W == 0 || W % 32 == 0;
  if (lanes) {
    const int per = W < 32 ? 32 / W : 1, lane = threadIdx.x & 31;   // modes side by side in a warp
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const int k0 = lane / min(W, 32), w = blockIdx.z * 32 + lane % min(W, 32);
    const double* p = z + off + strip * s_strip + (int64_t)i * s_n + w;
    double odd = 0.0, even = 0.0;
    int k = k0;
    for (; k + 7 * per < modes; k += 8 * per) {
      double v[8], e[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u] = p[(int64_t)(k + u * per) * s_c];
        e[u] = __ldg(es + k + u * per);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u & 1) even = fma(e[u], v[u], even);
        else odd = fma(e[u], v[u], odd);
      }
    }
    for (; k < modes; k += per) {
      const double v = p[(int64_t)k * s_c], e = __ldg(es + k);
      if (per == 1 && (k & 1)) even = fma(e, v, even);
      else odd = fma(e, v, odd);
    }
    if (per > 1) {   // an even number: a lane's modes are all odd or all even, and both sums are one
      const double sum = odd + even;
      odd = k0 & 1 ? 0.0 : sum;
      even = k0 & 1 ? sum : 0.0;
    }
    for (int o = W; o < 32; o <<= 1) {
      odd += __shfl_xor_sync(0xffffffffu, odd, o);
      even += __shfl_xor_sync(0xffffffffu, even, o);
    }
    if (k0 == 0) {
      double* e = edge + (((int64_t)i * strips + strip0 + strip) * 2) * W + w;
      e[0] = odd + even;   // first line
      e[W] = odd - even;   // last line
    }
    return;
  }
  __shared__ double part[2][256];
  const int tw = min(W, 256), slices = 256 / tw, slice = threadIdx.x / tw, w = blockIdx.z * tw + threadIdx.x % tw;
  const int i = blockIdx.x;
  double odd = 0.0, even = 0.0;   // modes 1, 3, ... and 2, 4, ...
  if (slice < slices && w < W) {
    const double* p = z + off + strip * s_strip + (int64_t)i * s_n + w;
#pragma unroll 4
    for (int k = slice; k < modes; k += slices) {
      const double v = p[(int64_t)k * s_c], e = __ldg(es + k);
      if (k & 1) even = fma(e, v, even);
      else odd = fma(e, v, odd);
    }
  }
  part[0][threadIdx.x] = odd;
  part[1][threadIdx.x] = even;
  __syncthreads();
  if (slice == 0 && w < W) {
    for (int k = 1; k < slices; ++k) {
      odd += part[0][k * tw + threadIdx.x];
      even += part[1][k * tw + threadIdx.x];
    }
    double* e = edge + (((int64_t)i * strips + strip0 + strip) * 2) * W + w;
    e[0] = odd + even;
    e[W] = odd - even;
  }
}

// the separators' right-hand sides; the transformed vector is zeroed for the product that follows
__global__ void __launch_bounds__(256) k_sep_rhs(SineStrips S, const double* __restrict__ b, int W, FastDiv by_W) {
  pdl_begin();
  const int64_t n = (int64_t)S.n * S.seps * W;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = by_W(e), w = e - r * W, i = r / S.seps;
    const int s = (int)(r - i * S.seps);
    const double* ed = S.edge + ((i * (S.seps + 1) + s) * 2) * W + w;   // strip s, then strip s + 1
    S.rhs[e] = fma(b[i * S.s_n + (int64_t)__ldg(S.sep_x + s) * S.s_x + w], S.inv_kappa, ed[W] + ed[2 * W]);
    S.hat[e] = 0.0;
  }
}

// across the separators, per transverse mode and problem; zeroes g for the product that follows
__global__ void __launch_bounds__(256) k_sep_solve(SineStrips S, int W, FastDiv by_W) {
  pdl_begin();
  const int64_t n = (int64_t)S.n * W;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = by_W(e), w = e - q * W;
    double* h = S.hat + q * S.seps * W + w;
    double* g = S.g + q * S.seps * W + w;
    const double *piv = S.piv + q * S.seps, *cpl = S.cpl + q * S.seps;
    double y = 0.0;
    for (int s = 0; s < S.seps; ++s) {   // y_s = (r_s + c_s y_{s-1}) / pivot
      y = (s ? fma(__ldg(cpl + s - 1), y, h[(int64_t)s * W]) : h[0]) * __ldg(piv + s);
      h[(int64_t)s * W] = y;
      g[(int64_t)s * W] = 0.0;
    }
    for (int s = S.seps - 2; s >= 0; --s) {
      y = fma(__ldg(cpl + s) * __ldg(piv + s), y, h[(int64_t)s * W]);
      h[(int64_t)s * W] = y;
    }
  }
}

// the separators' values into the solution
__global__ void __launch_bounds__(256) k_sep_store(SineStrips S, double* __restrict__ x, int W, FastDiv by_W) {
  pdl_begin();
  const int64_t n = (int64_t)S.n * S.seps * W;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = by_W(e), w = e - r * W, i = r / S.seps;
    x[i * S.s_n + (int64_t)__ldg(S.sep_x + (int)(r - i * S.seps)) * S.s_x + w] = S.g[e];
  }
}

// digits of the odd and even half matrices scale * sin(pi k j / (m + 1)), |scale| <= 1, in the MMA
// operand layout: half, 8-point group of j, digit, mode, j within the group
std::vector<uint16_t> sine_matrix(int m, int kp, long double scale) {
  const long double pi_l = 3.141592653589793238462643383279502884L;
  const int half = m / 2, groups = kp / 8, N = m + 1;
  std::vector<uint16_t> out((size_t)2 * kMatDigits * kp * kp, 0);
  auto put = [&](int parity, int i, int mode, int j, int digit) {
    const __half h = __float2half((float)digit);
    memcpy(&out[(((size_t)(parity * groups + j / 8) * kMatDigits + i) * kp + mode) * 8 + j % 8], &h, 2);
  };
  for (int parity = 0; parity < 2; ++parity) {
    const int count = parity ? half : m - half;
    for (int a = 0; a < count; ++a)
      for (int j = 0; j < count; ++j) {
        const int k = 2 * a + 1 + parity;
        const long arg = ((long)k * (j + 1)) % (2L * N);   // sin(pi arg / N), reduced to the first quadrant
        const long r = arg % N, f = std::min(r, N - r);
        const long double s = scale * sinl(pi_l * (long double)f / N) * (arg >= N ? -1 : 1);
        int64_t X = (int64_t)llroundl(s * 9007199254740992.0L);   // 2^53
        int64_t t = X;
        for (int i = 0; i < kMatDigits; ++i) t += 256ll << (9 * i);
        for (int i = 0; i < kMatDigits; ++i) {
          const int64_t f9 = t >> (9 * (kMatDigits - 1 - i));
          put(parity, i, a, j, (int)((i ? (f9 & 511) : f9) - 256));
        }
      }
  }
  return out;
}

}  // namespace
