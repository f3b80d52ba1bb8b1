// Whole runs of small circuits in one launch (included by jja_gb300.cu).
//
// A circuit of up to kResMaxFaces faces fits one SM: its state, and the inverse of its face-space
// matrix, stay in shared memory and one block per problem steps all the steps of a call. The
// launch sequence it replaces is 6 launches a step, each a few microseconds of latency for a few
// hundred FP64 operations (SquareArray(10,10): 15.6 us a step replayed from graphs, 40 us when
// every step is stored and the launches are issued one by one).
//
// Measured: 10x10, one problem, 2000 steps with every step stored, 81 -> 11 ms per call, 3.2 us a
// step; 64 problems 24.8 -> 3.2 us, 512 problems 25.7 -> 8.2 us a step (64 registers per thread:
// two blocks per SM; one block measured 12.1).
//
// What bounds a step here is the chain sources -> J -> phases and its five block barriers. The
// product J = K^-1 b is formed in fixed point: GB300's FP64 pipe does 2 operations per clock and
// SM, so the n^2 multiply-adds of one 10x10 array would take 1.7 us; 28-bit halves of 56-bit
// integers multiplied and summed in 64 bits (3 integer multiply-adds per product) take a tenth of
// that. The inverse is refined once on the host (residuals in twice the working precision). With
// 2^e > the largest |K^-1| of the row and 2^f > the largest |b|: the entries of K^-1 are off by at most
// 2^(e-56), b by 2^(f-56), and the product of two lower halves, which is left out, is below 2^(e+f-56), so a
// term is off by at most 3 2^(e+f-56) and usually by a tenth of that. Phase increments against long double,
// error of the Cholesky sweeps' (rms, equal resistances / lognormal spread of 0.4 / of 1): 10x10 0.47 / 0.46 /
// 0.38, 13x13 0.53 / 0.45 / 0.43; with one scale for the whole inverse, not refined, and b cut instead of
// rounded 1.09 / 1.13 / 1.44 and 1.10 / 1.09 / 1.60.

namespace {

constexpr int kResMaxFaces = 160;       // K^-1 in shared memory: 8 bytes x 160^2 = 200 KB
constexpr int kResMaxJunctions = 1024;  // two a thread; the default plan's rule stops at 512
constexpr int kResThreads = 512;
constexpr int kResChunk = 8192;         // steps per launch (26 ms for one 10x10 array, 160 ms for 512 of 13x13)
constexpr int kResHalf = 28;            // bits of the lower half of a fixed-point number

struct ResidentArgs {
  const int2* inv;     // K^-1 by columns, fixed point: (upper, lower half), value = (hi 2^28 + lo) 2^(e - 55)
  const int* e_row;    // per row: e
  int n, nj, nsteps;
  int64_t step0, src_t0;
  const int64_t* th_slots;   // per step: output slot or -1 (null: none; unused with store_all)
  const int64_t* I_slots;
  int64_t slot0;             // store_all: slot of the launch's first step
};

__host__ __device__ inline size_t resident_smem_bytes(int n, int nj, int nh) {
  const int rows = (n + 31) / 32 * 32;
  return (size_t)n * n * sizeof(int2) + ((size_t)(kResThreads / rows) * n * 2 + (nh + 2) * (size_t)nj + 2 * (size_t)n) *
                                            sizeof(double) + 32 * sizeof(uint32_t);
}

// x 2^(55 - E), rounded, in halves of 28 bits, E = emax - 1022 (see fixed_of)
__device__ __forceinline__ int2 resident_halves(double x, int emax) {
  const int64_t v = (fixed_of(x, emax) + (1 << 5)) >> (61 - 55);
  const int lo = (int)((uint32_t)v << (32 - kResHalf)) >> (32 - kResHalf);
  return make_int2((int)((v - lo) >> kResHalf), lo);
}

__global__ void __launch_bounds__(kResThreads, 2) k_resident(StepArgs a, Tables t, ResidentArgs g) {
  extern __shared__ __align__(16) unsigned char res_sh[];
  const int n = g.n, nj = g.nj, nh = a.width - 1, tid = threadIdx.x, w = blockIdx.x;
  const int rows = (n + 31) / 32 * 32, slices = kResThreads / rows, per = (n + slices - 1) / slices;
  int2* inv = reinterpret_cast<int2*>(res_sh);
  int64_t* part = reinterpret_cast<int64_t*>(inv + (size_t)n * n);   // slices x n x (upper, cross)
  double* hist = reinterpret_cast<double*>(part + (size_t)slices * n * 2);
  double* q = hist + (size_t)nh * nj;
  double* ths = q + nj;
  double* J = ths + nj;
  int2* bf = reinterpret_cast<int2*>(J + n);
  uint32_t* wmax = reinterpret_cast<uint32_t*>(bf + n);
  const int64_t NjW = (int64_t)nj * a.W;
  for (int i = tid; i < n * n; i += kResThreads) inv[i] = __ldg(g.inv + i);
  // ring of the phase history: th(t - 1 - k) at slot (newest + k) % nh
  int newest = 0;
  auto old_phase = [&](int k, int j) -> double {
    const int s = newest + k;
    return hist[(s < nh ? s : s - nh) * nj + j];
  };
  for (int j = tid; j < nj; j += kResThreads) {
    const int64_t e = (int64_t)j * a.W + w;
    double th[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      th[k] = k < nh ? a.h[k][e] : 0.0;
      if (k < nh) hist[k * nj + j] = th[k];
    }
    ths[j] = a.theta_s ? a.theta_s[e] : 0.0;
    q[j] = junction_q(a, t, e, j, w, th, g.step0, g.step0 - g.src_t0);
  }
  if (tid < 32) wmax[tid] = 0u;
  __syncthreads();
  const int row = tid % rows, slice = tid / rows;
  const int c_lo = slice * per, c_hi = min(n, c_lo + per);
  const int e_row = tid < n ? __ldg(g.e_row + tid) : 0;
  bool diverged = false;
  for (int i = 0; i < g.nsteps; ++i) {
    const int64_t step = g.step0 + i, tt = step - g.src_t0;
    // b = A (q - theta_s) - 2 pi f, and its largest exponent
    double b = 0.0;
    if (tid < n) {
      if (t.face_deg) {
#pragma unroll
        for (int d = 0; d < kEllMax; ++d) {
          const int code = d < t.face_deg ? __ldg(t.fj_ell + tid * t.face_deg + d) : -1;
          if (code >= 0) {
            const double v = signed_by(a.theta_s ? q[code >> 1] - ths[code >> 1] : q[code >> 1], code & 1);
            b = d ? b + v : v;
          }
        }
      } else {
        const int64_t i0 = __ldg(t.fj_ptr + tid), i1 = __ldg(t.fj_ptr + tid + 1);
        for (int64_t k = i0; k < i1; ++k) {
          const int code = __ldg(t.fj_col + k);
          const double v = signed_by(a.theta_s ? q[code >> 1] - ths[code >> 1] : q[code >> 1], code & 1);
          b = k == i0 ? v : b + v;
        }
      }
      if (a.f.ptr) b = fma(-kTwoPi, view_at(a.f, __ldg(t.face_orig + tid), w, tt), b);
    }
    const uint32_t mag = __reduce_max_sync(0xffffffffu, (uint32_t)__double2hiint(b) * 2u);
    if ((tid & 31) == 0 && tid < rows) wmax[tid >> 5] = mag;
    __syncthreads();
    uint32_t top = 0;
    for (int k = 0; k < rows / 32; ++k) top = max(top, wmax[k]);
    const int emax = max((int)(top >> 21), 64);
    if (tid < n) bf[tid] = resident_halves(b, emax);
    __syncthreads();
    // partial rows of K^-1 b
    if (slice < slices && row < n) {
      int64_t hi = 0, cross = 0;
#pragma unroll 4
      for (int c = c_lo; c < c_hi; ++c) {
        const int2 A = inv[c * n + row], B = bf[c];
        hi += (int64_t)A.x * B.x;
        cross += (int64_t)A.x * B.y;
        cross += (int64_t)A.y * B.x;
      }
      part[(slice * n + row) * 2] = hi;
      part[(slice * n + row) * 2 + 1] = cross;
    }
    __syncthreads();
    if (tid < n) {
      int64_t hi = 0, cross = 0;
      for (int k = 0; k < slices; ++k) {
        hi += part[(k * n + tid) * 2];
        cross += part[(k * n + tid) * 2 + 1];
      }
      const int64_t R = hi + ((cross + (1ll << (kResHalf - 1))) >> kResHalf);   // 2^-54 units
      J[tid] = emax == 0x7ff ? __longlong_as_double((long long)kNaNBits) : double_of_fixed(R, e_row + emax - 1022 - 1);
    }
    __syncthreads();
    const int64_t th_slot = a.store_all ? g.slot0 + i : (g.th_slots ? __ldg(g.th_slots + i) : -1);
    const int64_t I_slot = a.store_all ? g.slot0 + i : (g.I_slots ? __ldg(g.I_slots + i) : -1);
    const int oldest = newest == 0 ? nh - 1 : newest - 1;
    for (int j = tid; j < nj; j += kResThreads) {
      const int64_t e = (int64_t)j * a.W + w;
      const int p0 = __ldg(t.jf_face + 2 * j), p1 = __ldg(t.jf_face + 2 * j + 1);
      double y = p0 >= 0 ? signed_by(J[p0 >> 1], p0 & 1) : 0.0;
      if (p1 >= 0) y += signed_by(J[p1 >> 1], p1 & 1);
      const double th = fma(y, __ldg(t.inv_c0 + j), -q[j]);
      diverged |= non_finite(th);
      if (a.th_out && th_slot >= 0) a.th_out[th_slot * NjW + e] = th;
      if (a.I_out && I_slot >= 0) a.I_out[I_slot * NjW + e] = y + view_at(a.Is, j, w, tt);
      if (a.theta_s && a.Vs.ptr) ths[j] += view_at(a.Vs, j, w, tt) * a.dt;
      if (i + 1 < g.nsteps) {
        double past[4];
        past[0] = th;
#pragma unroll
        for (int k = 1; k < 4; ++k) past[k] = k < nh ? old_phase(k - 1, j) : 0.0;
        q[j] = junction_q(a, t, e, j, w, past, step + 1, tt + 1);
      }
      hist[oldest * nj + j] = th;
    }
    newest = oldest;
    __syncthreads();
  }
  if (diverged) *t.nonfinite = 1;
  for (int j = tid; j < nj; j += kResThreads) {
    const int64_t e = (int64_t)j * a.W + w;
    for (int k = 0; k < nh; ++k) const_cast<double*>(a.h[k])[e] = old_phase(k, j);
    if (a.theta_s && a.Vs.ptr) a.theta_s[e] = ths[j];
  }
}

}  // namespace
