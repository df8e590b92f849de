// CUDA-core sweep kernels and FP64 reductions for the B200 statevector engine (sm_100a).
//
// Layout: the state is Structure-of-Arrays, re[2^n] and im[2^n] in HBM, the layout qsv's
// StateVector uses (crates/qsv-core/src/state/mod.rs:25-29) so `download` is a straight copy.
// Every kernel here is HBM-bound except the dense sweeps of five and six qubits (FP64 pipe); each moves
// whole 32-byte sectors, most of them as 16-byte vectors (4 x f32 or 2 x f64 amplitudes per component), and
// walks the state with a grid-stride loop sized to a multiple of the SM count.
//
// Index math follows qsv's layout helpers (crates/qsv-core/src/state/layout.rs:22-86):
// insert_zero_bit(s) anchors a pair/block, scatter_bits/gather_bits map a gate sub-index to
// state bits (bit j of the sub-index <-> qubits[j]).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <utility>

#include "qsvb_internal.h"

namespace qsvb {

namespace {

constexpr int kThreads = 256;

template <class R> struct VecT;
template <> struct VecT<float> {
  using T = float4;
  using Pair = float2;
  static constexpr int N = 4, LOG = 2;
};
template <> struct VecT<double> {
  using T = double2;
  using Pair = double2;
  static constexpr int N = 2, LOG = 1;
};

template <class R> __device__ __forceinline__ void vld(const R* p, R (&x)[VecT<R>::N]);
template <> __device__ __forceinline__ void vld<float>(const float* p, float (&x)[4]) {
  float4 v = *reinterpret_cast<const float4*>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
template <> __device__ __forceinline__ void vld<double>(const double* p, double (&x)[2]) {
  double2 v = *reinterpret_cast<const double2*>(p);
  x[0] = v.x; x[1] = v.y;
}
template <class R> __device__ __forceinline__ void vst(R* p, const R (&x)[VecT<R>::N]);
template <> __device__ __forceinline__ void vst<float>(float* p, const float (&x)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
template <> __device__ __forceinline__ void vst<double>(double* p, const double (&x)[2]) {
  *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
}

// Work enumerator: work item w -> base index. The low `cb` bits of the base are zero (the chunk
// the item covers), zeros are inserted at the sorted `fixed` positions (all >= cb), and
// `set_mask` is OR'd in (control bits pinned to 1). This is insert_zero_bits (layout.rs:70-86)
// applied to chunks instead of single amplitudes.
struct Enum {
  uint32_t nfixed;
  uint32_t fixed[7];
  uint64_t set_mask;
  uint64_t flip;  // XORed to the work item (LaunchEnv::flip)
};

__device__ __forceinline__ uint64_t enum_base(uint64_t w, uint32_t cb, const Enum& e) {
  uint64_t x = (w ^ e.flip) << cb;
#pragma unroll
  for (uint32_t j = 0; j < 7; ++j) {
    if (j < e.nfixed) {
      const uint32_t b = e.fixed[j];
      const uint64_t lo = x & ((1ull << b) - 1ull);
      x = ((x - lo) << 1) | lo;
    }
  }
  return x | e.set_mask;
}

template <class R> struct M2 {
  R a[8];  // g00 re, im, g01 re, im, g10 re, im, g11 re, im
};

template <class R>
__device__ __forceinline__ void cmac(R& yr, R& yi, R ar, R ai, R xr, R xi) {
  yr = fma(ar, xr, yr);
  yr = fma(-ai, xi, yr);
  yi = fma(ar, xi, yi);
  yi = fma(ai, xr, yi);
}

template <class R>
__device__ __forceinline__ void apply2(const M2<R>& g, R& r0, R& i0, R& r1, R& i1) {
  R y0r = 0, y0i = 0, y1r = 0, y1i = 0;
  cmac(y0r, y0i, g.a[0], g.a[1], r0, i0);
  cmac(y0r, y0i, g.a[2], g.a[3], r1, i1);
  cmac(y1r, y1i, g.a[4], g.a[5], r0, i0);
  cmac(y1r, y1i, g.a[6], g.a[7], r1, i1);
  r0 = y0r; i0 = y0i; r1 = y1r; i1 = y1i;
}

__device__ __forceinline__ uint64_t gtid() { return blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint64_t gstride() { return (uint64_t)gridDim.x * blockDim.x; }

// ---------------------------------------------------------------------------------------------
// 1-qubit / controlled-1-qubit butterflies (qsv kernels.cu:52-70 computes the same 2x2 update
// per pair with scalar 8-byte accesses; here every access is a coalesced 16-byte vector).
// ---------------------------------------------------------------------------------------------

// Target bit inside one 16-byte vector: pairs are formed in registers.
template <class R, int T>
__global__ void __launch_bounds__(kThreads) k_pair_invec(R* __restrict__ re, R* __restrict__ im,
                                                         uint64_t nwork, Enum en, uint32_t ctrl_low,
                                                         M2<R> g) {
  // the target bit T is a template parameter: with a run-time bit the partner index e | 1 << t
  // indexes the register array dynamically, which puts it in local memory
  constexpr int N = VecT<R>::N, LOG = VecT<R>::LOG;
  static_assert(T < LOG, "in-vector target");
  constexpr uint32_t t = T;
  early_next();
  wait_prior();
  for (uint64_t w = gtid(); w < nwork; w += gstride()) {
    const uint64_t b = enum_base(w, LOG, en);
    R xr[N], xi[N];
    vld(re + b, xr);
    vld(im + b, xi);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      if (((e >> t) & 1) == 0 && (uint32_t(e) & ctrl_low) == ctrl_low) {
        const int f = e | (1 << t);
        apply2(g, xr[e], xi[e], xr[f], xi[f]);
      }
    }
    vst(re + b, xr);
    vst(im + b, xi);
  }
}

// Target bit within one warp's 32 contiguous vectors: each lane loads its own vector (the warp
// reads 512 contiguous bytes per component) and fetches its partner with a warp shuffle, so
// every HBM sector is read and written exactly once.
template <class R>
__global__ void __launch_bounds__(kThreads) k_pair_shfl(R* __restrict__ re, R* __restrict__ im,
                                                        uint64_t nwork, Enum en, uint32_t t,
                                                        uint32_t ctrl_low, M2<R> g) {
  constexpr int N = VecT<R>::N, LOG = VecT<R>::LOG;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lanemask = 1u << (t - LOG);
  const bool upper = (lane & lanemask) != 0;
  early_next();
  wait_prior();
  const uint64_t nwarps = gstride() >> 5;
  for (uint64_t w = gtid() >> 5; w < nwork; w += nwarps) {
    const uint64_t b = enum_base(w, LOG + 5, en) + uint64_t(lane) * N;
    R xr[N], xi[N];
    vld(re + b, xr);
    vld(im + b, xi);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const R pr = __shfl_xor_sync(0xffffffffu, xr[e], lanemask);
      const R pi = __shfl_xor_sync(0xffffffffu, xi[e], lanemask);
      if (((lane * N + e) & ctrl_low) == ctrl_low) {
        R yr = 0, yi = 0;
        if (upper) {  // this lane holds |1>: y = g10 x0 + g11 x1
          cmac(yr, yi, g.a[4], g.a[5], pr, pi);
          cmac(yr, yi, g.a[6], g.a[7], xr[e], xi[e]);
        } else {      // y = g00 x0 + g01 x1
          cmac(yr, yi, g.a[0], g.a[1], xr[e], xi[e]);
          cmac(yr, yi, g.a[2], g.a[3], pr, pi);
        }
        xr[e] = yr;
        xi[e] = yi;
      }
    }
    vst(re + b, xr);
    vst(im + b, xi);
  }
}

// Target bit above one warp's span: each thread owns a vector pair 2^t apart; a warp's 32 lanes
// still read 512 contiguous bytes per access.
template <class R>
__global__ void __launch_bounds__(kThreads) k_pair_strided(R* __restrict__ re, R* __restrict__ im,
                                                           uint64_t nwork, Enum en, uint32_t t,
                                                           uint32_t ctrl_low, M2<R> g) {
  constexpr int N = VecT<R>::N, LOG = VecT<R>::LOG;
  const uint64_t half = 1ull << t;
  early_next();
  wait_prior();
  for (uint64_t w = gtid(); w < nwork; w += gstride()) {
    const uint64_t b = enum_base(w, LOG, en);
    R r0[N], i0[N], r1[N], i1[N];
    vld(re + b, r0);
    vld(im + b, i0);
    vld(re + b + half, r1);
    vld(im + b + half, i1);
#pragma unroll
    for (int e = 0; e < N; ++e)
      if ((uint32_t(e) & ctrl_low) == ctrl_low) apply2(g, r0[e], i0[e], r1[e], i1[e]);
    vst(re + b, r0);
    vst(im + b, i0);
    vst(re + b + half, r1);
    vst(im + b + half, i1);
  }
}

// Scalar fallback for tiny states: one pair per thread (fixed = sorted {t} U controls).
template <class R>
__global__ void k_pair_scalar(R* __restrict__ re, R* __restrict__ im, uint64_t nwork, Enum en,
                              uint32_t t, M2<R> g) {
  early_next();
  wait_prior();
  for (uint64_t w = gtid(); w < nwork; w += gstride()) {
    const uint64_t a0 = enum_base(w, 0, en), a1 = a0 | (1ull << t);
    R r0 = re[a0], i0 = im[a0], r1 = re[a1], i1 = im[a1];
    apply2(g, r0, i0, r1, i1);
    re[a0] = r0; im[a0] = i0; re[a1] = r1; im[a1] = i1;
  }
}

// ---------------------------------------------------------------------------------------------
// Diagonal sweep: psi_i *= d[gather_bits(i, qs)] (qsv kernels.cu:73-85 / cpu.rs:100-146). The
// table lives in shared memory; qubits whose 0-half is the identity are pinned to 1 by the
// enumerator so those amplitudes are never touched (CZ / CPHASE touch a quarter of the state).
// ---------------------------------------------------------------------------------------------
template <class R> struct DiagP {
  uint32_t m;
  uint32_t q[6];
  R d[128];  // interleaved (re, im), 2^m entries
};

template <class R>
__global__ void __launch_bounds__(kThreads) k_diag(R* __restrict__ re, R* __restrict__ im,
                                                   uint64_t nwork, Enum en, DiagP<R> p) {
  constexpr int N = VecT<R>::N, LOG = VecT<R>::LOG;
  __shared__ R tab[128];
  for (int i = threadIdx.x; i < (2 << p.m); i += blockDim.x) tab[i] = p.d[i];
  __syncthreads();
  uint32_t lowsub[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    uint32_t s = 0;
    for (uint32_t j = 0; j < p.m; ++j)
      if (p.q[j] < uint32_t(LOG)) s |= ((uint32_t(e) >> p.q[j]) & 1u) << j;
    lowsub[e] = s;
  }
  early_next();
  wait_prior();
  for (uint64_t w = gtid(); w < nwork; w += gstride()) {
    const uint64_t b = enum_base(w, LOG, en);
    uint32_t shi = 0;
    for (uint32_t j = 0; j < p.m; ++j) shi |= uint32_t((b >> p.q[j]) & 1ull) << j;
    R xr[N], xi[N];
    vld(re + b, xr);
    vld(im + b, xi);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const uint32_t s = shi | lowsub[e];
      const R dr = tab[2 * s], di = tab[2 * s + 1];
      const R a = xr[e], c = xi[e];
      xr[e] = fma(dr, a, -di * c);
      xi[e] = fma(dr, c, di * a);
    }
    vst(re + b, xr);
    vst(im + b, xi);
  }
}

template <class R>
__global__ void k_diag_scalar(R* __restrict__ re, R* __restrict__ im, uint64_t dim, DiagP<R> p) {
  early_next();
  wait_prior();
  for (uint64_t i = gtid(); i < dim; i += gstride()) {
    uint32_t s = 0;
    for (uint32_t j = 0; j < p.m; ++j) s |= uint32_t((i >> p.q[j]) & 1ull) << j;
    const R dr = p.d[2 * s], di = p.d[2 * s + 1];
    const R a = re[i], c = im[i];
    re[i] = fma(dr, a, -di * c);
    im[i] = fma(dr, c, di * a);
  }
}

// ---------------------------------------------------------------------------------------------
// Phase-polynomial sweep: psi_i *= exp(i * sum_t ang_t[gather_bits(i, q_t)]) over many <= 2-qubit
// diagonal terms (a whole QAOA cost layer of RZZ gates in one pass). The phase is summed and
// evaluated in FP64 for both precisions.
// ---------------------------------------------------------------------------------------------
struct PhaseTermDev {
  uint32_t q0, q1;  // q1 == 64 for a 1-qubit term
  double ang[4];
};

template <class R>
__global__ void __launch_bounds__(kThreads) k_phase(R* __restrict__ re, R* __restrict__ im,
                                                    uint64_t dim, const PhaseTermDev* __restrict__ terms,
                                                    uint32_t nterms) {
  extern __shared__ char smem_raw[];
  PhaseTermDev* st = reinterpret_cast<PhaseTermDev*>(smem_raw);
  for (uint32_t i = threadIdx.x; i < nterms; i += blockDim.x) st[i] = terms[i];
  __syncthreads();
  constexpr int N = VecT<R>::N;
  const uint64_t nvec = dim / N;
  for (uint64_t w = gtid(); w < nvec; w += gstride()) {
    const uint64_t b = w * N;
    R xr[N], xi[N];
    vld(re + b, xr);
    vld(im + b, xi);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const uint64_t i = b + e;
      double th = 0.0;
      for (uint32_t k = 0; k < nterms; ++k) {
        const PhaseTermDev& T = st[k];
        const uint32_t s = uint32_t((i >> T.q0) & 1ull) | (T.q1 < 64 ? uint32_t((i >> T.q1) & 1ull) << 1 : 0u);
        th += T.ang[s];
      }
      double sn, cs;
      sincos(th, &sn, &cs);
      const double a = double(xr[e]), c = double(xi[e]);
      xr[e] = R(cs * a - sn * c);
      xi[e] = R(cs * c + sn * a);
    }
    vst(re + b, xr);
    vst(im + b, xi);
  }
}

// Phase polynomial in Ising form for states of >= 12 qubits. Any product of <= 2-qubit diagonal
// phases is exp(i theta(x)) with theta = C + sum_q h_q z_q + sum_(a<b) J_ab z_a z_b, z_q = 1 - 2 x_q.
// A CTA walks chunks of 4096 consecutive amplitudes. The edge terms inside the low 12 bits are
// tabulated once per CTA; per chunk, the high bits are constant, so the high-high terms fold into one
// scalar and the high-low edges into the linear coefficients of the low bits, kept as two 64-entry
// tables. All three tables hold unit complex factors exp(i angle) (the chunk scalar folded into the
// first 64-entry one), so an amplitude's factor is a product of three shared loads: two complex
// multiplies in FP64 instead of one sincos per amplitude. The low-bit table is 64 KB of dynamic
// shared memory.
constexpr int kIsingMaxEdges = 160;
constexpr int kIsingChunkBits = 12;
struct IsingP {
  double c0;
  double h[64];
  double J[kIsingMaxEdges];
  uint8_t ea[kIsingMaxEdges], eb[kIsingMaxEdges];  // ea < eb
  uint32_t nedges;
};

__device__ __forceinline__ double zsign(uint64_t x, uint32_t q) { return 1.0 - 2.0 * double((x >> q) & 1ull); }

template <class R>
__global__ void __launch_bounds__(kThreads) k_ising(R* __restrict__ re, R* __restrict__ im, uint64_t nchunks,
                                                    IsingP p) {
  constexpr int CB = kIsingChunkBits, CH = 1 << CB, N = VecT<R>::N;
  extern __shared__ double2 tll[];  // CH entries: (cos, sin) of the low-bit edge phases
  __shared__ double2 l1[64], l2[64];
  __shared__ double hp[CB];
  __shared__ double thh;
  const int tid = threadIdx.x;
  for (int l = tid; l < CH; l += kThreads) {
    double s = 0.0;
    for (uint32_t e = 0; e < p.nedges; ++e)
      if (p.eb[e] < CB) s += p.J[e] * zsign(uint64_t(l), p.ea[e]) * zsign(uint64_t(l), p.eb[e]);
    double sn, cs;
    sincos(s, &sn, &cs);
    tll[l] = make_double2(cs, sn);
  }
  for (uint64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    const uint64_t base = ch << CB;
    __syncthreads();  // the previous chunk is done with l1 / l2 / thh (and tll is built)
    if (tid < CB) {
      double v = p.h[tid];
      for (uint32_t e = 0; e < p.nedges; ++e)
        if (p.ea[e] == uint32_t(tid) && p.eb[e] >= CB) v += p.J[e] * zsign(base, p.eb[e]);
      hp[tid] = v;
    } else if (tid == 32) {
      double v = p.c0;
      for (uint32_t q = CB; q < 64; ++q)
        if (p.h[q] != 0.0) v += p.h[q] * zsign(base, q);
      for (uint32_t e = 0; e < p.nedges; ++e)
        if (p.ea[e] >= CB) v += p.J[e] * zsign(base, p.ea[e]) * zsign(base, p.eb[e]);
      thh = v;
    }
    __syncthreads();
    if (tid < 64) {
      double v = thh;
      for (int q = 0; q < 6; ++q) v += hp[q] * zsign(uint64_t(tid), q);
      double sn, cs;
      sincos(v, &sn, &cs);
      l1[tid] = make_double2(cs, sn);
    } else if (tid < 128) {
      double v = 0.0;
      for (int q = 0; q < 6; ++q) v += hp[6 + q] * zsign(uint64_t(tid - 64), q);
      double sn, cs;
      sincos(v, &sn, &cs);
      l2[tid - 64] = make_double2(cs, sn);
    }
    __syncthreads();
    for (int v = tid; v < CH / N; v += kThreads) {
      const uint32_t l = uint32_t(v * N);
      R xr[N], xi[N];
      vld(re + base + l, xr);
      vld(im + base + l, xi);
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const uint32_t x = l + e;
        const double2 f0 = tll[x], f1 = l1[x & 63u], f2 = l2[x >> 6];
        const double ur = f0.x * f1.x - f0.y * f1.y, ui = f0.x * f1.y + f0.y * f1.x;
        const double cs = ur * f2.x - ui * f2.y, sn = ur * f2.y + ui * f2.x;
        const double a = double(xr[e]), c = double(xi[e]);
        xr[e] = R(cs * a - sn * c);
        xi[e] = R(cs * c + sn * a);
      }
      vst(re + base + l, xr);
      vst(im + base + l, xi);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Dense k-qubit sweep (qsv kernels.cu:91-120 gathers one 2^m block per thread into local arrays).
// Matrices are packed row-major, interleaved (re, im) in the state's precision; the classifier lists a
// dense gate's qubits in ascending order. Two kernels; launch_dense_of states which one runs where.
// Either can multiply its result by a diagonal sweep's factors before the write-back (`Tail`, chosen
// by attach_diagonals), which saves that sweep's own read and write of the state.
// ---------------------------------------------------------------------------------------------

// Dense sweep on the FP64 matrix instruction (mma.m8n8k4), no shared-memory staging of the state. A
// warp owns G groups of 8 columns (the lowest non-gate bits) and computes Y^T = X^T W^T with the real
// 2M x 2M form W = [[Ur, -Ui], [Ui, Ur]] (M = 2^K): the 8 columns are the instruction's rows, the K
// index of one instruction is the value of the gate's two lowest state bits, and its 8 result columns
// are those two bits and (re, im). So lane (column, low gate bits) loads, and later stores, exactly
// its own amplitudes: the accumulator pair of a lane is (re, im) of one of them. A complex128 load or
// store instruction touches whole 32-byte sectors wherever the gate bits lie, because state bits 0
// and 1 are always among its 3 column bits and 2 low gate bits. All loads of the warp's 2^K x 8G
// amplitudes are in flight before the first product, warps never wait for one another, and each
// matrix fragment (16 bytes of shared memory a lane) feeds 2 G products. complex64 amplitudes are
// widened on load and rounded once on store.
//   The scalar tile it replaces was bound by its operands: every FP64 FMA pair needed a broadcast
// coefficient from shared memory, and tile, product and write-back were separated by block barriers.
// Bound now: HBM for K <= 4, the FP64 pipe (37 TFLOP/s measured) for K = 5, 6. Measured on 27-qubit
// complex128 states (4.3 GB moved), mean over low, middle and high gate bits, before -> after:
//   K = 2: 0.87 -> 0.68 ms, K = 3: 0.94 -> 0.70 ms, K = 4: 1.39 -> 0.75 ms (5.7 TB/s),
//   K = 5: 2.26 -> 1.20 ms (28.5 TFLOP/s), K = 6: 3.85 -> 2.02 ms (34 TFLOP/s).
//
// Tail: the diagonal D applied after the dense product, in the order and the rounding of a separate
// diagonal sweep (the product rounded to R, then one complex multiply in R), so results are the same
// bit for bit. Bits of the sub-index that must be 1 for D to act (`need`) are honoured per amplitude.
// Cost at 27 qubits: K = 2, 3 within 0.03 ms of the plain sweep; K = 4 complex64 0.37 -> 0.49 ms and
// complex128 0.72 -> 0.91 ms, against 0.36 and 0.73 ms for the diagonal sweep that it replaces.
template <class R> struct Tail {
  uint32_t q[6];  // state bit of each sub-index bit (63: unused)
  uint32_t need;
  uint32_t m;
  // sub-index bits that an offset brings in, so that a thread extracts them from its address once:
  // the gate's bits (in the kernel's order), and the group bits (k_dense_mma) or extra columns and
  // vector elements (k_dense_cols)
  uint32_t gate[6], grp[3], ext[2], elem[2];
  uint32_t neg;  // kTailSign: bit x is set where entry x is -1
  R d[128];      // interleaved (re, im), 2^m entries
};
// How a kernel applies its tail: none; by the table; or by flipping signs, where every entry is 1 or -1 and
// m <= 5 (layers of CZ): no table look-up and no multiplication (27 qubits, K = 4, gate bits 10..13:
// complex64 0.50 -> 0.40 ms, complex128 0.91 -> 0.79 ms).
constexpr int kTailNone = 0, kTailTable = 1, kTailSign = 2;

template <class R> __device__ __forceinline__ uint32_t tail_index(const Tail<R>& t, uint64_t a) {
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < 6; ++j) s |= uint32_t((a >> t.q[j]) & 1ull) << j;
  return s;
}

__device__ __forceinline__ float flip_sign(float x, uint32_t sign) { return __uint_as_float(__float_as_uint(x) ^ sign); }
__device__ __forceinline__ double flip_sign(double x, uint32_t sign) {
  return __hiloint2double(__double2hiint(x) ^ int(sign), __double2loint(x));
}

template <int TAIL, class R, class R2>
__device__ __forceinline__ void tail_apply(const R2* tab, const Tail<R>& t, uint32_t sub, R& xr, R& xi) {
  if constexpr (TAIL == kTailSign) {
    const uint32_t sign = (t.neg >> sub) << 31;
    xr = flip_sign(xr, sign);
    xi = flip_sign(xi, sign);
    return;
  }
  const uint32_t need = t.need;
  const R2 d = tab[sub];
  const R a = xr, c = xi;
  const bool acts = (sub & need) == need;  // (selected, not branched on)
  xr = acts ? fma(d.x, a, -d.y * c) : a;
  xi = acts ? fma(d.x, c, d.y * a) : c;
}

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

struct NoTail {};
template <class R, int TAIL> using TailIf = std::conditional_t<TAIL != kTailNone, Tail<R>, NoTail>;

struct DenseMmaP {
  uint64_t bit[6];  // address of the gate bits, ascending
  uint64_t grp[3];  // address of the column bits that number a warp's groups
  uint64_t flip;    // XORed to the item (LaunchEnv::flip)
};

template <class R, int K, int G, int TH, int MINB, int TAIL>
__global__ void __launch_bounds__(TH, MINB) k_dense_mma(R* __restrict__ re, R* __restrict__ im, uint64_t nitems,
                                                        const R* __restrict__ u, DenseMmaP p,
                                                        const __grid_constant__ TailIf<R, TAIL> t) {
  constexpr int M = 1 << K, H = M / 4;  // H: values of the gate bits above the two lowest
  early_next();
  extern __shared__ __align__(16) char smem_raw[];
  // fragment (r >> 2, s >> 2): lane 8 (r & 3) + 4 part + (s & 3) holds the two values that multiply the
  // real and the imaginary part of column s for the real (part 0) or imaginary part of row r
  double2* ws = reinterpret_cast<double2*>(smem_raw);
  for (int i = threadIdx.x; i < H * H * 32; i += TH) {
    const int f = i >> 5, r = (f / H) * 4 + ((i >> 3) & 3), s = (f % H) * 4 + (i & 3);
    const double ar = u[2 * (r * M + s)], ai = u[2 * (r * M + s) + 1];
    ws[i] = (i & 4) ? make_double2(ai, ar) : make_double2(ar, -ai);
  }
  __shared__ __align__(16) typename VecT<R>::Pair tab[TAIL == kTailTable ? 64 : 1];
  if constexpr (TAIL == kTailTable)
    for (int i = threadIdx.x; i < (1 << t.m); i += TH) tab[i] = {t.d[2 * i], t.d[2 * i + 1]};
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t low = ((lane & 1u) ? p.bit[0] : 0ull) + ((lane & 2u) ? p.bit[1] : 0ull);
  auto row = [&](int h) {  // address offset of the higher gate bits' value h
    uint64_t o = 0;
#pragma unroll
    for (int j = 2; j < K; ++j)
      if ((h >> (j - 2)) & 1) o += p.bit[j];
    return o;
  };
  auto group = [&](int g) {
    uint64_t o = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if ((g >> j) & 1) o += p.grp[j];
    return o;
  };
  wait_prior();
  const uint64_t nwarps = uint64_t(gridDim.x) * (TH / 32);
#pragma unroll 1
  for (uint64_t w = blockIdx.x * uint64_t(TH / 32) + (threadIdx.x >> 5); w < nitems; w += nwarps) {
    uint64_t base = (w ^ p.flip) * (G * 8) + (lane >> 2);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint64_t lo = base & (p.bit[j] - 1ull);
      base = ((base - lo) << 1) | lo;
    }
    // (the group bits lie between the columns' and w's, so they are zero in it)
    base += low;
    uint32_t tsub = 0;  // tail sub-index of this lane's row 0 in group 0
    if constexpr (TAIL) tsub = tail_index(t, base);
    R x[G][2 * H];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        x[g][2 * h] = re[base + group(g) + row(h)];
        x[g][2 * h + 1] = im[base + group(g) + row(h)];
      }
#pragma unroll
    for (int r = 0; r < H; ++r) {
      double y[G][2];
#pragma unroll
      for (int g = 0; g < G; ++g) y[g][0] = y[g][1] = 0.0;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const double2 b = ws[(r * H + h) * 32 + lane];
#pragma unroll
        for (int g = 0; g < G; ++g) {
          mma_f64(y[g], double(x[g][2 * h]), b.x);
          mma_f64(y[g], double(x[g][2 * h + 1]), b.y);
        }
      }
      // in place: a lane stores only addresses that it has loaded itself
#pragma unroll
      for (int g = 0; g < G; ++g) {
        R yr = R(y[g][0]), yi = R(y[g][1]);
        if constexpr (TAIL) {
          uint32_t sub = tsub;
#pragma unroll
          for (int j = 2; j < K; ++j)
            if ((r >> (j - 2)) & 1) sub |= t.gate[j];
#pragma unroll
          for (int j = 0; j < 3; ++j)
            if ((g >> j) & 1) sub |= t.grp[j];
          tail_apply<TAIL>(tab, t, sub, yr, yi);
        }
        re[base + group(g) + row(r)] = yr;
        im[base + group(g) + row(r)] = yi;
      }
    }
  }
}

// complex64 dense sweep of K = 2..4 on paired FP32 FMAs, large states. A thread holds the 2^K rows of 4
// columns in registers and walks the matrix two or more rows a step: one broadcast coefficient from
// shared memory feeds 8 paired FMAs. Loads and stores are 16-byte vectors (state bits 0 and 1 are
// always in the thread: L0 / L1 say which of them are gate bits; as many further column bits, `ext`,
// above the lanes then make up the 4 columns). The lanes are the lowest remaining bits. Where state
// bit 2 is a gate bit (L2) a lane's vectors would be half sectors 32 bytes apart, so a lane pair loads
// whole sectors, trading bit 2 against the lowest lane bit, and swaps back with shuffles.
//   Before, each product of the shared-memory tile needed one operand from shared memory for every
// two FMAs and three block barriers a tile. Bound now: HBM (K = 2, 3); FP32 FMA issue together with
// HBM (K = 4: 240 of 380 us are FMA issue). Measured on 27-qubit states (2.1 GB moved), mean over low,
// middle and high gate bits, before -> after: K = 2: 0.50 -> 0.35 ms, K = 3: 0.59 -> 0.37 ms,
// K = 4: 0.77 -> 0.43 ms (0.58 -> 0.39 ms with the gate bits above bit 6).
struct DenseColP {
  uint32_t ins[6], nins;  // the register bits (gate bits and state bits 0, 1), ascending
  uint32_t zero;          // 0: see `fresh`
  uint64_t hi[4];         // address of the gate bits that are not in the vector
  uint64_t ext[2];        // address of the extra column bits
  uint64_t flip;          // XORed to the item (LaunchEnv::flip)
};

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int K, int L0, int L1, int L2, int TH, int TAIL>
__global__ void __launch_bounds__(TH, 1) k_dense_cols(float* __restrict__ re, float* __restrict__ im, uint64_t nitems,
                                                      const float2* __restrict__ u, const __grid_constant__ DenseColP p,
                                                      const __grid_constant__ TailIf<float, TAIL> t) {
  constexpr int M = 1 << K, NL = L0 + L1, NH = K - NL, VH = 1 << NH, NX = 1 << NL, RV = 1 << NL;
  constexpr int VB = (L2 || (K == 4 && NL == 0)) ? 2 : 1;  // vectors (groups of RV rows) a step
  constexpr int RB = RV * VB;
  early_next();
  __shared__ __align__(16) float2 us[M * M];
  for (int i = threadIdx.x; i < M * M; i += TH) us[i] = u[i];
  __shared__ __align__(16) float2 tab[TAIL == kTailTable ? 64 : 1];
  if constexpr (TAIL == kTailTable)
    for (int i = threadIdx.x; i < (1 << t.m); i += TH) tab[i] = make_float2(t.d[2 * i], t.d[2 * i + 1]);
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  auto insert = [&](uint64_t x) {
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (j < int(p.nins)) {
        const uint64_t lo = x & ((1ull << p.ins[j]) - 1ull);
        x = ((x - lo) << 1) | lo;
      }
    return x;
  };
  const bool up = L2 && (lane & 1u);
  const uint64_t lane_bit = insert(1);  // state bit of the lowest lane bit
  const uint64_t lane_off = L2 ? insert(lane & ~1u) + (up ? p.hi[0] : 0ull) : insert(lane);
  // register bit 0 of the higher rows: with L2 it walks the lane bit's two columns in memory
  const uint64_t first = L2 ? lane_bit : p.hi[0];
  auto ext = [&](int x) { return ((x & 1) ? p.ext[0] : 0ull) + ((x & 2) ? p.ext[1] : 0ull); };
  // vector element e of vector (row group, x): its row within the group and its column
  auto elem_row = [](int e) { return L0 && L1 ? e : L0 ? (e & 1) : L1 ? (e >> 1) : 0; };
  auto elem_col = [](int e, int x) { return L0 && L1 ? x : L0 ? ((e >> 1) | (x << 1)) : L1 ? ((e & 1) | (x << 1)) : e; };
  auto swap = [&](float& v0, float& v1) {  // lane pair: v0 <-> the other lane's v1 crosswise
    const float got = __shfl_xor_sync(0xffffffffu, up ? v0 : v1, 1);
    if (up) v0 = got;
    else v1 = got;
  };
  // Column pairs that are not adjacent in a loaded vector (L0) move to their register pair once, here:
  // without an operation of its own the assembler repeats the moves in every step (K = 4: 0.60 against
  // 0.46 ms).
  auto fresh = [&](float v) { return L0 && !L2 ? __uint_as_float(__float_as_uint(v) ^ p.zero) : v; };
  wait_prior();
  const uint64_t nwarps = uint64_t(gridDim.x) * (TH / 32);
#pragma unroll 1
  for (uint64_t w = blockIdx.x * uint64_t(TH / 32) + (threadIdx.x >> 5); w < nitems; w += nwarps) {
    const uint64_t base = insert((w ^ p.flip) << (5 + NL)) + lane_off;
    asm volatile("" ::: "memory");  // the matrix stays in shared memory (hoisted, it would spill)
    uint32_t tsub = 0;  // tail sub-index of the thread's first amplitude
    if constexpr (TAIL) tsub = tail_index(t, base);
    float xr[M][4], xi[M][4];
#pragma unroll
    for (int v = 0; v < VH; ++v)
#pragma unroll
      for (int x = 0; x < NX; ++x) {
        uint64_t a = base + ext(x) + ((v & 1) ? first : 0ull);
#pragma unroll
        for (int j = 1; j < NH; ++j)
          if ((v >> j) & 1) a += p.hi[j];
        float fr[4], fi[4];
        vld(re + a, fr);
        vld(im + a, fi);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          xr[(v << NL) | elem_row(e)][elem_col(e, x)] = fr[e];
          xi[(v << NL) | elem_row(e)][elem_col(e, x)] = fi[e];
        }
      }
    if constexpr (L2) {
#pragma unroll
      for (int r = 0; r < M; ++r)
        if (!((r >> NL) & 1))
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            swap(xr[r][c], xr[r | RV][c]);
            swap(xi[r][c], xi[r | RV][c]);
          }
    }
    f32x2 pr[M][2], pi[M][2];
#pragma unroll
    for (int s = 0; s < M; ++s)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        pr[s][c] = pack2(fresh(xr[s][2 * c]), fresh(xr[s][2 * c + 1]));
        pi[s][c] = pack2(fresh(xi[s][2 * c]), fresh(xi[s][2 * c + 1]));
      }
#pragma unroll 1
    for (int v0 = 0; v0 < VH; v0 += VB) {
      f32x2 rr[RB][2], ii[RB][2], ri[RB][2];  // sums of ar xr, ai xi, ar xi + ai xr
#pragma unroll
      for (int q = 0; q < RB; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c) rr[q][c] = ii[q][c] = ri[q][c] = 0ull;
      const float2* um = us + (v0 << NL) * M;
#pragma unroll
      for (int s = 0; s < M; ++s)
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          const float2 g = um[q * M + s];
          const f32x2 ar = pack2(g.x, g.x), ai = pack2(g.y, g.y);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            fma2(rr[q][c], ar, pr[s][c]);
            fma2(ii[q][c], ai, pi[s][c]);
            fma2(ri[q][c], ar, pi[s][c]);
            fma2(ri[q][c], ai, pr[s][c]);
          }
        }
      float yr[RB][4], yi[RB][4];
#pragma unroll
      for (int q = 0; q < RB; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float2 a = unpack2(rr[q][c]), b = unpack2(ii[q][c]), d = unpack2(ri[q][c]);
          yr[q][2 * c] = a.x - b.x;
          yr[q][2 * c + 1] = a.y - b.y;
          yi[q][2 * c] = d.x;
          yi[q][2 * c + 1] = d.y;
        }
      if constexpr (L2) {
#pragma unroll
        for (int q = 0; q < RV; ++q)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            swap(yr[q][c], yr[q + RV][c]);
            swap(yi[q][c], yi[q + RV][c]);
          }
      }
      uint64_t group = 0;  // address of this step's first row group
      if (VB == 1 && (v0 & 1)) group += first;
#pragma unroll
      for (int j = 1; j < NH; ++j)
        if ((v0 >> j) & 1) group += p.hi[j];
      uint32_t gsub = tsub;
      if constexpr (TAIL) {
#pragma unroll
        for (int j = 0; j < NH; ++j)
          if ((v0 >> j) & 1) gsub |= t.gate[j];
      }
      // in place: a thread stores only the vectors that it has loaded itself
#pragma unroll
      for (int v = 0; v < VB; ++v)
#pragma unroll
        for (int x = 0; x < NX; ++x) {
          const uint64_t a = base + ext(x) + group + (v ? first : 0ull);
          float fr[4], fi[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            fr[e] = yr[v * RV + elem_row(e)][elem_col(e, x)];
            fi[e] = yi[v * RV + elem_row(e)][elem_col(e, x)];
            if constexpr (TAIL)
              tail_apply<TAIL>(tab, t, gsub | (v ? t.gate[0] : 0u) | ((x & 1) ? t.ext[0] : 0u) |
                         ((x & 2) ? t.ext[1] : 0u) | ((e & 1) ? t.elem[0] : 0u) | ((e & 2) ? t.elem[1] : 0u), fr[e], fi[e]);
          }
          vst(re + a, fr);
          vst(im + a, fi);
        }
    }
  }
}

// Small-state fallback: one 2^K block per thread (gather, matvec, scatter).
template <class R, int K>
__global__ void k_dense_small(R* __restrict__ re, R* __restrict__ im, uint64_t nblocks,
                              const R* __restrict__ ut, Enum en, uint32_t q0, uint32_t q1,
                              uint32_t q2, uint32_t q3, uint32_t q4, uint32_t q5) {
  constexpr int M = 1 << K;
  const uint32_t qs[6] = {q0, q1, q2, q3, q4, q5};
  early_next();
  wait_prior();
  for (uint64_t w = gtid(); w < nblocks; w += gstride()) {
    const uint64_t base = enum_base(w, 0, en);
    R xr[M], xi[M];
#pragma unroll
    for (int s = 0; s < M; ++s) {
      uint64_t idx = base;
#pragma unroll
      for (int j = 0; j < K; ++j) idx |= uint64_t((s >> j) & 1) << qs[j];
      xr[s] = re[idx];
      xi[s] = im[idx];
    }
#pragma unroll 1
    for (int r = 0; r < M; ++r) {
      R yr = 0, yi = 0;
#pragma unroll
      for (int s = 0; s < M; ++s) cmac(yr, yi, ut[2 * (r * M + s)], ut[2 * (r * M + s) + 1], xr[s], xi[s]);
      uint64_t idx = base;
#pragma unroll
      for (int j = 0; j < K; ++j) idx |= uint64_t((r >> j) & 1) << qs[j];
      re[idx] = yr;
      im[idx] = yi;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// State preparation
// ---------------------------------------------------------------------------------------------
// |basis>: one kernel for what were two memsets and a kernel of one thread.
template <class R>
__global__ void __launch_bounds__(kThreads) k_init_basis(R* __restrict__ re, R* __restrict__ im, uint64_t dim,
                                                         uint64_t basis) {
  constexpr int N = VecT<R>::N;
  early_next();
  wait_prior();
  if (dim % N == 0) {
    for (uint64_t w = gtid(); w < dim / N; w += gstride()) {
      R x[N] = {}, z[N] = {};
#pragma unroll
      for (int e = 0; e < N; ++e)
        if (w * N + e == basis) x[e] = R(1);
      vst(re + w * N, x);
      vst(im + w * N, z);
    }
  } else {
    for (uint64_t i = gtid(); i < dim; i += gstride()) {
      re[i] = i == basis ? R(1) : R(0);
      im[i] = R(0);
    }
  }
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Counter-based complex Gaussian: two SplitMix64 outputs of (seed, index) -> Box-Muller.
template <class R>
__global__ void k_gaussian(R* __restrict__ re, R* __restrict__ im, uint64_t dim, uint64_t seed) {
  const uint64_t G = 0x9E3779B97F4A7C15ull;
  for (uint64_t i = gtid(); i < dim; i += gstride()) {
    const uint64_t h1 = mix64(seed + (2 * i + 1) * G), h2 = mix64(seed + (2 * i + 2) * G);
    const double u1 = double((h1 >> 11) + 1) * 0x1.0p-53;  // (0, 1]
    const double u2 = double(h2 >> 11) * 0x1.0p-53;        // [0, 1)
    const double r = sqrt(-2.0 * log(u1));
    double sn, cs;
    sincospi(2.0 * u2, &sn, &cs);
    re[i] = R(r * cs);
    im[i] = R(r * sn);
  }
}

template <class R>
__global__ void k_scale(R* __restrict__ re, R* __restrict__ im, uint64_t dim, const double* d_norm) {
  const double inv = 1.0 / sqrt(d_norm[0]);
  for (uint64_t i = gtid(); i < dim; i += gstride()) {
    re[i] = R(double(re[i]) * inv);
    im[i] = R(double(im[i]) * inv);
  }
}

// ---------------------------------------------------------------------------------------------
// FP64 reductions (norm, <Z_mask>, <a|b>): grid-stride partial sums per CTA; the CTA that finishes last
// sums the partials in a fixed order (deterministic) and writes the two results, and beside them the
// context's error flag, to `out` (device memory, or pinned host memory that the host reads after waiting
// for the stream: no copy to enqueue). partials ends with a counter of finished CTAs, zero between calls.
// ---------------------------------------------------------------------------------------------
constexpr int kReduceBlocksPerSM = 4;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void block_sum2(double& a, double& b) {
  __shared__ double sa[32], sb[32];
  a = warp_sum(a);
  b = warp_sum(b);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sa[wid] = a;
    sb[wid] = b;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    a = lane < nw ? sa[lane] : 0.0;
    b = lane < nw ? sb[lane] : 0.0;
    a = warp_sum(a);
    b = warp_sum(b);
  }
}

__device__ __forceinline__ void finish_reduce(double a, double b, double* partials, uint32_t* counter, double* out,
                                              const int* err) {
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = a;
    partials[2 * blockIdx.x + 1] = b;
    __threadfence();
    s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  a = b = 0.0;
  for (int i = threadIdx.x; i < int(gridDim.x); i += blockDim.x) {
    a += __ldcg(partials + 2 * i);
    b += __ldcg(partials + 2 * i + 1);
  }
  block_sum2(a, b);
  if (threadIdx.x == 0) {
    *counter = 0;
    out[0] = a;
    out[1] = b;
    if (err) out[2] = double(*reinterpret_cast<const volatile int*>(err));
    __threadfence_system();
  }
}

template <class R>
__global__ void __launch_bounds__(kThreads) k_reduce(int op, const R* __restrict__ re, const R* __restrict__ im,
                                                     const R* __restrict__ re2, const R* __restrict__ im2,
                                                     uint64_t dim, uint64_t mask, double* partials, uint32_t* counter,
                                                     double* out, const int* err) {
  constexpr int N = VecT<R>::N;
  early_next();
  wait_prior();
  double a = 0.0, b = 0.0;
  if (dim % N == 0) {
    const uint64_t nvec = dim / N;
    for (uint64_t w = gtid(); w < nvec; w += gstride()) {
      R xr[N], xi[N];
      vld(re + w * N, xr);
      vld(im + w * N, xi);
      if (op == RED_INNER) {
        R yr[N], yi[N];
        vld(re2 + w * N, yr);
        vld(im2 + w * N, yi);
#pragma unroll
        for (int e = 0; e < N; ++e) {  // conj(x) * y
          a += double(xr[e]) * double(yr[e]) + double(xi[e]) * double(yi[e]);
          b += double(xr[e]) * double(yi[e]) - double(xi[e]) * double(yr[e]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < N; ++e) {
          const double p = double(xr[e]) * double(xr[e]) + double(xi[e]) * double(xi[e]);
          if (op == RED_EXPZ && (__popcll((w * N + e) & mask) & 1)) a -= p;
          else a += p;
        }
      }
    }
  } else {
    for (uint64_t i = gtid(); i < dim; i += gstride()) {
      const double xr = re[i], xi = im[i];
      if (op == RED_INNER) {
        a += xr * double(re2[i]) + xi * double(im2[i]);
        b += xr * double(im2[i]) - xi * double(re2[i]);
      } else {
        const double p = xr * xr + xi * xi;
        if (op == RED_EXPZ && (__popcll(i & mask) & 1)) a -= p;
        else a += p;
      }
    }
  }
  block_sum2(a, b);
  finish_reduce(a, b, partials, counter, out, err);
}

template <class R> __device__ __forceinline__ void load4(const R* p, R (&x)[4]) {
  if constexpr (sizeof(R) == 4) {
    vld(p, x);
  } else {
    R a[2], b[2];
    vld(p, a);
    vld(p + 2, b);
    x[0] = a[0]; x[1] = a[1]; x[2] = b[0]; x[3] = b[1];
  }
}

// <a|b> across precisions (complex64 state vs its FP64 twin), FP64 accumulation.
template <class RA, class RB>
__global__ void __launch_bounds__(kThreads) k_inner_mixed(const RA* __restrict__ are, const RA* __restrict__ aim,
                                                          const RB* __restrict__ bre, const RB* __restrict__ bim,
                                                          uint64_t dim, double* partials, uint32_t* counter,
                                                          double* out, const int* err) {
  early_next();
  wait_prior();
  double a = 0.0, b = 0.0;
  if (dim % 4 == 0) {
    for (uint64_t w = gtid(); w < dim / 4; w += gstride()) {
      RA xr[4], xi[4];
      RB yr[4], yi[4];
      load4(are + 4 * w, xr);
      load4(aim + 4 * w, xi);
      load4(bre + 4 * w, yr);
      load4(bim + 4 * w, yi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a += double(xr[e]) * double(yr[e]) + double(xi[e]) * double(yi[e]);
        b += double(xr[e]) * double(yi[e]) - double(xi[e]) * double(yr[e]);
      }
    }
  } else {
    for (uint64_t i = gtid(); i < dim; i += gstride()) {
      a += double(are[i]) * double(bre[i]) + double(aim[i]) * double(bim[i]);
      b += double(are[i]) * double(bim[i]) - double(aim[i]) * double(bre[i]);
    }
  }
  block_sum2(a, b);
  finish_reduce(a, b, partials, counter, out, err);
}

template <class R>
__global__ void k_probs(const R* __restrict__ re, const R* __restrict__ im, uint64_t off, uint64_t count,
                        void* out, int out_f64) {
  for (uint64_t i = gtid(); i < count; i += gstride()) {
    const double xr = re[off + i], xi = im[off + i];
    const double p = xr * xr + xi * xi;
    if (out_f64) static_cast<double*>(out)[i] = p;
    else static_cast<float*>(out)[i] = float(p);
  }
}

// ---------------------------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------------------------
// Blocks of a kernel an SM holds at a time. A grid of persistent blocks launched programmatically has to fill
// every SM: its blocks start wherever the kernel before it leaves room, so with fewer of them than fit, the SMs
// that finish first take more than their share (26-qubit complex128 two-qubit sweeps back to back, three
// blocks an SM where four fit: 413 us a sweep, against 337 us alone).
inline int resident_blocks(const void* kern, int threads, size_t smem) {
  int blocks = 0;
  QSVB_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, threads, smem));
  QSVB_REQUIRE(blocks >= 1, "kernel does not fit on an SM");
  return blocks;
}

inline unsigned grid_for(uint64_t items, int per_block, int num_sms, int blocks_per_sm = 8) {
  const uint64_t need = (items + per_block - 1) / per_block;
  const uint64_t cap = uint64_t(num_sms) * blocks_per_sm;
  return unsigned(std::max<uint64_t>(1, std::min(need, cap)));
}

inline void check_launch() { QSVB_CK(cudaGetLastError()); }

template <class R> M2<R> to_m2(const std::vector<cd>& u) {
  M2<R> g;
  for (int i = 0; i < 4; ++i) {
    g.a[2 * i] = R(u[i].real());
    g.a[2 * i + 1] = R(u[i].imag());
  }
  return g;
}

Enum make_enum(std::vector<uint32_t> fixed, uint64_t set_mask, uint64_t flip = 0) {
  Enum e{};
  e.flip = flip;
  std::sort(fixed.begin(), fixed.end());
  QSVB_REQUIRE(fixed.size() <= 7, "too many fixed bits");
  e.nfixed = uint32_t(fixed.size());
  for (size_t i = 0; i < fixed.size(); ++i) e.fixed[i] = fixed[i];
  e.set_mask = set_mask;
  return e;
}

template <class R>
void launch_pair(const LaunchEnv& env, R* re, R* im, uint32_t n, uint32_t t, const uint32_t* ctrl,
                 uint32_t nctrl, const std::vector<cd>& u) {
  constexpr uint32_t LOG = VecT<R>::LOG;
  const M2<R> g = to_m2<R>(u);
  uint64_t cmask = 0;
  for (uint32_t i = 0; i < nctrl; ++i) cmask |= 1ull << ctrl[i];
  auto split = [&](uint32_t cb, std::vector<uint32_t>& fixed, uint32_t& low) {
    low = 0;
    uint64_t set = 0;
    for (uint32_t i = 0; i < nctrl; ++i) {
      if (ctrl[i] >= cb) {
        fixed.push_back(ctrl[i]);
        set |= 1ull << ctrl[i];
      } else {
        low |= 1u << ctrl[i];
      }
    }
    return set;
  };
  const uint32_t nfix_ctrl_hi_max = nctrl;
  if (n >= 12 && n >= LOG + 6 + nfix_ctrl_hi_max) {
    std::vector<uint32_t> fixed;
    uint32_t low;
    if (t < LOG) {
      const uint64_t set = split(LOG, fixed, low);
      const uint64_t nwork = 1ull << (n - LOG - fixed.size());
      auto kern = t == 0 ? k_pair_invec<R, 0> : k_pair_invec<R, LOG - 1>;  // LOG is 1 or 2
      launch_pdl(kern, grid_for(nwork, kThreads, env.num_sms), kThreads, 0, env, re, im, nwork,
                 make_enum(fixed, set, env.flip(nwork)), low, g);
    } else if (t < LOG + 5) {
      const uint64_t set = split(LOG + 5, fixed, low);
      const uint64_t nwork = 1ull << (n - LOG - 5 - fixed.size());
      launch_pdl(k_pair_shfl<R>, grid_for(nwork * 32, kThreads, env.num_sms), kThreads, 0, env,
          re, im, nwork, make_enum(fixed, set, env.flip(nwork)), t, low, g);
    } else {
      const uint64_t set = split(LOG, fixed, low);
      fixed.push_back(t);
      const uint64_t nwork = 1ull << (n - LOG - fixed.size());
      launch_pdl(k_pair_strided<R>, grid_for(nwork, kThreads, env.num_sms), kThreads, 0, env,
          re, im, nwork, make_enum(fixed, set, env.flip(nwork)), t, low, g);
    }
  } else {
    std::vector<uint32_t> fixed(ctrl, ctrl + nctrl);
    fixed.push_back(t);
    const uint64_t nwork = 1ull << (n - fixed.size());
    launch_pdl(k_pair_scalar<R>, grid_for(nwork, kThreads, env.num_sms), kThreads, 0, env,
        re, im, nwork, make_enum(fixed, cmask, env.flip(nwork)), t, g);
  }
  check_launch();
}

template <class R>
void launch_diag(const LaunchEnv& env, R* re, R* im, uint32_t n, const Sweep& s) {
  constexpr uint32_t LOG = VecT<R>::LOG;
  DiagP<R> p{};
  p.m = s.m;
  for (uint32_t j = 0; j < 6; ++j) p.q[j] = j < s.m ? s.q[j] : 63u;
  for (size_t i = 0; i < s.mat.size(); ++i) {
    p.d[2 * i] = R(s.mat[i].real());
    p.d[2 * i + 1] = R(s.mat[i].imag());
  }
  if (n >= 12) {
    // qubits whose 0-half is the identity (the "controls" the classifier found) are skipped
    std::vector<uint32_t> fixed;
    uint64_t set = 0;
    for (uint32_t i = 0; i < s.nctrl; ++i)
      if (s.ctrl[i] >= LOG) {
        fixed.push_back(s.ctrl[i]);
        set |= 1ull << s.ctrl[i];
      }
    const uint64_t nwork = 1ull << (n - LOG - fixed.size());
    launch_pdl(k_diag<R>, grid_for(nwork, kThreads, env.num_sms), kThreads, 0, env,
        re, im, nwork, make_enum(fixed, set, env.flip(nwork)), p);
  } else {
    const uint64_t dim = 1ull << n;
    launch_pdl(k_diag_scalar<R>, grid_for(dim, kThreads, env.num_sms), kThreads, 0, env, re, im, dim, p);
  }
  check_launch();
}

// Launch shape of k_dense_mma for K gate bits: column groups of 8 a warp works on at a time, threads a
// block, blocks an SM. More groups keep more bytes in flight and use each matrix fragment more often,
// as far as registers allow (27-qubit complex128 states, gate bits 10..17: K = 4 0.99 / 0.78 / 0.71 ms
// with 1 / 2 / 4 groups, K = 3 0.81 / 0.74 ms with 2 / 4, K = 5 1.27 / 1.24 ms with 1 / 2. K = 2 is one
// block of 12 warps: with four blocks of four warps, which also fit, 26 qubits take 0.38 instead of 0.33 ms).
struct DenseMmaShape {
  int groups, threads, blocks;
};
constexpr DenseMmaShape dense_mma_shape(int K) {
  return K == 2 ? DenseMmaShape{8, 384, 1}
         : K == 3 ? DenseMmaShape{4, 128, 4}
         : K == 4 ? DenseMmaShape{4, 128, 3}
         : K == 5 ? DenseMmaShape{2, 128, 3}
                  : DenseMmaShape{1, 512, 1};
}

template <class R, int K, int G, int TH, int MINB, int TAIL>
void launch_dense_mma_shape(const LaunchEnv& env, R* re, R* im, uint64_t ngroups, const R* u, DenseMmaP p,
                            const TailIf<R, TAIL>& t) {
  constexpr size_t smem = size_t(32) << (2 * K);
  auto kern = k_dense_mma<R, K, G, TH, MINB, TAIL>;
  if constexpr (smem > 48 * 1024)
    QSVB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  const uint64_t items = ngroups / G;
  p.flip = env.flip(items);
  static const int per_sm = resident_blocks(reinterpret_cast<const void*>(kern), TH, smem);
  // After k_diag a large K = 4 sweep launches ordinarily: that kernel's 0.5 or 1 KB a block leave the SM a split
  // with room for one of these blocks' matrices, not three, and an SM that holds one keeps the split, so blocks
  // started early found SMs with one or two and the others waited for a second wave. A CZ and such a sweep,
  // complex128, programmatic -> ordinary: 28 qubits 2.25 -> 1.81 ms, 25 qubits 267 -> 225 us, 23 qubits 67 -> 62
  // us; at 22 qubits the saved launch counts for more (30 -> 32 us). K = 2, 3 fit as they are, K = 5, 6 not at all.
  LaunchEnv e = env;
  if constexpr (sizeof(R) == 8 && K == 4 && G > 1)
    e.early = e.early && !(env.after_diag && items * G * 8 * (1u << K) >= uint64_t(1) << 23);
  launch_pdl(kern, grid_for(items, TH / 32, env.num_sms, per_sm), TH, smem, e, re, im, items, u, p, t);
  check_launch();
}

// The value with zero bits inserted at the ascending positions q (layout.rs:70-86).
inline uint64_t insert_bits(uint64_t x, const uint32_t* q, size_t count) {
  for (size_t j = 0; j < count; ++j) {
    const uint64_t lo = x & ((1ull << q[j]) - 1ull);
    x = ((x - lo) << 1) | lo;
  }
  return x;
}

template <class R> uint32_t tail_bits(const Tail<R>& t, uint64_t address) {
  uint32_t s = 0;
  for (uint32_t j = 0; j < t.m; ++j) s |= uint32_t((address >> t.q[j]) & 1u) << j;
  return s;
}

template <class R, int K, int TAIL>
void launch_dense_mma(const LaunchEnv& env, R* re, R* im, uint32_t n, const uint32_t* q, const R* u,
                      TailIf<R, TAIL> t) {
  DenseMmaP p{};
  for (int j = 0; j < K; ++j) p.bit[j] = 1ull << q[j];
  for (int j = 0; j < 3; ++j) p.grp[j] = insert_bits(8ull << j, q, K);
  if constexpr (TAIL) {
    for (int j = 0; j < K; ++j) t.gate[j] = tail_bits(t, p.bit[j]);
    for (int j = 0; j < 3; ++j) t.grp[j] = tail_bits(t, p.grp[j]);
  }
  constexpr DenseMmaShape sh = dense_mma_shape(K);
  const uint64_t ngroups = 1ull << (n - K - 3);
  // several groups a warp only once every resident warp has an item of its own; below that, one group
  // a warp in small blocks spreads the state over more SMs
  if (ngroups / sh.groups >= uint64_t(env.num_sms) * sh.blocks * (sh.threads / 32))
    launch_dense_mma_shape<R, K, sh.groups, sh.threads, sh.blocks, TAIL>(env, re, im, ngroups, u, p, t);
  else if constexpr (K < 6)
    launch_dense_mma_shape<R, K, 1, 64, 4, TAIL>(env, re, im, ngroups, u, p, t);
  else
    launch_dense_mma_shape<R, K, 1, 128, 1, TAIL>(env, re, im, ngroups, u, p, t);
}

// k_dense_cols holds 2^K x 4 amplitudes a thread: one block of as many warps as the registers allow
// (K = 4 with all gate bits above bit 1: 12 warps 0.38 ms, 8 warps 0.41 ms; with shuffles or more rows a
// step 8 warps win, 0.44-0.47 against 0.44-0.51 ms).
constexpr int dense_cols_threads(int K, int nlow, int l2) {
  return K == 4 ? (nlow == 0 && l2 == 0 ? 384 : 256) : 512;
}

template <int K, int L0, int L1, int L2, int TAIL>
void launch_dense_cols_at(const LaunchEnv& env, float* re, float* im, uint32_t n, const float* u, DenseColP p,
                          const TailIf<float, TAIL>& t) {
  constexpr int TH = dense_cols_threads(K, L0 + L1, L2);
  const uint64_t items = 1ull << (n - K - 7);
  p.flip = env.flip(items);
  launch_pdl(k_dense_cols<K, L0, L1, L2, TH, TAIL>, grid_for(items, TH / 32, env.num_sms, 1), TH, 0, env, re, im,
             items, reinterpret_cast<const float2*>(u), p, t);
  check_launch();
}

template <int K, int TAIL>
void launch_dense_cols(const LaunchEnv& env, float* re, float* im, uint32_t n, const uint32_t* q, const float* u,
                       TailIf<float, TAIL> t) {
  auto has = [&](uint32_t b) { return std::find(q, q + K, b) != q + K; };
  const bool l0 = has(0), l1 = has(1), l2 = has(2);
  const uint32_t nlow = uint32_t(l0) + uint32_t(l1);
  DenseColP p{};
  std::vector<uint32_t> ins(q, q + K);
  for (uint32_t b = 0; b < 2; ++b)
    if (!has(b)) ins.push_back(b);
  std::sort(ins.begin(), ins.end());
  p.nins = uint32_t(ins.size());
  std::copy(ins.begin(), ins.end(), p.ins);
  for (uint32_t j = nlow; j < uint32_t(K); ++j) p.hi[j - nlow] = 1ull << q[j];
  // the extra columns lie above the 5 lane bits
  for (uint32_t j = 0; j < nlow; ++j) p.ext[j] = insert_bits(1ull << (5 + j), p.ins, p.nins);
  if constexpr (TAIL) {
    for (uint32_t j = 0; j < 2; ++j) t.ext[j] = tail_bits(t, p.ext[j]), t.elem[j] = tail_bits(t, 1ull << j);
    for (uint32_t j = 0; j < uint32_t(K) - nlow; ++j) t.gate[j] = tail_bits(t, p.hi[j]);
    // bit 0 of the kernel's row groups: see `first`
    if (l2 && nlow < 2) t.gate[0] = tail_bits(t, insert_bits(1, p.ins, p.nins));
  }
  if (l0 && l1) launch_dense_cols_at<K, 1, 1, 0, TAIL>(env, re, im, n, u, p, t);  // a thread has whole sectors
  else if (l0 && l2) launch_dense_cols_at<K, 1, 0, 1, TAIL>(env, re, im, n, u, p, t);
  else if (l0) launch_dense_cols_at<K, 1, 0, 0, TAIL>(env, re, im, n, u, p, t);
  else if (l1 && l2) launch_dense_cols_at<K, 0, 1, 1, TAIL>(env, re, im, n, u, p, t);
  else if (l1) launch_dense_cols_at<K, 0, 1, 0, TAIL>(env, re, im, n, u, p, t);
  else if (l2) launch_dense_cols_at<K, 0, 0, 1, TAIL>(env, re, im, n, u, p, t);
  else launch_dense_cols_at<K, 0, 0, 0, TAIL>(env, re, im, n, u, p, t);
}

// Which kernel runs a dense sweep:
//  * fewer than 8 columns: one block of amplitudes per thread;
//  * complex64 with K <= 4 once every resident warp has 2^K x 128 amplitudes of its own (n >= 21 or 22):
//    paired FP32 FMAs;
//  * everything else: the FP64 matrix instruction. That is complex128, complex64 states below that
//    size (a warp there needs only 2^K x 8 amplitudes, so more SMs take part) and complex64 K = 5, 6 on
//    CUDA cores (27 qubits: 1.20 ms against 1.20 (K = 5) and 2.02 against 2.09 ms (K = 6) for an FP32
//    shared-memory tile, with one rounding instead of 2^(K+1)).
template <class R, int K, int TAIL>
void launch_dense_of(const LaunchEnv& env, R* re, R* im, uint32_t n, const Sweep& s, const R* u) {
  const uint32_t* q = s.q;  // ascending
  if (n < uint32_t(K + 3)) {
    if constexpr (!TAIL) {  // (attach_diagonals leaves such states alone)
      const uint64_t nb = 1ull << (n - K);
      launch_pdl(k_dense_small<R, K>, grid_for(nb, 128, env.num_sms), 128, 0, env, re, im, nb, u, make_enum(std::vector<uint32_t>(q, q + K), 0), q[0], q[1], q[2], q[3], q[4], q[5]);
      check_launch();
      return;
    }
    throw Error(QSVB_E_INVALID, "dense sweep with a tail needs at least 8 columns");
  }
  TailIf<R, TAIL> t{};
  if constexpr (TAIL) {
    t.m = s.tail_m;
    t.need = s.tail_need;
    for (uint32_t j = 0; j < 6; ++j) t.q[j] = j < s.tail_m ? s.tail_q[j] : 63u;
    for (size_t i = 0; i < s.tail.size(); ++i) {
      t.d[2 * i] = R(s.tail[i].real());
      t.d[2 * i + 1] = R(s.tail[i].imag());
      if (i < 32 && s.tail[i] == cd(-1, 0)) t.neg |= 1u << i;
    }
  }
  if constexpr (sizeof(R) == 4 && K <= 4) {
    if (n >= uint32_t(K + 7) &&
        (1ull << (n - K - 7)) >= uint64_t(env.num_sms) * (dense_cols_threads(K, 0, 0) / 32)) {
      launch_dense_cols<K, TAIL>(env, re, im, n, q, u, t);
      return;
    }
  }
  launch_dense_mma<R, K, TAIL>(env, re, im, n, q, u, t);
}

template <class R, int TAIL>
void launch_dense(const LaunchEnv& env, R* re, R* im, uint32_t n, const Sweep& s, const void* dev_mat) {
  const R* u = static_cast<const R*>(dev_mat);
  switch (s.m) {
    case 2: launch_dense_of<R, 2, TAIL>(env, re, im, n, s, u); break;
    case 3: launch_dense_of<R, 3, TAIL>(env, re, im, n, s, u); break;
    case 4: launch_dense_of<R, 4, TAIL>(env, re, im, n, s, u); break;
    case 5: launch_dense_of<R, 5, TAIL>(env, re, im, n, s, u); break;
    case 6: launch_dense_of<R, 6, TAIL>(env, re, im, n, s, u); break;
    default: throw Error(QSVB_E_INVALID, "dense sweep arity must be 2..6");
  }
}

template <class R>
void launch_phase(const LaunchEnv& env, R* re, R* im, uint32_t n, const Sweep& s, const void* dev_terms) {
  const uint64_t dim = 1ull << n;
  const uint32_t nt = uint32_t(s.terms.size());
  if (n >= uint32_t(kIsingChunkBits)) {
    // Walsh transform of every term: theta = c0 + c1 z0 (+ c2 z1 + c3 z0 z1), index = b0 + 2 b1
    IsingP p{};
    std::vector<std::pair<uint32_t, uint32_t>> keys;
    std::vector<double> js;
    for (const PhaseTerm& t : s.terms) {
      const double* a = t.ang;
      if (t.m == 1) {
        p.c0 += 0.5 * (a[0] + a[1]);
        p.h[t.q[0]] += 0.5 * (a[0] - a[1]);
        continue;
      }
      p.c0 += 0.25 * (a[0] + a[1] + a[2] + a[3]);
      p.h[t.q[0]] += 0.25 * (a[0] - a[1] + a[2] - a[3]);
      p.h[t.q[1]] += 0.25 * (a[0] + a[1] - a[2] - a[3]);
      const double j = 0.25 * (a[0] - a[1] - a[2] + a[3]);
      const auto key = std::make_pair(std::min(t.q[0], t.q[1]), std::max(t.q[0], t.q[1]));
      const auto it = std::find(keys.begin(), keys.end(), key);
      if (it == keys.end()) {
        keys.push_back(key);
        js.push_back(j);
      } else {
        js[size_t(it - keys.begin())] += j;
      }
    }
    QSVB_REQUIRE(keys.size() <= size_t(kIsingMaxEdges), "phase polynomial has too many distinct pairs");
    p.nedges = uint32_t(keys.size());
    for (size_t e = 0; e < keys.size(); ++e) {
      p.ea[e] = uint8_t(keys[e].first);
      p.eb[e] = uint8_t(keys[e].second);
      p.J[e] = js[e];
    }
    const uint64_t nchunks = dim >> kIsingChunkBits;
    const size_t tsm = sizeof(double2) << kIsingChunkBits;
    QSVB_CK(cudaFuncSetAttribute(k_ising<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tsm)));
    k_ising<R><<<grid_for(nchunks, 1, env.num_sms, 3), kThreads, tsm, env.stream>>>(re, im, nchunks, p);
    check_launch();
    return;
  }
  const size_t smem = nt * sizeof(PhaseTermDev);
  QSVB_REQUIRE(smem <= 200 * 1024, "phase polynomial too large");
  QSVB_CK(cudaFuncSetAttribute(k_phase<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  QSVB_REQUIRE(dim % VecT<R>::N == 0, "phase sweep needs >= 2 qubits");
  k_phase<R><<<grid_for(dim / VecT<R>::N, kThreads, env.num_sms), kThreads, smem, env.stream>>>(
      re, im, dim, static_cast<const PhaseTermDev*>(dev_terms), nt);
  check_launch();
}

}  // namespace

// ------------------------------------------------------------------------------ public launchers

size_t sweep_matrix_bytes(const Sweep& s, int dtype) {
  const size_t r = dtype == QSVB_C128 ? 8 : 4;
  switch (s.kind) {
    case SK_DENSE: return 2 * r * (size_t(1) << (2 * s.m));
    case SK_DENSE_TC: return tc_matrix_bytes(s);
    case SK_PHASE: return s.terms.size() * sizeof(PhaseTermDev);
    case SK_TILE: return s.tile_blob.size();
    case SK_TC_CHAIN: return tc_chain_matrix_bytes(s);
    default: return 0;
  }
}

void pack_sweep_matrix(const Sweep& s, int dtype, void* dst) {
  if (s.kind == SK_DENSE) {
    const uint32_t M = 1u << s.m;
    for (uint32_t r = 0; r < M; ++r)
      for (uint32_t c = 0; c < M; ++c) {
        const cd v = s.mat[size_t(r) * M + c];
        const size_t o = 2 * (size_t(r) * M + c);
        if (dtype == QSVB_C128) {
          static_cast<double*>(dst)[o] = v.real();
          static_cast<double*>(dst)[o + 1] = v.imag();
        } else {
          static_cast<float*>(dst)[o] = float(v.real());
          static_cast<float*>(dst)[o + 1] = float(v.imag());
        }
      }
  } else if (s.kind == SK_TILE) {
    std::memcpy(dst, s.tile_blob.data(), s.tile_blob.size());
  } else if (s.kind == SK_DENSE_TC) {
    tc_pack_matrix(s, dst);
  } else if (s.kind == SK_TC_CHAIN) {
    tc_chain_pack(s, dst);
  } else if (s.kind == SK_PHASE) {
    PhaseTermDev* t = static_cast<PhaseTermDev*>(dst);
    for (size_t i = 0; i < s.terms.size(); ++i) {
      t[i].q0 = s.terms[i].q[0];
      t[i].q1 = s.terms[i].m == 2 ? s.terms[i].q[1] : 64u;
      for (int k = 0; k < 4; ++k) t[i].ang[k] = s.terms[i].ang[k];
    }
  }
}

template <class R>
void launch_sweep(const LaunchEnv& env, R* re, R* im, uint32_t n, const Sweep& s, const void* dev_mat, bool tail) {
  switch (s.kind) {
    case SK_1Q: launch_pair<R>(env, re, im, n, s.target, nullptr, 0, s.mat); break;
    case SK_CTRL: launch_pair<R>(env, re, im, n, s.target, s.ctrl, s.nctrl, s.mat); break;
    case SK_DIAG: launch_diag<R>(env, re, im, n, s); break;
    case SK_PHASE: launch_phase<R>(env, re, im, n, s, dev_mat); break;
    case SK_DENSE:
      if (!tail || !s.tail_m) {
        launch_dense<R, kTailNone>(env, re, im, n, s, dev_mat);
      } else {
        bool signs = s.tail_m <= 5;
        for (const cd& z : s.tail) signs = signs && (z == cd(1, 0) || z == cd(-1, 0));
        if (signs) launch_dense<R, kTailSign>(env, re, im, n, s, dev_mat);
        else launch_dense<R, kTailTable>(env, re, im, n, s, dev_mat);
      }
      break;
    case SK_DENSE_TC:
      if constexpr (sizeof(R) == 4) {
        launch_tc_dense(env, reinterpret_cast<float*>(re), reinterpret_cast<float*>(im), n, s, dev_mat);
        break;
      }
      throw Error(QSVB_E_UNSUPPORTED, "tensor-core sweeps need a complex64 state");
    case SK_TILE: launch_tile<R>(env, re, im, n, s, dev_mat); break;
    case SK_TC_CHAIN:
      if constexpr (sizeof(R) == 4) {
        launch_tc_chain(env, reinterpret_cast<float*>(re), reinterpret_cast<float*>(im), n, s, dev_mat);
        break;
      }
      throw Error(QSVB_E_UNSUPPORTED, "tensor-core chain passes need a complex64 state");
    case SK_PERMUTE: launch_permute<R>(env, re, im, n, s); break;
    case SK_NONE: break;
    default: throw Error(QSVB_E_UNSUPPORTED, "unknown sweep kind");
  }
}

template <class R> void launch_init_basis(const LaunchEnv& e, R* re, R* im, uint32_t n, uint64_t basis) {
  const uint64_t dim = 1ull << n;
  launch_pdl(k_init_basis<R>, grid_for(dim / VecT<R>::N + 1, kThreads, e.num_sms), kThreads, 0, e, re, im, dim, basis);
}

template <class R> void launch_init_gaussian(const LaunchEnv& e, R* re, R* im, uint32_t n, uint64_t seed) {
  const uint64_t dim = 1ull << n;
  k_gaussian<R><<<grid_for(dim, kThreads, e.num_sms), kThreads, 0, e.stream>>>(re, im, dim, seed);
  check_launch();
}

template <class R> void launch_scale(const LaunchEnv& e, R* re, R* im, uint32_t n, const double* d_norm) {
  const uint64_t dim = 1ull << n;
  k_scale<R><<<grid_for(dim, kThreads, e.num_sms), kThreads, 0, e.stream>>>(re, im, dim, d_norm);
  check_launch();
}

size_t reduce_partials_needed(int num_sms) { return size_t(2) * num_sms * kReduceBlocksPerSM + 1; }

// the counter of finished CTAs behind the partial sums
static uint32_t* reduce_counter(const LaunchEnv& e, double* partials) {
  return reinterpret_cast<uint32_t*>(partials + reduce_partials_needed(e.num_sms) - 1);
}

template <class R>
void launch_reduce(const LaunchEnv& e, int op, const R* re, const R* im, const R* re2, const R* im2,
                   uint32_t n, uint64_t mask, double* partials, double* d_out) {
  const uint64_t dim = 1ull << n;
  const unsigned grid = grid_for(dim / VecT<R>::N + 1, kThreads, e.num_sms, kReduceBlocksPerSM);
  launch_pdl(k_reduce<R>, grid, kThreads, 0, e, op, re, im, re2, im2, dim, mask, partials,
             reduce_counter(e, partials), d_out, e.err_flag);
}

template <class RA, class RB>
void launch_inner_mixed(const LaunchEnv& e, const RA* are, const RA* aim, const RB* bre, const RB* bim, uint32_t n,
                        double* partials, double* d_out) {
  const uint64_t dim = 1ull << n;
  const unsigned grid = grid_for(dim / 4 + 1, kThreads, e.num_sms, kReduceBlocksPerSM);
  launch_pdl(k_inner_mixed<RA, RB>, grid, kThreads, 0, e, are, aim, bre, bim, dim, partials,
             reduce_counter(e, partials), d_out, e.err_flag);
}
template void launch_inner_mixed<float, double>(const LaunchEnv&, const float*, const float*, const double*,
                                                const double*, uint32_t, double*, double*);
template void launch_inner_mixed<double, float>(const LaunchEnv&, const double*, const double*, const float*,
                                                const float*, uint32_t, double*, double*);

template <class R>
void launch_probabilities(const LaunchEnv& e, const R* re, const R* im, uint64_t offset, uint64_t count,
                          void* out, int out_f64) {
  k_probs<R><<<grid_for(count, kThreads, e.num_sms), kThreads, 0, e.stream>>>(re, im, offset, count, out, out_f64);
  check_launch();
}

#define QSVB_INST(R)                                                                                   \
  template void launch_sweep<R>(const LaunchEnv&, R*, R*, uint32_t, const Sweep&, const void*, bool); \
  template void launch_init_basis<R>(const LaunchEnv&, R*, R*, uint32_t, uint64_t);                   \
  template void launch_init_gaussian<R>(const LaunchEnv&, R*, R*, uint32_t, uint64_t);                \
  template void launch_scale<R>(const LaunchEnv&, R*, R*, uint32_t, const double*);                   \
  template void launch_reduce<R>(const LaunchEnv&, int, const R*, const R*, const R*, const R*,       \
                                 uint32_t, uint64_t, double*, double*);                               \
  template void launch_probabilities<R>(const LaunchEnv&, const R*, const R*, uint64_t, uint64_t,     \
                                        void*, int);
QSVB_INST(float)
QSVB_INST(double)

}  // namespace qsvb
