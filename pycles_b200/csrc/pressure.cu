// Anelastic pressure solve on one GPU.
//
// The reference's pencil transposes (ParallelMPI.Pencil) become a choice of
// layout: the spectral work array is W[k][j][m] (complex, m fastest), so
// the x-FFT reads physical rows and writes contiguous m, the y-FFT works on
// j-lines batched over contiguous m, and the Thomas solver gives one thread
// to each (kx,ky) column with consecutive threads on consecutive m.
//
// The reference transforms the real right-hand side with a complex FFT and
// solves every (kx,ky) column.  The field is real, so the x-spectrum of each
// row is Hermitian, X[n0 - m] = conj(X[m]); the tridiagonal matrix is real
// and depends on kx only through kx^2, which is even in m; so the columns
// m > n0/2 hold the conjugates of the columns n0 - m (with ky reflected) and
// carry no information.  W keeps the n0/2 + 1 columns m = 0..n0/2.  Two real
// rows (levels 2p, 2p+1) share one complex FFT, z = a + i b, and are
// separated by A[m] = (Z[m] + conj Z[n0-m]) / 2, B[m] = (Z[m] - conj Z[n0-m]) / 2i;
// the inverse rebuilds Z = A + i B over all m from the stored half and
// returns a = Re z, b = Im z.  This halves the x-FFT work, and the y-FFT,
// Thomas and spectral-array traffic, with the same mathematics as the
// reference's full-spectrum solve.
//
//   hsum_* (plain form)        HorizontalMean(w) in the reference's order
//   hmean_partial/hmean_final  (precision form) deterministic two-pass sum
//   (remove_mean_u3)           w -= mean[k] on every cell, applied where w is
//                              read: in the divergence and in the correction
//   zero_ghosts                divergence ghosts = 0 (the reference zeroes the
//                              whole array before adding the interior terms);
//                              in the one-GPU solve part of the last ghost_sym
//   fft_x_fwd                  second_order_divergence (d = 0,1,2 in order)
//                              + x-FFT of each (j, k) row
//   fft_y                      y-FFT (forward, or inverse with 1/n1)
//   tdma                       per-column Thomas (SparseSolvers.pyx:24-44) on
//                              the complex coefficients, mode (0,0) := 0
//   fft_x_inv                  inverse x-FFT, 1/n0, real part -> pressure
//   (ghost fill, sym)          DiagnosticVariables.communicate_variable
//   correction                 second_order_pressure_correction
#include <math.h>
#include <string.h>

#include <vector>

#include "pb_common.cuh"

namespace {

constexpr int kPartials = 1184;  // 8 x 148 SMs
constexpr int kFftThreads = 256;  // stockham_pass: nlines * N <= 16 * kFftThreads
constexpr int kMaxKC = 32;        // levels per x-FFT block at most (two per line, 16 lines)

struct PLayout {
  long long partial, mean, twx, twy, twxf, twyf, kx2, ky2, spec, scr, total;
};

long long align256(long long x) { return (x + 255) / 256 * 256; }

PLayout playout(const pb_dims* d) {
  PLayout L;
  const long long n0 = d->n[0], n1 = d->n[1], n2 = d->n[2];
  const long long nlg2 = d->nlg[2];
  long long off = 0;
  L.partial = off; off += align256((long long)kPartials * nlg2 * 8);
  L.mean = off;    off += align256(nlg2 * 8);
  L.twx = off;     off += align256(n0 * 16);
  L.twy = off;     off += align256(n1 * 16);
  L.twxf = off;    off += align256(n0 * 8);
  L.twyf = off;    off += align256(n1 * 8);
  L.kx2 = off;     off += align256(n0 * 8);
  L.ky2 = off;     off += align256(n1 * 8);
  // spectral array W[k][j][m], m < n0/2 + 1 (Hermitian half in x)
  L.spec = off;    off += align256((n0 / 2 + 1) * n1 * n2 * 16);
  L.scr = off;     off += align256((n0 / 2 + 1) * n1 * n2 * 8);
  L.total = off;
  return L;
}

__device__ __forceinline__ bool is_pow2(int n) { return (n & (n - 1)) == 0; }

// Lines per FFT block for a power-of-two length 2^lg (16 lines, or fewer so
// that a block's passes hold nlines * N <= 16 * kFftThreads elements); the
// host's lines_for gives the same count for every power of two.
__host__ __device__ constexpr int ct_lines(int lg) { return (16 * 256 >> lg) < 16 ? (16 * 256 >> lg) : 16; }

// Complex arithmetic on double2 (plain form) or float2 (precision form).
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
template <class C> __device__ __forceinline__ C czero();
template <> __device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }
template <> __device__ __forceinline__ float2 czero<float2>() { return make_float2(0.0f, 0.0f); }
template <class C> __device__ __forceinline__ C creal(double x);
template <> __device__ __forceinline__ double2 creal<double2>(double x) { return make_double2(x, 0.0); }
template <> __device__ __forceinline__ float2 creal<float2>(double x) { return make_float2((float)x, 0.0f); }

// ---- line FFTs in shared memory --------------------------------------------
// A block transforms `nlines` lines of length N held in shared memory.  Line l
// element x lives at l*line_ld(N) + swz(x): the swizzle (one pad element per
// 8) and the odd line stride keep the strided accesses of the passes and of
// the global loads/stores (consecutive threads on consecutive lines) free of
// bank conflicts.
// The stride is chosen for the transposing loads and stores: a half-warp
// touches IC lines at 16/IC consecutive positions (IC = 4096/N lines for
// powers of two >= 256, 16 below), so with ld = 16/IC (mod 16) its 16
// accesses fall on distinct bank pairs; other lengths take an odd stride.
__host__ __device__ __forceinline__ int line_ld(int N) {
  const int base = N + N / 8;
  if ((N & (N - 1)) != 0) return base | 1;
  if (N < 256) return base + 1;
  const int want = (N / 256) & 15;  // 16 / IC mod 16
  return base + ((want - base % 16) + 16) % 16;
}
__device__ __forceinline__ int swz(int x) { return x + (x >> 3); }

template <class C>
__device__ __forceinline__ C mul_mi(C a, bool inverse) {  // a * (-i), or a * (+i) for the inverse
  C r;
  if (!inverse) { r.x = a.y; r.y = -a.x; } else { r.x = -a.y; r.y = a.x; }
  return r;
}

// 2-, 4- and 8-point DFTs in registers, y_k = sum_n x_n exp(-+2 pi i n k / R).
template <class C>
__device__ __forceinline__ void dft2(C* v) {
  const C t = v[0];
  v[0] = cadd(t, v[1]);
  v[1] = csub(t, v[1]);
}
template <class C>
__device__ __forceinline__ void dft4(C& x0, C& x1, C& x2, C& x3, bool inverse) {
  const C a0 = cadd(x0, x2), a1 = csub(x0, x2);
  const C b0 = cadd(x1, x3), b1 = mul_mi(csub(x1, x3), inverse);
  x0 = cadd(a0, b0);
  x2 = csub(a0, b0);
  x1 = cadd(a1, b1);
  x3 = csub(a1, b1);
}
template <class C>
__device__ __forceinline__ void dft8(C* v, bool inverse) {
  // radix-2 decimation in time over two 4-point DFTs
  C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  C o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4(e0, e1, e2, e3, inverse);
  dft4(o0, o1, o2, o3, inverse);
  using R = decltype(o1.x);
  const R h = (R)0.70710678118654752440;  // 1/sqrt(2)
  C t1, t3;
  if (!inverse) {  // W8 = (1-i)/sqrt2, W8^3 = (-1-i)/sqrt2
    t1.x = (o1.x + o1.y) * h; t1.y = (o1.y - o1.x) * h;
    t3.x = (o3.y - o3.x) * h; t3.y = -(o3.x + o3.y) * h;
  } else {         // conjugates
    t1.x = (o1.x - o1.y) * h; t1.y = (o1.x + o1.y) * h;
    t3.x = -(o3.x + o3.y) * h; t3.y = (o3.x - o3.y) * h;
  }
  const C t2 = mul_mi(o2, inverse);
  v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
  v[1] = cadd(e1, t1); v[5] = csub(e1, t1);
  v[2] = cadd(e2, t2); v[6] = csub(e2, t2);
  v[3] = cadd(e3, t3); v[7] = csub(e3, t3);
}

// One radix-R pass of the Stockham autosort FFT over all lines, in place:
// every thread reads its items (R values each, stride N/R), twiddles them by
// exp(-+2 pi i (j mod Ns) r / (Ns R)), transforms, and after a barrier
// writes them to (j div Ns) Ns R + (j mod Ns) + r Ns.  Input and output are
// in natural order.  Needs nlines * N <= 16 * kFftThreads (the FFT kernels'
// block size).  When lgN, lgNs and nlines are compile-time constants (the
// kernels instantiated for one length) all index arithmetic folds away.
template <class C, int R>
__device__ __forceinline__ void stockham_pass(C* buf, int nlines, int lgN, int lgNs, const C* __restrict__ tw,
                                              bool inverse) {
  constexpr int MAXI = 16 / R;
  constexpr int lgR = R == 8 ? 3 : (R == 4 ? 2 : 1);
  const int N = 1 << lgN;
  const int lg_per = lgN - lgR;              // per_line = N / R
  const int per_line = 1 << lg_per;
  const int total = nlines << lg_per;
  const int ld = line_ld(N);
  const int lg_tw = lgN - lgNs - lgR;        // twiddle step N / (Ns R)
  const int ns_mask = (1 << lgNs) - 1;
  C v[MAXI][R];
#pragma unroll
  for (int it = 0; it < MAXI; ++it) {
    const int b = threadIdx.x + it * kFftThreads;
    if (b < total) {
      const int l = b >> lg_per;
      const int j = b & (per_line - 1);
      const C* line = buf + l * ld;
#pragma unroll
      for (int r = 0; r < R; ++r) v[it][r] = line[swz(j + r * per_line)];
      if (lgNs > 0) {
        const int k = j & ns_mask;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          C w = tw[(k * r) << lg_tw];
          if (inverse) w.y = -w.y;
          v[it][r] = cmul(v[it][r], w);
        }
      }
      if constexpr (R == 8) dft8(v[it], inverse);
      else if constexpr (R == 4) dft4(v[it][0], v[it][1], v[it][2], v[it][3], inverse);
      else dft2(v[it]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < MAXI; ++it) {
    const int b = threadIdx.x + it * kFftThreads;
    if (b < total) {
      const int l = b >> lg_per;
      const int j = b & (per_line - 1);
      const int k = j & ns_mask;
      const int base = ((j - k) << lgR) + k;
      C* line = buf + l * ld;
#pragma unroll
      for (int r = 0; r < R; ++r) line[swz(base + (r << lgNs))] = v[it][r];
    }
  }
  __syncthreads();
}

// Power-of-two N: radix-8 passes, then one radix-4 or radix-2 pass.
template <class C>
__device__ __forceinline__ void fft_lines_pow2(C* buf, int nlines, int N, const C* __restrict__ tw, bool inverse) {
  const int lgN = __ffs(N) - 1;
  int lgNs = 0;
#pragma unroll
  for (; lgNs + 3 <= lgN; lgNs += 3) stockham_pass<C, 8>(buf, nlines, lgN, lgNs, tw, inverse);
  if (lgNs + 2 == lgN) stockham_pass<C, 4>(buf, nlines, lgN, lgNs, tw, inverse);
  else if (lgNs + 1 == lgN) stockham_pass<C, 2>(buf, nlines, lgN, lgNs, tw, inverse);
}

// e -> (e / d, e % d) with a shift and a mask when d is a power of two
// (the usual case: line counts are powers of two, and so are most N).
__device__ __forceinline__ void split_idx(int e, int d, int& q, int& r) {
  if ((d & (d - 1)) == 0) {
    const int lg = __ffs(d) - 1;
    q = e >> lg;
    r = e & (d - 1);
  } else {
    q = e / d;
    r = e - q * d;
  }
}

// Lengths that are not powers of two: direct sums out[m] = sum_n w^(mn)
// in[n], n ascending, both line sets in the swizzled layout.  A thread takes
// TM outputs of one line, m = m0 + q G, so that one input load serves TM
// products and consecutive threads read consecutive lines at one position
// with the same twiddles (broadcasts); the twiddles are staged in shared
// memory, conjugated for the inverse.  One output per thread, with its own
// input and global twiddle loads and index, ran at a tenth of the FP64 pipe.
// Measured, one y-FFT: 36 us at 96x96x150 (FP64; 113 before), 37 at
// 150x120x90 (FP32; 105 before); lengths without such a divisor (dft_any), one
// solve: 127x127x40 275 us (FP64; 608), FP32 form 410 (506), 997x48x30 1348
// (3167) and 2068 (3883).
__device__ __forceinline__ double mul_add(double a, double b, double c, double d, double acc) {  // acc + (a b + c d)
  return __dadd_rn(acc, __fma_rn(a, b, __dmul_rn(c, d)));
}
__device__ __forceinline__ float mul_add(float a, float b, float c, float d, float acc) {
  return __fadd_rn(acc, __fmaf_rn(a, b, __fmul_rn(c, d)));
}
// acc + w x, each product's rounding as it always was, the two directions' too
template <class C, bool INV>
__device__ __forceinline__ void dft_term(C& acc, C w, C x) {
  acc.x = mul_add(w.x, x.x, -w.y, x.y, acc.x);
  acc.y = INV ? mul_add(w.x, x.y, w.y, x.x, acc.y) : mul_add(w.y, x.x, w.x, x.y, acc.y);
}

// N = TM G: with n = n0 + r, n0 a multiple of TM, the twiddle of output q is
// number m0 n + G (q r mod TM) mod N.  The table holds row[b][c] = number
// b + G c, so the TM twiddles of an input are one row, and which output takes
// which is known at compile time: the index is one step per input instead of
// one per product.
template <class C, int TM, bool INV>
__device__ __forceinline__ void dft_rows(const C* in, C* out, C* table, int nlines, int N, const C* __restrict__ tw) {
  const int ld = line_ld(N), G = N / TM;
  for (int e = threadIdx.x; e < N * TM; e += kFftThreads) {
    const int b = e / TM, m = b + (e - b * TM) * G;
    C w = tw[m < N ? m : m - N];
    if (INV) w.y = -w.y;
    table[e] = w;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nlines * G; e += kFftThreads) {
    const int m0 = e / nlines, l = e - m0 * nlines;
    C acc[TM];
#pragma unroll
    for (int q = 0; q < TM; ++q) acc[q] = czero<C>();
    const C* line = in + l * ld;
    int b = 0;
    for (int n0 = 0; n0 < N; n0 += TM) {
#pragma unroll
      for (int r = 0; r < TM; ++r) {
        const C x = line[swz(n0 + r)];
        C w[TM];
#pragma unroll
        for (int c = 0; c < TM; ++c) w[c] = table[b * TM + c];
#pragma unroll
        for (int q = 0; q < TM; ++q) dft_term<C, INV>(acc[q], w[(q * r) % TM], x);
        b += m0;
        if (b >= N) b -= N;
      }
    }
#pragma unroll
    for (int q = 0; q < TM; ++q) out[l * ld + swz(m0 + q * G)] = acc[q];
  }
  __syncthreads();
}

// Any N: G = N / TM rounded up, an index per output.  An output past the last
// (m = m0 + q G >= N) computes number m - N and is not stored.
template <class C, int TM, bool INV>
__device__ __forceinline__ void dft_any(const C* in, C* out, C* stw, int nlines, int N, const C* __restrict__ tw) {
  const int ld = line_ld(N), G = (N + TM - 1) / TM;
  for (int m = threadIdx.x; m < N; m += kFftThreads) {
    C w = tw[m];
    if (INV) w.y = -w.y;
    stw[m] = w;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nlines * G; e += kFftThreads) {
    const int m0 = e / nlines, l = e - m0 * nlines;
    C acc[TM];
    int idx[TM], step[TM];
#pragma unroll
    for (int q = 0; q < TM; ++q) {
      const int m = m0 + q * G;
      acc[q] = czero<C>();
      idx[q] = 0;
      step[q] = m < N ? m : m - N;
    }
    const C* line = in + l * ld;
#pragma unroll 4
    for (int n = 0; n < N; ++n) {
      const C x = line[swz(n)];
#pragma unroll
      for (int q = 0; q < TM; ++q) {
        dft_term<C, INV>(acc[q], stw[idx[q]], x);
        idx[q] += step[q];
        if (idx[q] >= N) idx[q] -= N;
      }
    }
#pragma unroll
    for (int q = 0; q < TM; ++q) {
      const int m = m0 + q * G;
      if (m < N) out[l * ld + swz(m)] = acc[q];
    }
  }
  __syncthreads();
}

// The kernels' LGN beside the compile-time lengths: any length, or the few
// points of dft_any with two outputs (in kernels of its own: beside the others,
// inlined or called, it changed the allocation of their registers; precision
// form, one solve of 190x190x40, kernels: 471 us, 479 with it called, 466
// without; all of dft_any apart: 483).
constexpr int kFftRuntime = 0, kFftShort = -1;

template <class C, bool INV, bool SHORT>
__device__ __forceinline__ void dft_lines(const C* in, C* out, C* table, int nlines, int N, int tm,
                                          const C* __restrict__ tw) {
  if constexpr (SHORT) {
    dft_any<C, 2, INV>(in, out, table, nlines, N, tw);
    return;
  }
  switch (tm) {
    case 4: dft_rows<C, 4, INV>(in, out, table, nlines, N, tw); break;
    case 5: dft_rows<C, 5, INV>(in, out, table, nlines, N, tw); break;
    case 6: dft_rows<C, 6, INV>(in, out, table, nlines, N, tw); break;
    case 8: dft_rows<C, 8, INV>(in, out, table, nlines, N, tw); break;
    case 10: dft_rows<C, 10, INV>(in, out, table, nlines, N, tw); break;
    default: dft_any<C, 6, INV>(in, out, table, nlines, N, tw); break;
  }
}

// Transform the lines in `in`; returns where the result is.
template <class C, bool SHORT>
__device__ __forceinline__ C* fft_lines(C* in, int nlines, int maxlines, int N, const C* __restrict__ tw,
                                        int tm, bool inverse) {
  if constexpr (!SHORT) {
    if (is_pow2(N)) {
      fft_lines_pow2<C>(in, nlines, N, tw, inverse);
      return in;
    }
  }
  C* out = in + (size_t)maxlines * line_ld(N);
  C* table = out + (size_t)maxlines * line_ld(N);
  if (inverse) dft_lines<C, true, SHORT>(in, out, table, nlines, N, tm, tw);
  else dft_lines<C, false, SHORT>(in, out, table, nlines, N, tm, tw);
  return out;
}

struct PArgs {
  const double* rho0;
  const double* rho0_half;
  const double* alpha0;
  const double* alpha0_half;
  double* u;
  double* v;
  double* w;
  double* div;
  double* p;
  double* partial;
  double* mean;
  const double2* twx;
  const double2* twy;
  const float2* twxf;
  const float2* twyf;
  const double* kx2;
  const double* ky2;
  void* spec;     // double2 (plain form) or float2 (precision form) W[k][j][i]
  double* scr;
  // sharded solves (pressure_shard): the x-FFT reads the right-hand side from
  // a dense [i][j][k] interior array, the inverse x-FFT writes the result to
  // one, and the Thomas solve of a slab of j rows starts at global row j0
  const double* src_dense;
  double* dst_dense;
  int j0;
  int tmx, tmy;  // outputs per thread of a direct transform along x and y (direct_outputs)
};

template <class C> __device__ __forceinline__ const C* twx_of(const PArgs& a);
template <> __device__ __forceinline__ const double2* twx_of<double2>(const PArgs& a) { return a.twx; }
template <> __device__ __forceinline__ const float2* twx_of<float2>(const PArgs& a) { return a.twxf; }
template <class C> __device__ __forceinline__ const C* twy_of(const PArgs& a);
template <> __device__ __forceinline__ const double2* twy_of<double2>(const PArgs& a) { return a.twy; }
template <> __device__ __forceinline__ const float2* twy_of<float2>(const PArgs& a) { return a.twyf; }

// ---- line FFTs of compile-time lengths 2^LG, LG = 5 .. 10 --------------------
// LINES lines in shared memory, LINES N / 8 threads, one radix-8 item (8
// values) per thread.  64 registers a thread at 512 threads keep 1024 threads
// on an SM in FP64, twice what 16 values per thread allowed, and these
// kernels are bound by the latency of their loads and of the passes.  The
// first pass takes its inputs and the last one leaves its results where the
// kernel says (global memory for the y-FFTs and the inverse x-FFT), so a
// line crosses shared memory once per pass instead of twice.  Measured at
// 256x256x128, FP64: forward x-FFT 155 -> 108 us, y-FFTs 63 and 53 -> 33 and
// 29, inverse x-FFT 67 -> 49; FP32 at 512x512x256: y-FFT 240 -> 150.
// Line stride: consecutive threads take consecutive lines at one position
// (8 of 16 bytes or 16 of 8 bytes make a phase of a shared-memory access), so
// the stride is odd where a phase holds one position and 2 or 4 where it
// holds 2 or 4 consecutive ones: free of bank conflicts.
template <class C, int LG>
struct Ct {
  static constexpr int N = 1 << LG;
  static constexpr int LINES = ct_lines(LG);
  static constexpr int LGL = LINES == 16 ? 4 : (LINES == 8 ? 3 : 2);
  static constexpr int NT = LINES * N / 8;
  static constexpr int PHASE = 128 / (int)sizeof(C);
  static constexpr int LD = N + N / 8 + (LINES >= PHASE ? 1 : PHASE / LINES);
  static constexpr int LGLAST = LG % 3 == 0 ? 3 : LG % 3;  // radix of the last pass (radix 8 before it)
  static constexpr size_t SMEM = (size_t)LINES * LD * sizeof(C);
  static __device__ __forceinline__ int at(int l, int x) { return l * LD + swz(x); }
};

// One radix-2^LGR pass of the Stockham FFT after LGNS bits are done: load(l,
// x, r) gives input x of line l, store(l, x, value) takes output x; SYNC: a
// barrier between the last load and the first store (both in the buffer).
// LFAST: consecutive threads take consecutive lines, else positions.
template <class C, int LG, int LGR, int LGNS, bool SYNC, bool LFAST, class Load, class Store>
__device__ __forceinline__ void ct_pass(const C* __restrict__ tw, bool inverse, Load load, Store store) {
  using T = Ct<C, LG>;
  constexpr int R = 1 << LGR, IT = 8 / R, LGPER = LG - LGR;
  C v[IT][R];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int b = threadIdx.x + it * T::NT;
    const int l = LFAST ? b & (T::LINES - 1) : b >> LGPER;
    const int j = LFAST ? b >> T::LGL : b & ((1 << LGPER) - 1);
#pragma unroll
    for (int r = 0; r < R; ++r) v[it][r] = load(l, j + (r << LGPER));
    if constexpr (LGNS > 0) {
      const int k = j & ((1 << LGNS) - 1);
#pragma unroll
      for (int r = 1; r < R; ++r) {
        C w = tw[(k * r) << (LG - LGNS - LGR)];
        if (inverse) w.y = -w.y;
        v[it][r] = cmul(v[it][r], w);
      }
    }
    if constexpr (R == 8) dft8(v[it], inverse);
    else if constexpr (R == 4) dft4(v[it][0], v[it][1], v[it][2], v[it][3], inverse);
    else dft2(v[it]);
  }
  if constexpr (SYNC) __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int b = threadIdx.x + it * T::NT;
    const int l = LFAST ? b & (T::LINES - 1) : b >> LGPER;
    const int j = LFAST ? b >> T::LGL : b & ((1 << LGPER) - 1);
    const int k = j & ((1 << LGNS) - 1);
    const int base = ((j - k) << LGR) + k;
#pragma unroll
    for (int r = 0; r < R; ++r) store(l, base + (r << LGNS), v[it][r]);
  }
}

// All passes: the first from `load`, the last to `store` (TO_BUF: into the
// buffer itself).  The buffer must be free when it is called (FROM_BUF: hold
// the input, synchronised).
template <class C, int LG, bool FROM_BUF, bool TO_BUF, bool LFAST1, class Load, class Store>
__device__ __forceinline__ void ct_fft(C* buf, const C* __restrict__ tw, bool inverse, Load load, Store store) {
  using T = Ct<C, LG>;
  auto get = [&](int l, int x) { return buf[T::at(l, x)]; };
  auto put = [&](int l, int x, C v) { buf[T::at(l, x)] = v; };
  ct_pass<C, LG, 3, 0, FROM_BUF, LFAST1>(tw, inverse, load, put);
  __syncthreads();
  if constexpr (LG >= 7) {
    ct_pass<C, LG, 3, 3, true, true>(tw, inverse, get, put);
    __syncthreads();
  }
  if constexpr (LG == 10) {
    ct_pass<C, LG, 3, 6, true, true>(tw, inverse, get, put);
    __syncthreads();
  }
  ct_pass<C, LG, T::LGLAST, LG - T::LGLAST, TO_BUF, true>(tw, inverse, get, store);
}

// ---- HorizontalMean (ParallelMPI.pyx:196-241) ------------------------------
// Block b sums a contiguous chunk of interior columns for every level (one
// thread per level, four interleaved accumulators for memory-level
// parallelism); the partition and the order of the sums are fixed, so the
// mean is deterministic.
__global__ void hmean_partial(Geo g, const double* __restrict__ w, double* __restrict__ partial) {
  const long long nl0 = g.n0 - 2 * g.gw, nl1 = g.n1 - 2 * g.gw;
  const long long ncol = nl0 * nl1;
  const long long per = (ncol + gridDim.x - 1) / gridDim.x;
  const long long c0 = (long long)blockIdx.x * per;
  const long long c1 = min(ncol, c0 + per);
  // the chunk's first column, then a walk along j wrapping to the next i
  // (no index division per element)
  const long long i0 = g.gw + c0 / nl1, j0 = g.gw + c0 % nl1;
  for (long long k = threadIdx.x; k < g.n2; k += blockDim.x) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    long long off = i0 * g.is + j0 * g.js + k;
    long long j = j0;
    long long c = c0;
    for (; c + 3 < c1; c += 4) {
      double v[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        v[m] = w[off];
        off += g.js;
        if (++j == g.gw + nl1) {
          j = g.gw;
          off += g.is - nl1 * g.js;
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) s[m] += v[m];
    }
    for (; c < c1; ++c) {
      s[0] += w[off];
      off += g.js;
      if (++j == g.gw + nl1) {
        j = g.gw;
        off += g.is - nl1 * g.js;
      }
    }
    partial[(long long)blockIdx.x * g.n2 + k] = (s[0] + s[1]) + (s[2] + s[3]);
  }
}

// One block per level: each thread sums a fixed strided subset of the
// partials, then a fixed-order tree in shared memory (deterministic).
__global__ void hmean_final(Geo g, const double* __restrict__ partial, double* __restrict__ mean, int np,
                            double n_horizontal_i) {
  __shared__ double red[256];
  const long long k = blockIdx.x;
  double s = 0.0;
  for (int b = threadIdx.x; b < np; b += blockDim.x) s += partial[(long long)b * g.n2 + k];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) mean[k] = red[0] * n_horizontal_i;
}

// The horizontal sums of a field in the reference's order, for callers
// without scratch memory (pb_horizontal_sums) and for few columns: one chain
// of rounded additions per level.  A block owns 32 levels, one lane each.  Warp 0 only adds: it walks a tile
// of kSerialTile columns in shared memory, one dependent addition per column,
// while the other 31 warps load the next tile (kSerialPer columns each, all
// loads in flight at once) into the other half of a double buffer.
constexpr int kSerialWarps = 32;
constexpr int kSerialPer = 12;
constexpr int kSerialTile = (kSerialWarps - 1) * kSerialPer;  // columns per tile
constexpr int kSerialLd = 33;  // doubles per column in the tile (odd: no bank conflicts)
__global__ void __launch_bounds__(kSerialWarps * 32, 1) hmean_serial(Geo g, const double* __restrict__ w,
                                                                     double* __restrict__ mean,
                                                                     double n_horizontal_i) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* tile = reinterpret_cast<double*>(smraw);  // [2][kSerialTile][kSerialLd]
  const int nl1 = (int)(g.n1 - 2 * g.gw);
  const int ncol = (int)(g.n0 - 2 * g.gw) * nl1;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long k = (long long)blockIdx.x * 32 + lane;
  const bool kok = k < g.n2;
  const int ntiles = (ncol + kSerialTile - 1) / kSerialTile;
  auto produce = [&](int t) {
    double v[kSerialPer];
#pragma unroll
    for (int q = 0; q < kSerialPer; ++q) {
      const int col = t * kSerialTile + (wid - 1) * kSerialPer + q;
      v[q] = 0.0;
      if (col < ncol && kok) {
        const int i = col / nl1, j = col - (col / nl1) * nl1;
        v[q] = w[(g.gw + i) * g.is + (g.gw + j) * g.js + k];
      }
    }
    double* dst = tile + (t & 1) * kSerialTile * kSerialLd + (wid - 1) * kSerialPer * kSerialLd + lane;
#pragma unroll
    for (int q = 0; q < kSerialPer; ++q) dst[q * kSerialLd] = v[q];
  };
  double s = 0.0;
  if (wid > 0) produce(0);
  __syncthreads();
  for (int t = 0; t < ntiles; ++t) {
    if (wid > 0) {
      if (t + 1 < ntiles) produce(t + 1);
    } else {
      const double* cur = tile + (t & 1) * kSerialTile * kSerialLd + lane;
      const int nc = min(kSerialTile, ncol - t * kSerialTile);
      if (nc == kSerialTile) {
#pragma unroll 12
        for (int c = 0; c < kSerialTile; ++c) s = add_rn(s, cur[c * kSerialLd]);
      } else {
        for (int c = 0; c < nc; ++c) s = add_rn(s, cur[c * kSerialLd]);
      }
    }
    __syncthreads();
  }
  if (wid == 0 && kok) mean[k] = mul_rn(s, n_horizontal_i);
}

static int launch_hmean_serial(const Geo& g, const double* w, double* mean, double scale, cudaStream_t st) {
  const size_t sm = 2 * (size_t)kSerialTile * kSerialLd * sizeof(double);
  PB_CUDA_TRY(cudaFuncSetAttribute(hmean_serial, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  hmean_serial<<<ceil_div(g.n2, 32), kSerialWarps * 32, sm, st>>>(g, w, mean, scale);
  pb_note_launch();
  return PB_OK;
}

// Plain form: HorizontalMean in the reference's order (ParallelMPI.pyx:219-
// 226).  Each level's sum is one chain of rounded additions over the
// interior columns, i outer and j inner, which no reordering may change:
// w's horizontal mean cancels, and the solve subtracts it from every cell.
// One lane adding the chain (hmean_serial) is bound by the latency of a
// dependent FP64 addition, ~20 cycles a column.  Here the chain is cut into
// segments of about L columns that run side by side, each from a predicted
// start, and the true sum is moved through their results with the same bits
// as the chain:
//
//   * The prediction p of a segment's start comes from parallel sums of the
//     columns before it (hsum_parts, hsum_prefix).  It misses the true value
//     s by some units u in p's last place.
//   * Two chains of additions of the same columns whose starts differ by a
//     multiple d of 2 u' (u' the rounding unit of every partial sum they
//     pass through; the 2 keeps ties to even alike) stay exactly d apart as
//     long as both are in the same binade after every addition: there the
//     rounding is a fixed grid.  So kHmChains = 16 chains start at p, p + u,
//     ..., p + 15u (hsum_chains); s is a multiple of 16u away from one of
//     them, which covers sums that grow by up to three binades (u' <= 8u),
//     and the true sum at the segment's end is that chain's end plus s minus
//     its start (hsum_walk).
//   * Two more chains start kHmSlack units below and above p.  Rounded
//     addition is monotone, so a start within kHmSlack / 2 stays between
//     them; when the two have equal sign and exponent after an addition, so
//     has everything between.
//   * After an addition that leaves the two in different binades (a sum that
//     cancels: w a wave along y passes zero at the end of every row) the
//     distances stay as they are if nothing between was rounded: all starts
//     and the column are multiples of a unit g, and the larger result is below
//     2^53 g.  g is the unit of the binade that they were in last, and at most
//     that of the columns added since.
//   * Where neither holds (a sum that starts small and grows, or passes a
//     power of two within the slack), the walk adds the segment's columns one
//     by one.  A segment therefore begins at the largest |p| among the first
//     kHmHead columns around its nominal start: few sums start small there.
//     s == p takes the first chain as it is.
//
// The walk (one warp per level, ~170 cycles a segment) and the two reads of w
// bound it.  Measured, FP64 form, the mean in one solve: 256x256 columns of
// 134 levels 95 us against 748 for the one-lane chain, 96x96x158 31 (108),
// 64x64x81 21 (50).  A whole solve with w a sine along y, where the exact
// additions count: 64x64x64 90 us, 143 without them (129 with the one-lane
// chain), 256x256x64 698 (1160, 1153).  Segments of 128 columns; 64 on grids of
// up to 8192 columns, where the walk is short and more segments fill the GPU.
// Up to 1280 columns hmean_serial stays the faster one (15 us at 32x32 against
// 20 for the four launches).
constexpr int kHmChains = 16;
constexpr int kHmGrow = 3;  // binades a segment's sums may grow by: 2^(kHmGrow + 1) = kHmChains
constexpr long long kHmSlack = 1 << 14;
constexpr int kHmHead = 16;
constexpr int kHmRow = kHmChains + 2;  // a segment's record: the ends, p, flag and bounds

__device__ __forceinline__ double from_bits(long long b) { return __longlong_as_double(b); }

// The interior columns of a level in the reference's order, from column c on.
struct ColumnWalk {
  const double* src;
  long long js, wrap;
  int j, nl1;
  __device__ __forceinline__ ColumnWalk(const Geo& g, const double* w, int c, long long k) {
    nl1 = (int)(g.n1 - 2 * g.gw);
    const int i = c / nl1;
    j = c - i * nl1;
    js = g.js;
    wrap = g.is - (long long)nl1 * g.js;
    src = w + (g.gw + i) * g.is + (g.gw + j) * g.js + k;
  }
  // the next n columns, +0 (which changes no sum) past the `left` that exist
  template <int n>
  __device__ __forceinline__ void take(double (&x)[n], int left) {
#pragma unroll
    for (int q = 0; q < n; ++q) {
      x[q] = q < left ? *src : 0.0;
      src += js;
      if (++j == nl1) {
        j = 0;
        src += wrap;
      }
    }
  }
};

// Parallel sum of every nominal segment; a warp takes one segment of 32 levels.
template <int L>
__global__ void __launch_bounds__(256) hsum_parts(Geo g, const double* __restrict__ w, double* __restrict__ pre,
                                                  int nsegs) {
  const int seg = blockIdx.x * 8 + (threadIdx.x >> 5);
  const long long k = (long long)blockIdx.y * 32 + (threadIdx.x & 31);
  if (seg >= nsegs || k >= g.n2) return;
  const int left = (int)((g.n0 - 2 * g.gw) * (g.n1 - 2 * g.gw)) - seg * L;
  ColumnWalk cw(g, w, seg * L, k);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
  for (int c = 0; c < L; c += 16) {
    double x[16];
    cw.take(x, left - c);
#pragma unroll
    for (int q = 0; q < 16; ++q) s[q & 3] += x[q];
  }
  pre[(long long)seg * g.n2 + k] = (s[0] + s[1]) + (s[2] + s[3]);
}

// The sums of the segments before each segment, in place: a block takes 32
// levels, each warp a run of segments.
__global__ void __launch_bounds__(1024) hsum_prefix(long long n2, double* __restrict__ pre, int nsegs) {
  __shared__ double run[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long k = (long long)blockIdx.x * 32 + lane;
  const int per = (nsegs + 31) / 32, s0 = min(w * per, nsegs), s1 = min(s0 + per, nsegs);
  double t = 0.0;
  if (k < n2) {
#pragma unroll 8
    for (int q = s0; q < s1; ++q) t += pre[q * n2 + k];
  }
  run[w][lane] = t;
  __syncthreads();
  double before = 0.0;
  for (int q = 0; q < w; ++q) before += run[q][lane];
  if (k < n2) {
#pragma unroll 8
    for (int q = s0; q < s1; ++q) {
      const double v = pre[q * n2 + k];
      pre[q * n2 + k] = before;
      before += v;
    }
  }
}

// Where a segment begins: after the first b of its nominal columns x, p the
// prediction there.  (Both segments that meet there evaluate this, on the
// same values.)
__device__ __forceinline__ void hm_begin(double& p, int& b, const double (&x)[kHmHead]) {
  double run = p;
  b = 0;
#pragma unroll
  for (int q = 0; q + 1 < kHmHead; ++q) {
    run = add_rn(run, x[q]);
    if (fabs(run) > fabs(p)) {
      p = run;
      b = q + 1;
    }
  }
}

template <int L>
__global__ void __launch_bounds__(64, 8) hsum_chains(Geo g, const double* __restrict__ w,
                                                      const double* __restrict__ pre, double* __restrict__ rec,
                                                      int nsegs) {
  const int seg = blockIdx.x * 2 + (threadIdx.x >> 5);
  const long long k = (long long)blockIdx.y * 32 + (threadIdx.x & 31);
  if (seg >= nsegs || k >= g.n2) return;
  const int left = (int)((g.n0 - 2 * g.gw) * (g.n1 - 2 * g.gw)) - seg * L;
  ColumnWalk cw(g, w, seg * L, k);
  double x[kHmHead], y[kHmHead];
  cw.take(x, left);
  cw.take(y, left - kHmHead);
  double p = pre[(long long)seg * g.n2 + k];
  int b = 0;
  if (seg > 0) hm_begin(p, b, x);
  const long long pb = __double_as_longlong(p);
  double c[kHmChains];
#pragma unroll
  for (int r = 0; r < kHmChains; ++r) c[r] = from_bits(pb + r);
  double lo = from_bits(pb - kHmSlack), hi = from_bits(pb + kHmSlack);
  // (high words, without branches, between the additions of the chains)
  constexpr int kExp = 0x7ff00000, kMag = 0x7fffffff;
  int unit = __double2hiint(lo) & kExp;  // the exponent whose unit all values are multiples of
  bool kept = ((__double2hiint(lo) ^ __double2hiint(hi)) & ~0xfffff) == 0;
  int top = 0;  // the largest magnitude passed through
  auto add = [&](double v) {
#pragma unroll
    for (int r = 0; r < kHmChains; ++r) c[r] = add_rn(c[r], v);
    lo = add_rn(lo, v);
    hi = add_rn(hi, v);
    const int l = __double2hiint(lo), h = __double2hiint(hi), hv = __double2hiint(v) & kMag;
    const int m = max(l & kMag, h & kMag);
    const bool same = ((l ^ h) & ~0xfffff) == 0;
    const int u = (hv | __double2loint(v)) != 0 ? min(unit, hv & kExp) : unit;
    kept = kept && (same || m <= (u | 0xfffff));
    unit = same ? m & kExp : u;
    top = max(top, m);
  };
#pragma unroll
  for (int q = 0; q < kHmHead; ++q) add(q >= b ? x[q] : 0.0);
#pragma unroll 1
  for (int n = kHmHead; n < L; n += kHmHead) {
    // y holds columns n .. n + 15; the ones after them (the last time: the
    // next segment's first) are loaded meanwhile
    cw.take(x, left - n - kHmHead);
#pragma unroll
    for (int q = 0; q < kHmHead; ++q) add(y[q]);
#pragma unroll
    for (int q = 0; q < kHmHead; ++q) y[q] = x[q];
  }
  int bn = 0;
  if (seg + 1 < nsegs) {
    double pn = pre[(long long)(seg + 1) * g.n2 + k];
    hm_begin(pn, bn, y);
#pragma unroll
    for (int q = 0; q + 1 < kHmHead; ++q) add(q < bn ? y[q] : 0.0);
  }
  const int e0 = (int)(pb >> 52) & 0x7ff;
  top >>= 20;
  const long long ok = kept && top <= e0 + kHmGrow && top < 0x7fe;
  double2* row = reinterpret_cast<double2*>(rec + ((long long)k * nsegs + seg) * kHmRow);
#pragma unroll
  for (int r = 0; r < kHmChains; r += 2) row[r / 2] = make_double2(c[r], c[r + 1]);
  row[kHmChains / 2] = make_double2(p, from_bits(ok | (long long)b << 8 | (long long)bn << 16));
}

// s and the columns c0 .. c1 - 1 of a level, one by one (a warp; out of line,
// so that the walk's code stays in the instruction cache).
__device__ __noinline__ double hm_add_columns(double s, const double* w, long long is, long long js, int nl1, int c0,
                                              int c1) {
  const int lane = threadIdx.x & 31;
  for (int cb = c0; cb < c1; cb += 128) {
    double x[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int c = cb + h * 32 + lane;
      x[h] = c < c1 ? w[c / nl1 * is + c % nl1 * js] : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      if (cb + h * 32 >= c1) break;
#pragma unroll
      for (int m = 0; m < 32; ++m) s = add_rn(s, __shfl_sync(0xffffffffu, x[h], m));
    }
  }
  return s;
}

// One warp per level moves its sum through the segments, the same in every
// lane.  The records come through shared memory, kWalkRows at a time, the
// next ones copied (cp.async) while these are used.
constexpr int kWalkRows = 32;
template <int L>
__global__ void __launch_bounds__(32) hsum_walk(Geo g, const double* __restrict__ w, const double* __restrict__ rec,
                                                double* __restrict__ mean, double n_horizontal_i, int nsegs) {
  __shared__ __align__(16) double buf[2][kWalkRows * kHmRow];
  const int lane = threadIdx.x;
  const long long k = blockIdx.x;
  const int ncol = (int)((g.n0 - 2 * g.gw) * (g.n1 - 2 * g.gw));
  const double* row = rec + (long long)k * nsegs * kHmRow;
  auto copy = [&](int q0) {  // records q0 .. of the level
    const int n = min(kWalkRows, nsegs - q0) * kHmRow / 2;  // 16-byte pieces
    const unsigned dst = (unsigned)__cvta_generic_to_shared(buf[(q0 / kWalkRows) & 1]);
    for (int e = lane; e < n; e += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + e * 16),
                   "l"(row + (long long)q0 * kHmRow + 2 * e)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy(0);
  double s = 0.0;
  for (int q0 = 0; q0 < nsegs; q0 += kWalkRows) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    if (q0 + kWalkRows < nsegs) copy(q0 + kWalkRows);
    const double* r0 = buf[(q0 / kWalkRows) & 1];
    const int n = min(kWalkRows, nsegs - q0);
    for (int q = 0; q < n; ++q) {
      const double* e = r0 + q * kHmRow;
      const long long pb = __double_as_longlong(e[kHmChains]);
      const long long info = __double_as_longlong(e[kHmChains + 1]);
      const long long d = __double_as_longlong(s) - pb;
      const int r = (int)d & (kHmChains - 1);
      const bool near = (info & 1) && (unsigned long long)(d + kHmSlack / 2) <= (unsigned long long)kHmSlack;
      if (near) {
        s = add_rn(e[r], sub_rn(s, from_bits(pb + r)));  // the difference: a multiple of 16u
      } else if (d == 0) {
        s = e[0];
      } else {
        s = hm_add_columns(s, w + g.gw * g.is + g.gw * g.js + k, g.is, g.js, (int)(g.n1 - 2 * g.gw),
                           (q0 + q) * L + (int)((info >> 8) & 0xff), min((q0 + q + 1) * L + (int)(info >> 16), ncol));
      }
    }
    __syncwarp();
  }
  if (lane == 0) mean[k] = mul_rn(s, n_horizontal_i);
}

template <int L>
static void launch_hsum(const Geo& g, const double* w, double* mean, double scale, double* scratch, cudaStream_t st) {
  const long long ncol = (g.n0 - 2 * g.gw) * (g.n1 - 2 * g.gw);
  const int nsegs = (int)((ncol + L - 1) / L);
  double* rec = scratch;  // first: 16-byte stores
  double* pre = scratch + (long long)nsegs * g.n2 * kHmRow;
  const dim3 grid(ceil_div(nsegs, 8), ceil_div(g.n2, 32));
  hsum_parts<L><<<grid, 256, 0, st>>>(g, w, pre, nsegs);
  hsum_prefix<<<ceil_div(g.n2, 32), 1024, 0, st>>>(g.n2, pre, nsegs);
  hsum_chains<L><<<dim3(ceil_div(nsegs, 2), grid.y), 64, 0, st>>>(g, w, pre, rec, nsegs);
  hsum_walk<L><<<(unsigned)g.n2, 32, 0, st>>>(g, w, rec, mean, scale, nsegs);
  for (int q = 0; q < 4; ++q) pb_note_launch();
}

// scratch: the solve's spectral and Thomas arrays, not yet in use (12 bytes or
// more per column and interior level; the records and prefixes of segments of
// 64 columns take at most 9, ghost levels included: 19 doubles for each of
// at most 1.25 ncol / 64 segments and 3 nz levels).
static int launch_hmean_ordered(const Geo& g, const double* w, double* mean, double scale, double* scratch,
                                 cudaStream_t st) {
  const long long ncol = (g.n0 - 2 * g.gw) * (g.n1 - 2 * g.gw);
  if (ncol <= 1280) {
    return launch_hmean_serial(g, w, mean, scale, st);
  } else if (ncol <= 8192) {
    launch_hsum<64>(g, w, mean, scale, scratch, st);
  } else {
    launch_hsum<128>(g, w, mean, scale, scratch, st);
  }
  return PB_OK;
}

__global__ void zero_ghosts(Geo g, double* __restrict__ f, long long nghost) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nghost; t += stride) {
    long long i, j, k;
    ghost_decode(g, t, i, j, k);
    f[i * g.is + j * g.js + k] = 0.0;
  }
}

// Right-hand side of the forward x-FFT (fft_x_fwd's SRC) and destination of
// the inverse (fft_x_inv's DST).
constexpr int kSrcDivergence = 0, kSrcResidual = 1, kSrcDense = 2;
constexpr int kDstWrite = 0, kDstAccumulate = 1, kDstDense = 2;

// second_order_divergence (PressureSolver.pyx:138-175, d = 0, 1, 2 in order)
// of the cell ijk at level k, w taken after remove_mean_u3 (w - mean[k]).
// Plain form: the reference's divisions by alpha0 in its order, each
// correctly rounded, from the reciprocals 1/alpha0_half[k], 1/alpha0[k] and
// 1/alpha0[k-1] (yh, yf, yd); precision form: multiplications by
// rho0 = 1/alpha0.
// `divide` is set if d may differ from the divisions' (divergence_divided): from
// 2^-500 up to infinity it does not, for an infinity or a NaN among the
// velocities makes it a NaN here, and quotients too small for div_by_normal
// (below 2^-900) are absorbed; nor does a smaller d that the sum before it and
// a dz of that range cancel to.
template <bool PLAIN>
__device__ __forceinline__ double divergence_at(const Geo& g, const PArgs& a, long long ijk, long long k, double yh,
                                                double yf, double yd, bool& divide) {
  const double* __restrict__ U = a.u;
  const double* __restrict__ V = a.v;
  const double* __restrict__ Wv = a.w;
  const double wc = sub_rn(Wv[ijk], a.mean[k]);
  const double wm = sub_rn(Wv[ijk - 1], a.mean[k - 1]);
  if constexpr (PLAIN) {
    const double ah = a.alpha0_half[k];
    double d = 0.0;
    d = add_rn(d, mul_rn(sub_rn(div_by_normal(U[ijk], ah, yh), div_by_normal(U[ijk - g.is], ah, yh)), g.dxi0));
    d = add_rn(d, mul_rn(sub_rn(div_by_normal(V[ijk], ah, yh), div_by_normal(V[ijk - g.js], ah, yh)), g.dxi1));
    const double dz = mul_rn(sub_rn(div_by_normal(wc, a.alpha0[k], yf), div_by_normal(wm, a.alpha0[k - 1], yd)), g.dxi2);
    d = add_rn(d, dz);
    constexpr unsigned kLow = 0x20b00000u, kInf = 0x7ff00000u;  // high words
    const unsigned td = (unsigned)__double2hiint(d) & 0x7fffffffu, tz = (unsigned)__double2hiint(dz) & 0x7fffffffu;
    divide |= !((td - kLow < kInf - kLow) | ((td < kLow) & (tz - kLow < kInf - kLow)));
    return d;
  } else {
    const double rh = a.rho0_half[k];
    return (U[ijk] - U[ijk - g.is]) * rh * g.dxi0 + (V[ijk] - V[ijk - g.js]) * rh * g.dxi1 +
           (wc * a.rho0[k] - wm * a.rho0[k - 1]) * g.dxi2;
  }
}

// The same by divisions.
__device__ __forceinline__ double divergence_divided(const Geo& g, const PArgs& a, long long ijk, long long k) {
  const double ah = a.alpha0_half[k];
  const double wc = sub_rn(a.w[ijk], a.mean[k]), wm = sub_rn(a.w[ijk - 1], a.mean[k - 1]);
  double d = 0.0;
  d = add_rn(d, mul_rn(sub_rn(a.u[ijk] / ah, a.u[ijk - g.is] / ah), g.dxi0));
  d = add_rn(d, mul_rn(sub_rn(a.v[ijk] / ah, a.v[ijk - g.js] / ah), g.dxi1));
  return add_rn(d, mul_rn(sub_rn(wc / a.alpha0[k], wm / a.alpha0[k - 1]), g.dxi2));
}

// The refinement residual div - A p of the cell ijk (level k, kk = k - gw),
// A the operator the spectral solve inverts: second differences in x and y,
// the rows of compute_off_diagonals / compute_diagonal in z.
__device__ __forceinline__ double residual_at(const Geo& g, const PArgs& a, long long ijk, long long k, long long kk,
                                              long long nz) {
  const double* __restrict__ p = a.p;
  const double pc = p[ijk];
  const double lap_h = a.rho0_half[k] * ((p[ijk + g.is] - 2.0 * pc + p[ijk - g.is]) * (g.dxi0 * g.dxi0) +
                                         (p[ijk + g.js] - 2.0 * pc + p[ijk - g.js]) * (g.dxi1 * g.dxi1));
  double vert = 0.0;
  if (kk < nz - 1) vert += a.rho0[k] * (p[ijk + 1] - pc);
  if (kk > 0) vert -= a.rho0[k - 1] * (pc - p[ijk - 1]);
  return a.div[ijk] - (lap_h + vert * (g.dxi2 * g.dxi2));
}

// ---- divergence (or refinement residual) + forward x-FFT --------------------
// block = (interior j, chunk of KC = 2 LC interior levels); smem LC complex
// lines of n0, line p holding levels 2p (real part) and 2p + 1 (imaginary).
// SRC = kSrcDivergence: the right-hand side is second_order_divergence
//   (divergence_at), written to `div`.
// SRC = kSrcResidual: the right-hand side is the residual div - A p of the
//   current pressure (residual_at); used by the iterative refinement of the
//   precision form.
// SRC = kSrcDense: the right-hand side is read from a dense interior array
//   (a slab of levels of a sharded solve).
//
// LGN > 0 instantiates the kernel for N = 2^LGN (KC = 2 ct_lines(LGN)), with
// the compile-time transform; the others take N and KC at run time.
template <class C, int LGN>
__host__ __device__ constexpr int fft_threads() {
  if constexpr (LGN > 0) return Ct<C, LGN>::NT;
  return kFftThreads;
}
// resident blocks per SM the registers are held to: blocks of 512
// threads and FP64 ones of run-time lengths two, FP32 ones of run-time lengths
// three
template <class C, int LGN>
constexpr int fft_blocks() {
  if constexpr (LGN <= 0) return sizeof(C) == 16 ? 2 : 3;
  return LGN >= 8 ? 2 : 1;
}

template <class C, int SRC, int LGN>
__global__ void __launch_bounds__((fft_threads<C, LGN>()), (fft_blocks<C, LGN>())) fft_x_fwd(Geo g, PArgs a, int KCrt) {
  using R = decltype(C().x);
  constexpr bool CT = LGN > 0;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* in = reinterpret_cast<C*>(smraw);
  R* inr = reinterpret_cast<R*>(smraw);
  const int N = CT ? (1 << LGN) : (int)(g.n0 - 2 * g.gw);
  const int KC = CT ? 2 * ct_lines(LGN) : KCrt;
  const int Nh = N / 2 + 1;
  const int nz = (int)(g.n2 - 2 * g.gw);
  const int jl = blockIdx.x;
  const int k0 = blockIdx.y * KC;
  const int kc = min(KC, nz - k0);
  const int lc = (kc + 1) >> 1;
  const long long j = g.gw + jl;
  constexpr int NT = fft_threads<C, LGN>();
  const int ld = CT ? Ct<C, CT ? LGN : 5>::LD : line_ld(N);
  const long long ny = g.n1 - 2 * g.gw;
  double* __restrict__ div = a.div;
  constexpr bool PLAIN = SRC == kSrcDivergence && sizeof(C) == sizeof(double2);
  // reciprocals of the chunk's alpha0_half and (from the level below on) alpha0
  __shared__ double yh[PLAIN ? kMaxKC : 1], yf[PLAIN ? kMaxKC + 1 : 1];
  if constexpr (PLAIN) {
    if ((int)threadIdx.x < kc) yh[threadIdx.x] = 1.0 / a.alpha0_half[g.gw + k0 + threadIdx.x];
    if ((int)threadIdx.x <= kc) yf[threadIdx.x] = 1.0 / a.alpha0[g.gw + k0 - 1 + threadIdx.x];
    __syncthreads();
  }
  bool divide = false;
#pragma unroll 4
  for (int e = threadIdx.x; e < N * KC; e += NT) {
    int kl, il;
    split_idx(e, KC, il, kl);
    const int slot = 2 * ((kl >> 1) * ld + swz(il)) + (kl & 1);
    if (kl >= kc) {  // the imaginary half of an odd chunk's last line
      inr[slot] = (R)0;
      continue;
    }
    const long long k = g.gw + k0 + kl;
    const long long ijk = (g.gw + il) * g.is + j * g.js + k;
    double d;
    if constexpr (SRC == kSrcDivergence) {
      if constexpr (PLAIN)
        d = divergence_at<true>(g, a, ijk, k, yh[kl], yf[kl + 1], yf[kl], divide);
      else
        d = divergence_at<false>(g, a, ijk, k, 0.0, 0.0, 0.0, divide);
      div[ijk] = d;
    } else if constexpr (SRC == kSrcResidual) {
      d = residual_at(g, a, ijk, k, k - g.gw, nz);
    } else {  // a dense interior array (il, jl, k0 + kl)
      d = a.src_dense[((long long)il * ny + jl) * nz + k0 + kl];
    }
    inr[slot] = (R)d;
  }
  if constexpr (PLAIN) {
    // a thread's cells once more, where one needs the divisions (a branch in
    // the loop keeps its loads from running ahead: 11.8 us at 64x64x75, 11.0)
    if (divide) {
#pragma unroll 1
      for (int e = threadIdx.x; e < N * KC; e += NT) {
        int kl, il;
        split_idx(e, KC, il, kl);
        if (kl >= kc) continue;
        const long long ijk = (g.gw + il) * g.is + j * g.js + g.gw + k0 + kl;
        const double d = divergence_divided(g, a, ijk, g.gw + k0 + kl);
        div[ijk] = d;
        inr[2 * ((kl >> 1) * ld + swz(il)) + (kl & 1)] = d;
      }
    }
  }
  __syncthreads();
  const C* res = in;
  if constexpr (CT) {
    using T = Ct<C, LGN>;
    ct_fft<C, LGN, true, true, true>(in, twx_of<C>(a), false, [&](int l, int x) { return in[T::at(l, x)]; },
                                     [&](int l, int x, C v) { in[T::at(l, x)] = v; });
    __syncthreads();
  } else {
    res = fft_lines<C, LGN == kFftShort>(in, lc, KC >> 1, N, twx_of<C>(a), a.tmx, false);
  }
  // separate the two rows of each line; write the columns m = 0..N/2
  C* spec = reinterpret_cast<C*>(a.spec);
  const long long nxy = (long long)Nh * (g.n1 - 2 * g.gw);
  const R half = (R)0.5;
#pragma unroll 4
  for (int e = threadIdx.x; e < Nh * kc; e += NT) {
    const int kl = e / Nh;
    const int m = e - kl * Nh;
    const C* line = res + (kl >> 1) * ld;
    const C z = line[swz(m)];
    const C zr = line[swz(m == 0 ? 0 : N - m)];  // Z[N - m]
    C o;
    if ((kl & 1) == 0) {  // A = (Z[m] + conj Z[N-m]) / 2
      o.x = (z.x + zr.x) * half;
      o.y = (z.y - zr.y) * half;
    } else {              // B = (Z[m] - conj Z[N-m]) / 2i
      o.x = (z.y + zr.y) * half;
      o.y = (zr.x - z.x) * half;
    }
    spec[(long long)(k0 + kl) * nxy + (long long)jl * Nh + m] = o;
  }
}

// ---- y-FFT over W[k][j][m] lines along j, IC columns m per block ----------
// (LGN as for fft_x_fwd: N = 2^LGN and IC = ct_lines(LGN) at compile time.)
template <class C, bool INV, int LGN>
__global__ void __launch_bounds__((fft_threads<C, LGN>()), (fft_blocks<C, LGN>())) fft_y(Geo g, PArgs a, int ICrt) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C* in = reinterpret_cast<C*>(smraw);
  const int Nx = (int)(g.n0 - 2 * g.gw) / 2 + 1;  // stored x-modes
  const int kk = blockIdx.y;
  if constexpr (LGN > 0) {
    using T = Ct<C, LGN>;
    const int i0 = blockIdx.x * T::LINES, ic = Nx - i0;
    C* plane = reinterpret_cast<C*>(a.spec) + (long long)kk * T::N * Nx + i0;
    const double sc = INV ? 1.0 / (double)T::N : 1.0;
    ct_fft<C, LGN, false, false, true>(
        in, twy_of<C>(a), INV, [&](int l, int x) { return l < ic ? plane[x * Nx + l] : czero<C>(); },
        [&](int l, int x, C r) {
          if (INV) {
            r.x *= sc;
            r.y *= sc;
          }
          if (l < ic) plane[x * Nx + l] = r;
        });
    return;
  }
  const int N = (int)(g.n1 - 2 * g.gw);
  const int IC = ICrt;
  const int i0 = blockIdx.x * IC;
  const int ic = min(IC, Nx - i0);
  const int ld = line_ld(N);
  C* plane = reinterpret_cast<C*>(a.spec) + (long long)kk * N * Nx;
#pragma unroll 4
  for (int e = threadIdx.x; e < N * IC; e += kFftThreads) {
    int il, jl;
    split_idx(e, IC, jl, il);
    if (il >= ic) continue;
    in[il * ld + swz(jl)] = plane[(long long)jl * Nx + i0 + il];
  }
  __syncthreads();
  const C* res = fft_lines<C, LGN == kFftShort>(in, ic, IC, N, twy_of<C>(a), a.tmy, INV);
  const double sc = INV ? 1.0 / (double)N : 1.0;
#pragma unroll 4
  for (int e = threadIdx.x; e < N * IC; e += kFftThreads) {
    int il, jl;
    split_idx(e, IC, jl, il);
    if (il >= ic) continue;
    C r = res[il * ld + swz(jl)];
    if (INV) {
      r.x *= sc;
      r.y *= sc;
    }
    plane[(long long)jl * Nx + i0 + il] = r;
  }
}

__device__ __forceinline__ void to_d(double2 c, double& x, double& y) { x = c.x; y = c.y; }
__device__ __forceinline__ void to_d(float2 c, double& x, double& y) { x = c.x; y = c.y; }
template <class C> __device__ __forceinline__ C from_d(double x, double y);
template <> __device__ __forceinline__ double2 from_d<double2>(double x, double y) { return make_double2(x, y); }
template <> __device__ __forceinline__ float2 from_d<float2>(double x, double y) {
  return make_float2((float)x, (float)y);
}

// ---- per-column tridiagonal solve (always FP64 arithmetic) -----------------
// Matrix of PressureFFTParallel.compute_off_diagonals (:100-127) and
// compute_diagonal (:129-148); Thomas algorithm of TDMA.solve applied to the
// real and imaginary parts (the matrix is real, so both share m and scratch).
template <class C>
__global__ void __launch_bounds__(256, sizeof(C) == 8 ? 4 : 2) tdma_kernel(Geo g, PArgs a) {
  const int Nx = (int)(g.n0 - 2 * g.gw) / 2 + 1;  // stored x-modes
  const int Ny = (int)(g.n1 - 2 * g.gw);
  const int nz = (int)(g.n2 - 2 * g.gw);
  const long long ncol = (long long)Nx * Ny;
  const long long col = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= ncol) return;
  const int i = (int)(col % Nx);
  const int j = (int)(col / Nx) + a.j0;  // global row (a slab of rows in a sharded solve)
  C* x = reinterpret_cast<C*>(a.spec) + col;
  double* scr = a.scr + col;
  if (i == 0 && j == 0) {  // mode (0,0) is set to zero (:197-200)
    for (int k = 0; k < nz; ++k) x[(long long)k * ncol] = from_d<C>(0.0, 0.0);
    return;
  }
  const long long gw = g.gw;
  const double dzi = g.dxi2;
  const double kk = a.kx2[i] + a.ky2[j];
  const double* rho0 = a.rho0;
  const double* rho0h = a.rho0_half;
  // row 0 (for a single level the last-row formulas overwrite it, :119-127, :145-146)
  double b, c;
  if (nz > 1) {
    b = sub_rn(mul_rn(rho0h[gw], kk), mul_rn(mul_rn(rho0[gw], dzi), dzi));
    c = mul_rn(mul_rn(dzi, dzi), rho0[gw]);
  } else {
    b = sub_rn(mul_rn(rho0h[gw], kk), mul_rn(mul_rn(rho0[gw - 1], dzi), dzi));
    c = 0.0;
  }
  double s_prev = c / b;
  double xpx, xpy;
  to_d(x[0], xpx, xpy);
  xpx = xpx / b;
  xpy = xpy / b;
  x[0] = from_d<C>(xpx, xpy);
  scr[0] = s_prev;
  // The sweeps walk the levels in batches of kB; the loads of the next batch
  // are issued before the current one is processed, so every thread keeps
  // kB independent loads in flight behind its serial recurrence.
  constexpr int kB = sizeof(C) == 8 ? 4 : 8;  // FP32 spectra: 4 blocks per SM at 64 registers
  C cur[kB], nxt[kB];
#pragma unroll
  for (int m = 0; m < kB; ++m) cur[m] = (1 + m < nz) ? x[(long long)(1 + m) * ncol] : from_d<C>(0.0, 0.0);
  for (int kb = 1; kb < nz; kb += kB) {
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      const int kn = kb + kB + m;
      nxt[m] = (kn < nz) ? x[(long long)kn * ncol] : from_d<C>(0.0, 0.0);
    }
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      const int k = kb + m;
      if (k < nz) {
        const double ak = mul_rn(mul_rn(dzi, dzi), rho0[k + gw - 1]);
        double ck, bk;
        if (k < nz - 1) {
          ck = mul_rn(mul_rn(dzi, dzi), rho0[k + gw]);
          bk = sub_rn(mul_rn(rho0h[k + gw], kk), mul_rn(mul_rn(add_rn(rho0[k + gw], rho0[k + gw - 1]), dzi), dzi));
        } else {
          ck = 0.0;
          bk = sub_rn(mul_rn(rho0h[k + gw], kk), mul_rn(mul_rn(rho0[k + gw - 1], dzi), dzi));
        }
        const double m_ = 1.0 / sub_rn(bk, mul_rn(ak, s_prev));
        s_prev = mul_rn(ck, m_);
        scr[(long long)k * ncol] = s_prev;
        double xkx, xky;
        to_d(cur[m], xkx, xky);
        xkx = mul_rn(sub_rn(xkx, mul_rn(ak, xpx)), m_);
        xky = mul_rn(sub_rn(xky, mul_rn(ak, xpy)), m_);
        x[(long long)k * ncol] = from_d<C>(xkx, xky);
        xpx = xkx;
        xpy = xky;
      }
    }
#pragma unroll
    for (int m = 0; m < kB; ++m) cur[m] = nxt[m];
  }
  // back substitution from the last value, reading the stored sweep values,
  // in batches of kB levels going down
  double scur[kB], snxt[kB];
#pragma unroll
  for (int m = 0; m < kB; ++m) {
    const int k = nz - 2 - m;
    cur[m] = (k >= 0) ? x[(long long)k * ncol] : from_d<C>(0.0, 0.0);
    scur[m] = (k >= 0) ? scr[(long long)k * ncol] : 0.0;
  }
  for (int kb = nz - 2; kb >= 0; kb -= kB) {
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      const int kn = kb - kB - m;
      nxt[m] = (kn >= 0) ? x[(long long)kn * ncol] : from_d<C>(0.0, 0.0);
      snxt[m] = (kn >= 0) ? scr[(long long)kn * ncol] : 0.0;
    }
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      const int k = kb - m;
      if (k >= 0) {
        double xkx, xky;
        to_d(cur[m], xkx, xky);
        xkx = sub_rn(xkx, mul_rn(scur[m], xpx));
        xky = sub_rn(xky, mul_rn(scur[m], xpy));
        x[(long long)k * ncol] = from_d<C>(xkx, xky);
        xpx = xkx;
        xpy = xky;
      }
    }
#pragma unroll
    for (int m = 0; m < kB; ++m) {
      cur[m] = nxt[m];
      scur[m] = snxt[m];
    }
  }
}

// ---- inverse x-FFT -> pressure ----------------------------------------------
// DST = kDstWrite: write the pressure; kDstAccumulate: add to the current
// pressure (refinement); kDstDense: write a dense interior array (a slab of
// levels of a sharded solve).
// block = (interior j, chunk of KC = 2 LC levels).  Line p gets
// Z = A + i B over all m, A and B the stored half-spectra of levels 2p and
// 2p + 1 extended by A[N-m] = conj A[m]; the inverse transform returns the
// two real rows as Re z and Im z.
// (LGN as for fft_x_fwd.)
template <class C, int DST, int LGN>
__global__ void __launch_bounds__((fft_threads<C, LGN>()), (fft_blocks<C, LGN>())) fft_x_inv(Geo g, PArgs a, int KCrt) {
  constexpr bool ACC = DST == kDstAccumulate;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* in = reinterpret_cast<C*>(smraw);
  const int N = LGN > 0 ? (1 << LGN) : (int)(g.n0 - 2 * g.gw);
  const int KC = LGN > 0 ? 2 * ct_lines(LGN) : KCrt;
  const int Nh = N / 2 + 1;
  const int nz = (int)(g.n2 - 2 * g.gw);
  const int jl = blockIdx.x;
  const int k0 = blockIdx.y * KC;
  const int kc = min(KC, nz - k0);
  const int lc = (kc + 1) >> 1;
  const C* spec = reinterpret_cast<const C*>(a.spec);
  const long long ny = g.n1 - 2 * g.gw;
  const long long nxy = (long long)Nh * ny;
  const double sc = 1.0 / (double)N;
  // where the value of x position il and level k0 + kl goes
  double* __restrict__ out = DST == kDstDense ? a.dst_dense + (long long)jl * nz + k0
                                              : a.p + g.gw * g.is + (g.gw + jl) * g.js + g.gw + k0;
  const long long so = DST == kDstDense ? ny * nz : g.is;
  if constexpr (LGN > 0) {
    // Z[m] = A[m] + i B[m], and for m > N/2 conj A[N-m] + i conj B[N-m]
    using T = Ct<C, LGN>;
    const C* row = spec + (long long)k0 * nxy + (long long)jl * Nh;
    auto load = [&](int l, int x) {
      C z = czero<C>();
      if (l < lc) {
        const bool up = x > N / 2;
        const C* src = row + (long long)(2 * l) * nxy + (up ? N - x : x);
        const C A = src[0];
        const C B = 2 * l + 1 < kc ? src[nxy] : czero<C>();
        z.x = up ? A.x + B.y : A.x - B.y;
        z.y = up ? B.x - A.y : A.y + B.x;
      }
      return z;
    };
    auto store = [&](int l, int x, C z) {
      double* dst = out + x * so + 2 * l;
      const double x0 = (double)z.x * sc, x1 = (double)z.y * sc;
      if (2 * l < kc) dst[0] = ACC ? dst[0] + x0 : x0;
      if (2 * l + 1 < kc) dst[1] = ACC ? dst[1] + x1 : x1;
    };
    if constexpr (sizeof(C) == 16) {
      ct_fft<C, LGN, false, false, false>(in, twx_of<C>(a), true, load, store);
    } else {
      // FP32: the stores of the last pass, two levels a thread, would be half
      // of the kernel's accesses; through the buffer consecutive threads write
      // consecutive levels
      ct_fft<C, LGN, false, true, false>(in, twx_of<C>(a), true, load,
                                         [&](int l, int x, C z) { in[T::at(l, x)] = z; });
      __syncthreads();
      constexpr int kBatch = 4;  // the pressure loads of a batch are issued before its stores
#pragma unroll 1
      for (int e0 = threadIdx.x; e0 < N * KC; e0 += kBatch * T::NT) {
        double val[kBatch], old[kBatch];
#pragma unroll
        for (int h = 0; h < kBatch; ++h) {
          const int e = e0 + h * T::NT, il = e / KC, kl = e % KC;
          const C z = in[T::at(kl >> 1, il)];
          val[h] = (double)((kl & 1) ? z.y : z.x) * sc;
          old[h] = ACC && kl < kc ? out[il * so + kl] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < kBatch; ++h) {
          const int e = e0 + h * T::NT, il = e / KC, kl = e % KC;
          if (kl < kc) out[il * so + kl] = ACC ? old[h] + val[h] : val[h];
        }
      }
    }
    return;
  }
  const int ld = line_ld(N);
#pragma unroll 4
  for (int e = threadIdx.x; e < Nh * lc; e += kFftThreads) {
    const int p = e / Nh;
    const int m = e - p * Nh;
    const long long src = (long long)(k0 + 2 * p) * nxy + (long long)jl * Nh + m;
    const C A = spec[src];
    const C B = (2 * p + 1 < kc) ? spec[src + nxy] : czero<C>();
    C* line = in + p * ld;
    C z;
    z.x = A.x - B.y;
    z.y = A.y + B.x;
    line[swz(m)] = z;
    if (m >= 1 && m <= N - Nh) {  // Z[N-m] = conj A[m] + i conj B[m]
      C zr;
      zr.x = A.x + B.y;
      zr.y = B.x - A.y;
      line[swz(N - m)] = zr;
    }
  }
  __syncthreads();
  const C* res = fft_lines<C, LGN == kFftShort>(in, lc, KC >> 1, N, twx_of<C>(a), a.tmx, true);
#pragma unroll 4
  for (int e = threadIdx.x; e < N * KC; e += kFftThreads) {
    int kl = 0, il = 0;
    split_idx(e, KC, il, kl);
    if (kl >= kc) continue;
    const C z = res[(kl >> 1) * ld + swz(il)];
    const double x = mul_rn((double)((kl & 1) ? z.y : z.x), sc);
    out[il * so + kl] = ACC ? add_rn(out[il * so + kl], x) : x;
  }
}

// ---- pressure ghost fill (sym), communicate_variable on one rank -----------
// `zero`, if given: a field whose ghosts are set to 0 in the same pass (the
// divergence, whose ghosts no kernel of the solve reads: one launch less).
__global__ void ghost_sym(Geo g, double* __restrict__ f, double* __restrict__ zero, long long nghost) {
  const long long gw = g.gw, n0 = g.n0, n1 = g.n1, n2 = g.n2;
  const long long nl0 = n0 - 2 * gw, nl1 = n1 - 2 * gw;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nghost; t += stride) {
    long long i, j, k;
    ghost_decode(g, t, i, j, k);
    const long long is_ = (i < gw) ? i + nl0 : ((i >= n0 - gw) ? i - nl0 : i);
    const long long js_ = (j < gw) ? j + nl1 : ((j >= n1 - gw) ? j - nl1 : j);
    long long ks = k;
    if (k >= n2 - gw) ks = n2 - gw - 1 - (k - (n2 - gw));
    else if (k < gw) ks = gw + (gw - 1 - k);
    f[i * g.is + j * g.js + k] = f[is_ * g.is + js_ * g.js + ks];
    if (zero != nullptr) zero[i * g.is + j * g.js + k] = 0.0;
  }
}

// ---- second_order_pressure_correction (PressureSolver.pyx:83-110) ---------
// w enters as it was before remove_mean_u3; every cell first gets w - mean[k]
// (the reference's remove_mean_u3 over all cells), then the correction on
// [0, nlg-1) in every dimension.
__global__ void correction(Geo g, const double* __restrict__ p, double* __restrict__ u, double* __restrict__ v,
                           double* __restrict__ w, const double* __restrict__ mean) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < g.npg; t += stride) {
    long long i, j, k;
    if (g.npg < (1LL << 31)) {
      const unsigned tt = (unsigned)t, r = tt / (unsigned)g.n2, ii = r / (unsigned)g.n1;
      k = tt - r * (unsigned)g.n2;
      j = r - ii * (unsigned)g.n1;
      i = ii;
    } else {
      const long long r = t / g.n2;
      k = t - r * g.n2;
      i = r / g.n1;
      j = r - i * g.n1;
    }
    const double wt = sub_rn(w[t], mean[k]);
    if (i >= g.n0 - 1 || j >= g.n1 - 1 || k >= g.n2 - 1) {
      w[t] = wt;
      continue;
    }
    const double pc = p[t];
    u[t] = sub_rn(u[t], mul_rn(sub_rn(p[t + g.is], pc), g.dxi0));
    v[t] = sub_rn(v[t], mul_rn(sub_rn(p[t + g.js], pc), g.dxi1));
    w[t] = sub_rn(wt, mul_rn(sub_rn(p[t + 1], pc), g.dxi2));
  }
}

int stream_blocks(long long work) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long b = (work + 255) / 256;
  if (b > (long long)sms * 8) b = (long long)sms * 8;
  return (int)(b < 1 ? 1 : b);
}

bool pow2(long long n) { return (n & (n - 1)) == 0; }

// Horizontal sizes the line FFTs support: powers of two up to 4096 (a
// block's Stockham passes hold at most 16 * kFftThreads elements, one line of
// 4096) and other lengths up to 1024 (direct DFT).
bool fft_sizes_ok(const pb_dims* d) {
  for (int dim = 0; dim < 2; ++dim) {
    const long long n = d->n[dim];
    if (pow2(n) ? n > 4096 : n > 1024) return false;
  }
  return true;
}

// Outputs per thread of a direct transform (dft_rows): the smallest divisor
// of N among the built ones that gives all outputs of a block's lines a
// thread in one round, else the largest; the twiddle table (TM N values) has
// to leave room for two blocks of 80 KiB of lines per SM (FP64) or three of
// 48 KiB (FP32).  Where none divides N, dft_any: with 2 outputs per thread if
// that is one round (on few points the length of a thread's chain counts: a
// solve of 27x27x40 68 us, 76 with 6 outputs; FP32 form 113, 133), else with
// 6 (returned as 0, as for powers of two).
int direct_outputs(long long N, int lines, size_t elem) {
  if (pow2(N)) return 0;
  int best = lines * ((N + 1) / 2) <= kFftThreads ? 2 : 0;
  const int built[] = {4, 5, 6, 8, 10};
  for (int tm : built) {
    if (N % tm != 0 || tm * N * (long long)elem > 24 * 1024) continue;
    best = tm;
    if (lines * (N / tm) <= kFftThreads) break;
  }
  return best;
}

size_t fft_smem(long long N, int lines, size_t elem) {
  if (pow2(N)) return (size_t)line_ld((int)N) * lines * elem;
  const int tm = direct_outputs(N, lines, elem);  // a second set of lines and the twiddles
  return (2 * (size_t)line_ld((int)N) * lines + (size_t)N * (tm > 2 ? tm : 1)) * elem;
}

// Lines per FFT block: a power of two, up to 16, with nlines * N <=
// 16 * kFftThreads for the Stockham passes and the block's shared memory
// within 48 KiB (FP32) / 80 KiB (FP64), so that several blocks share an SM
// and one block's loads overlap another's passes.
int lines_for(long long N, size_t elem) {
  const long long per = (pow2(N) ? 1 : 2) * (long long)line_ld((int)N) * (long long)elem;
  long long L = (elem <= 8 ? 49152 : 81920) / per;
  if (L > 16) L = 16;
  if (pow2(N) && L * N > 16LL * kFftThreads) L = 16LL * kFftThreads / N;
  if (L < 1) L = 1;
  while (L & (L - 1)) L &= L - 1;  // a power of two: shifts in the index arithmetic
  return (int)L;
}

}  // namespace

extern "C" long long pb_pressure_workspace_bytes(const pb_dims* dims) {
  if (pb_check_dims(dims)) return -1;
  return playout(dims).total;
}

// PressureFFTParallel.initialize (:27-62): the modified wave numbers
// (compute_modified_wave_numbers, :64-98) are evaluated on the host with the
// C library cos, as the reference does, so they match it bit for bit; the
// FFT twiddles exp(-2 pi i m/N) are evaluated in long double and rounded.
extern "C" int pb_pressure_init(const pb_dims* dims, void* workspace, long long workspace_bytes) {
  int rc = pb_check_dims(dims);
  if (rc) return rc;
  const PLayout L = playout(dims);
  if (!workspace || workspace_bytes < L.total) return PB_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return PB_ERR_WORKSPACE;
  const double pi = 3.141592653589793;
  char* base = static_cast<char*>(workspace);
  for (int dim = 0; dim < 2; ++dim) {
    const long n = dims->n[dim];
    std::vector<double> k2(n);
    std::vector<double2> tw(n);
    for (long ii = 0; ii < n; ++ii) {
      const long i = dims->indx_lo[dim] + ii;
      double xi;
      if ((double)i <= (double)n / 2.0) xi = (double)i;
      else xi = (double)(i - n);
      k2[ii] = (2.0 * cos((2.0 * pi / (double)n) * xi) - 2.0) / dims->dx[dim] / dims->dx[dim];
      const long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)ii / (long double)n;
      tw[ii] = make_double2((double)cosl(ang), (double)sinl(ang));
    }
    if (dims->indx_lo[dim] == 0) k2[0] = 0.0;
    PB_CUDA_TRY(cudaMemcpy(base + (dim == 0 ? L.kx2 : L.ky2), k2.data(), n * sizeof(double),
                           cudaMemcpyHostToDevice));
    PB_CUDA_TRY(cudaMemcpy(base + (dim == 0 ? L.twx : L.twy), tw.data(), n * sizeof(double2),
                           cudaMemcpyHostToDevice));
    std::vector<float2> twf(n);
    for (long ii = 0; ii < n; ++ii) twf[ii] = make_float2((float)tw[ii].x, (float)tw[ii].y);
    PB_CUDA_TRY(cudaMemcpy(base + (dim == 0 ? L.twxf : L.twyf), twf.data(), n * sizeof(float2),
                           cudaMemcpyHostToDevice));
  }
  return PB_OK;
}

// log2 of a length that has compile-time FFT kernels (32 ... 1024), else 0
int ct_lg(long long n) {
  if (!pow2(n) || n < 32 || n > 1024) return 0;
  int lg = 0;
  while ((1LL << lg) < n) ++lg;
  return lg;
}

// Opt in to more than 48 KiB of shared memory where a launch needs it: the
// limit holds for the kernel's static part (the forward x-FFT's reciprocals,
// asked for once: a property of the compiled kernel) and the dynamic part
// together.  By the dynamic part alone an FP64 solve on 83 or 306 columns
// along x, of 48,944 and 49,056 bytes, was refused.
template <auto Kernel>
static int allow_smem(size_t dynamic) {
  static const size_t fixed = [] {
    cudaFuncAttributes at;
    return cudaFuncGetAttributes(&at, Kernel) == cudaSuccess ? at.sharedSizeBytes : size_t(48 * 1024);
  }();
  if (fixed + dynamic > 48 * 1024)
    PB_CUDA_TRY(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dynamic));
  return PB_OK;
}

template <class C, int SRC, int LG>
static int launch_x_fwd_src(const Geo& g, PArgs& a, dim3 grid, size_t sm, int KC, cudaStream_t st) {
  if (const int rc = allow_smem<fft_x_fwd<C, SRC, LG>>(sm)) return rc;
  fft_x_fwd<C, SRC, LG><<<grid, fft_threads<C, LG>(), sm, st>>>(g, a, KC);
  return PB_OK;
}

template <class C, int LG>
static int launch_x_fwd(const Geo& g, PArgs& a, int src, dim3 grid, size_t sm, int KC, cudaStream_t st) {
  if (src == kSrcDense) return launch_x_fwd_src<C, kSrcDense, LG>(g, a, grid, sm, KC, st);
  if constexpr (sizeof(C) == 8) {  // the refinement residual exists in the precision form only
    if (src == kSrcResidual) return launch_x_fwd_src<C, kSrcResidual, LG>(g, a, grid, sm, KC, st);
  }
  return launch_x_fwd_src<C, kSrcDivergence, LG>(g, a, grid, sm, KC, st);
}

template <class C, int DST, int LG>
static int launch_x_inv_dst(const Geo& g, PArgs& a, dim3 grid, size_t sm, int KC, cudaStream_t st) {
  if (const int rc = allow_smem<fft_x_inv<C, DST, LG>>(sm)) return rc;
  fft_x_inv<C, DST, LG><<<grid, fft_threads<C, LG>(), sm, st>>>(g, a, KC);
  return PB_OK;
}

template <class C, int LG>
static int launch_x_inv(const Geo& g, PArgs& a, int dst, dim3 grid, size_t sm, int KC, cudaStream_t st) {
  if (dst == kDstDense) return launch_x_inv_dst<C, kDstDense, LG>(g, a, grid, sm, KC, st);
  if constexpr (sizeof(C) == 8) {
    if (dst == kDstAccumulate) return launch_x_inv_dst<C, kDstAccumulate, LG>(g, a, grid, sm, KC, st);
  }
  return launch_x_inv_dst<C, kDstWrite, LG>(g, a, grid, sm, KC, st);
}

template <class C, int LG>
static int launch_y(const Geo& g, PArgs& a, bool inverse, dim3 grid, size_t sm, int IC, cudaStream_t st) {
  if (inverse) {
    if (const int rc = allow_smem<fft_y<C, true, LG>>(sm)) return rc;
    fft_y<C, true, LG><<<grid, fft_threads<C, LG>(), sm, st>>>(g, a, IC);
  } else {
    if (const int rc = allow_smem<fft_y<C, false, LG>>(sm)) return rc;
    fft_y<C, false, LG><<<grid, fft_threads<C, LG>(), sm, st>>>(g, a, IC);
  }
  return PB_OK;
}

// Dispatch on a length's instantiation (fft_kernel).
#define PB_FFT_DISPATCH(lg, call)         \
  switch (lg) {                           \
    case 5: { constexpr int L_ = 5; call; } break;   \
    case 6: { constexpr int L_ = 6; call; } break;   \
    case 7: { constexpr int L_ = 7; call; } break;   \
    case 8: { constexpr int L_ = 8; call; } break;   \
    case 9: { constexpr int L_ = 9; call; } break;   \
    case 10: { constexpr int L_ = 10; call; } break; \
    case kFftShort: { constexpr int L_ = kFftShort; call; } break; \
    default: { constexpr int L_ = kFftRuntime; call; } break; \
  }

// The kernels of a length: its compile-time ones, those of few points, or those
// of any length.
static int fft_kernel(long long n, int tm) {
  const int lg = ct_lg(n);
  return lg ? lg : (tm == 2 ? kFftShort : kFftRuntime);
}

template <class C>
static size_t ct_smem(int lg) {
  size_t sm = 0;
  PB_FFT_DISPATCH(lg, sm = (Ct<C, (L_ > 0 ? L_ : 5)>::SMEM));
  return sm;
}

// The spectral solve in phases, so that a sharded solve can exchange data
// between them: (1) forward x-FFT (from src) and forward y-FFT of every level
// of the grid; (2) the Thomas solve of every (kx, ky) column; (3) inverse
// y-FFT and inverse x-FFT (to dst).
struct FftShape {
  long long Nx, Ny, nz, Nh;
  int LC, KC, IC, lgx, lgy, tmx, tmy, kx, ky;
  size_t smx, smy;
  dim3 gx, gy;
};

template <class C>
static int fft_shape(const Geo& g, FftShape& f) {
  f.Nx = g.n0 - 2 * g.gw;
  f.Ny = g.n1 - 2 * g.gw;
  f.nz = g.n2 - 2 * g.gw;
  f.Nh = f.Nx / 2 + 1;  // stored x-modes
  f.lgx = ct_lg(f.Nx);
  f.lgy = ct_lg(f.Ny);
  f.LC = f.lgx ? ct_lines(f.lgx) : lines_for(f.Nx, sizeof(C));  // complex lines per x-FFT block
  f.KC = 2 * f.LC;                                               // levels per x-FFT block (two per line)
  f.smx = f.lgx ? ct_smem<C>(f.lgx) : fft_smem(f.Nx, f.LC, sizeof(C));
  f.IC = f.lgy ? ct_lines(f.lgy) : lines_for(f.Ny, sizeof(C));
  f.smy = f.lgy ? ct_smem<C>(f.lgy) : fft_smem(f.Ny, f.IC, sizeof(C));
  f.tmx = direct_outputs(f.Nx, f.LC, sizeof(C));
  f.tmy = direct_outputs(f.Ny, f.IC, sizeof(C));
  f.kx = fft_kernel(f.Nx, f.tmx);
  f.ky = fft_kernel(f.Ny, f.tmy);
  f.gx = dim3((unsigned)f.Ny, ceil_div(f.nz, f.KC));
  f.gy = dim3(ceil_div(f.Nh, f.IC), (unsigned)f.nz);
  return PB_OK;
}

template <class C>
static int fft_forward(const Geo& g, PArgs& a, int src, cudaStream_t st) {
  FftShape f;
  int rc = fft_shape<C>(g, f);
  if (rc) return rc;
  a.tmx = f.tmx;
  a.tmy = f.tmy;
  PB_FFT_DISPATCH(f.kx, rc = (launch_x_fwd<C, L_>(g, a, src, f.gx, f.smx, f.KC, st)));
  if (rc) return rc;
  pb_note_launch();
  PB_LAUNCH_CHECK();
  PB_FFT_DISPATCH(f.ky, rc = (launch_y<C, L_>(g, a, false, f.gy, f.smy, f.IC, st)));
  if (rc) return rc;
  pb_note_launch();
  PB_LAUNCH_CHECK();
  return PB_OK;
}

template <class C>
static int fft_columns(const Geo& g, PArgs& a, cudaStream_t st) {
  const long long Nh = (g.n0 - 2 * g.gw) / 2 + 1, Ny = g.n1 - 2 * g.gw;
  // one thread per column; on grids with fewer columns than 256 per SM the
  // blocks shrink (to a multiple of 32 threads) so that every SM gets some
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long per_sm = (Nh * Ny + sms - 1) / sms;
  const int threads = per_sm >= 256 ? 256 : (int)((per_sm + 31) / 32 * 32);
  tdma_kernel<C><<<ceil_div(Nh * Ny, threads), threads, 0, st>>>(g, a);
  pb_note_launch();
  PB_LAUNCH_CHECK();
  return PB_OK;
}

template <class C>
static int fft_inverse(const Geo& g, PArgs& a, int dst, cudaStream_t st) {
  FftShape f;
  int rc = fft_shape<C>(g, f);
  if (rc) return rc;
  a.tmx = f.tmx;
  a.tmy = f.tmy;
  PB_FFT_DISPATCH(f.ky, rc = (launch_y<C, L_>(g, a, true, f.gy, f.smy, f.IC, st)));
  if (rc) return rc;
  pb_note_launch();
  PB_LAUNCH_CHECK();
  PB_FFT_DISPATCH(f.kx, rc = (launch_x_inv<C, L_>(g, a, dst, f.gx, f.smx, f.KC, st)));
  if (rc) return rc;
  pb_note_launch();
  PB_LAUNCH_CHECK();
  return PB_OK;
}

template <class C>
static int fft_solve(const Geo& g, PArgs& a, bool resid, bool acc, cudaStream_t st) {
  int rc;
  if ((rc = fft_forward<C>(g, a, resid ? kSrcResidual : kSrcDivergence, st))) return rc;
  if ((rc = fft_columns<C>(g, a, st))) return rc;
  return fft_inverse<C>(g, a, acc ? kDstAccumulate : kDstWrite, st);
}
#undef PB_FFT_DISPATCH

static int pressure_solve_impl(const pb_dims* dims, const double* rho0, const double* rho0_half,
                               const double* alpha0, const double* alpha0_half, double* u, double* v, double* w,
                               double* divergence, double* dynamic_pressure, char* base, int precision,
                               int refine_sweeps, cudaStream_t st) {
  const Geo g = make_geo(dims);
  const PLayout L = playout(dims);
  PArgs a{};
  a.rho0 = rho0;
  a.rho0_half = rho0_half;
  a.alpha0 = alpha0;
  a.alpha0_half = alpha0_half;
  a.u = u;
  a.v = v;
  a.w = w;
  a.div = divergence;
  a.p = dynamic_pressure;
  a.partial = reinterpret_cast<double*>(base + L.partial);
  a.mean = reinterpret_cast<double*>(base + L.mean);
  a.twx = reinterpret_cast<const double2*>(base + L.twx);
  a.twy = reinterpret_cast<const double2*>(base + L.twy);
  a.twxf = reinterpret_cast<const float2*>(base + L.twxf);
  a.twyf = reinterpret_cast<const float2*>(base + L.twyf);
  a.kx2 = reinterpret_cast<const double*>(base + L.kx2);
  a.ky2 = reinterpret_cast<const double*>(base + L.ky2);
  a.spec = base + L.spec;
  a.scr = reinterpret_cast<double*>(base + L.scr);
  const long long Nx = dims->n[0], Ny = dims->n[1], nz = dims->n[2];
  const long long nghost = g.npg - Nx * Ny * nz;

  if (precision == PB_FP64) {  // the reference's summation order
    const int rc =
        launch_hmean_ordered(g, w, a.mean, 1.0 / (double)(Ny * Nx), static_cast<double*>(a.spec), st);
    if (rc) return rc;
  } else {  // precision form: a deterministic parallel sum
    const int kpad = (int)((g.n2 + 31) / 32 * 32);
    hmean_partial<<<kPartials, kpad < 1024 ? kpad : 1024, 0, st>>>(g, w, a.partial);
    pb_note_launch();
    hmean_final<<<(unsigned)g.n2, 256, 0, st>>>(g, a.partial, a.mean, kPartials, 1.0 / (double)(Ny * Nx));
    pb_note_launch();
  }
  PB_LAUNCH_CHECK();

  int rc;
  if (precision == PB_FP64) {
    if ((rc = fft_solve<double2>(g, a, false, false, st))) return rc;
  } else {
    // precision form: FP32 FFTs, FP64 tridiagonal solve, then refinement
    // sweeps p += solve(div - A p) on the FP64 residual
    if ((rc = fft_solve<float2>(g, a, false, false, st))) return rc;
    for (int s = 0; s < refine_sweeps; ++s) {
      if (nghost > 0) {
        ghost_sym<<<stream_blocks(nghost), 256, 0, st>>>(g, dynamic_pressure, nullptr, nghost);
        pb_note_launch();
      }
      if ((rc = fft_solve<float2>(g, a, true, true, st))) return rc;
    }
  }
  if (nghost > 0) {
    ghost_sym<<<stream_blocks(nghost), 256, 0, st>>>(g, dynamic_pressure, divergence, nghost);
    pb_note_launch();
  }
  correction<<<stream_blocks(g.npg), 256, 0, st>>>(g, dynamic_pressure, u, v, w, a.mean);
  pb_note_launch();
  PB_LAUNCH_CHECK();
  return PB_OK;
}

extern "C" int pb_pressure_solve(const pb_dims* dims, const double* rho0, const double* rho0_half,
                                 const double* alpha0, const double* alpha0_half, double* u, double* v, double* w,
                                 double* divergence, double* dynamic_pressure, void* workspace,
                                 long long workspace_bytes, int precision, int refine_sweeps, void* stream) {
  int rc = pb_check_dims(dims);
  if (rc) return rc;
  if (!rho0 || !rho0_half || !alpha0 || !alpha0_half || !u || !v || !w || !divergence || !dynamic_pressure)
    return PB_ERR_ARG;
  if (precision != PB_FP64 && precision != PB_FP32) return PB_ERR_ARG;
  if (refine_sweeps < 0 || refine_sweeps > 8) return PB_ERR_ARG;
  const PLayout L = playout(dims);
  if (!workspace || workspace_bytes < L.total) return PB_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return PB_ERR_WORKSPACE;
  if (!fft_sizes_ok(dims)) return PB_ERR_UNSUPPORTED;
  return pressure_solve_impl(dims, rho0, rho0_half, alpha0, alpha0_half, u, v, w, divergence, dynamic_pressure,
                             static_cast<char*>(workspace), precision, refine_sweeps, as_stream(stream));
}
