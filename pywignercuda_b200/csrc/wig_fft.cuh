// Shared-memory batched Stockham FFT for sm_100a (double and float).
//
// One CTA transforms NB independent sequences of length N (power of two) that
// live in shared memory.  The element layout is a template functor ("Map") so
// that the same code serves contiguous rows (x-pass: sequence = one grid row)
// and interleaved column tiles (p-pass: sequence = one grid column, the tile
// stored row-major, so element k of column c sits at k*NB + c).
//
// Stockham autosort, mixed radix 16/8/4/2: stage s combines R sub-transforms of
// length Ns into length Ns*R.  Butterfly j (0 <= j < N/R) reads elements
// j + r*N/R, applies twiddles W_{Ns R}^{(j mod Ns) r}, does an R-point DFT and
// writes to (j/Ns)*Ns*R + (j mod Ns) + r*Ns.  Output is in natural order.
// Each stage is done in place through registers: every thread loads all of
// its butterflies' inputs, the CTA synchronises, then every thread writes.
//
// Twiddles come from a table tw[m] = exp(-2 pi i m / N), m < N, computed on
// the host in extended precision; the inverse transform uses the conjugates.
// Forward = exp(-i ...), inverse unnormalised (the callers fold 1/N into a
// pointwise factor, which is exact because N is a power of two).
#pragma once

// WIG_BOUNDS_CHECK(what, i, n): 0 <= i < n.  Compiled in only when WIG_BOUNDS is
// defined, which only the host execution of this device code does (its shim
// provides wig_bounds_fail, which reports and aborts); the kernels the library
// compiles for the GPU carry no such checks and never trap.
#ifdef WIG_BOUNDS
#define WIG_BOUNDS_CHECK(what, i, n)                                                   \
  do {                                                                                 \
    if ((long long)(i) < 0 || (long long)(i) >= (long long)(n)) wig_bounds_fail(what, (long long)(i), (long long)(n)); \
  } while (0)
#else
#define WIG_BOUNDS_CHECK(what, i, n) \
  do {                               \
  } while (0)
#endif

namespace wig {

template <class T> struct V2;
template <> struct V2<double> { typedef double2 t; };
template <> struct V2<float>  { typedef float2 t;  };

__device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float2  mk(float a, float b)   { return make_float2(a, b); }

template <class C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <class C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// (a.x + i a.y)(b.x + i b.y), the textbook formula (same as pycuda::complex)
template <class C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
template <class C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }
template <class C, class T> __device__ __forceinline__ C cscale(C a, T s) { a.x *= s; a.y *= s; return a; }
// multiply by -i (forward) or +i (inverse)
template <bool INV, class C> __device__ __forceinline__ C mul_mi(C a) {
  C r;
  if (INV) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
  return r;
}

// Complex sum and difference; with WIG_PACKED_F32 one packed instruction for float2
// (both components rounded as by the two scalar ones: the batched FP32 transforms are
// bound by issue slots; 64-instance batch, step 522 -> 499 us, bit for bit the same).
// Used where neither operand is a free swap or sign change of another value.
template <class C> __device__ __forceinline__ C padd(C a, C b) { return cadd(a, b); }
template <class C> __device__ __forceinline__ C psub(C a, C b) { return csub(a, b); }
#if defined(__CUDA_ARCH__) && defined(WIG_PACKED_F32)
template <> __device__ __forceinline__ float2 padd<float2>(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n add.rn.f32x2 c, a, b;\n"
      " mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
template <> __device__ __forceinline__ float2 psub<float2>(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n sub.rn.f32x2 c, a, b;\n"
      " mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
#endif

// ---------------------------------------------------------------- R-point DFTs
template <bool INV, class C> __device__ __forceinline__ void dft2(C& a, C& b) {
  C t = a; a = padd(t, b); b = psub(t, b);
}

template <bool INV, class C> __device__ __forceinline__ void dft4(C& v0, C& v1, C& v2, C& v3) {
  C a0 = padd(v0, v2), a1 = psub(v0, v2), a2 = padd(v1, v3), a3 = mul_mi<INV>(psub(v1, v3));
  v0 = padd(a0, a2); v2 = psub(a0, a2); v1 = cadd(a1, a3); v3 = csub(a1, a3);
}

template <bool INV, class C> __device__ __forceinline__ void dft8(C* v) {
  typedef decltype(v[0].x) T;
  const T h = (T)0.70710678118654752440084436210485;   // sqrt(1/2)
  C a[4], b[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) { a[k] = cadd(v[k], v[k + 4]); b[k] = csub(v[k], v[k + 4]); }
  // b_k *= W8^k  (W8 = exp(-+ 2 pi i / 8))
  {
    C t = b[1];
    if (INV) { b[1].x = h * (t.x - t.y); b[1].y = h * (t.x + t.y); }
    else     { b[1].x = h * (t.x + t.y); b[1].y = h * (t.y - t.x); }
    b[2] = mul_mi<INV>(b[2]);
    t = b[3];
    if (INV) { b[3].x = -h * (t.x + t.y); b[3].y = h * (t.x - t.y); }
    else     { b[3].x = h * (t.y - t.x); b[3].y = -h * (t.x + t.y); }
  }
  dft4<INV>(a[0], a[1], a[2], a[3]);
  dft4<INV>(b[0], b[1], b[2], b[3]);
#pragma unroll
  for (int m = 0; m < 4; ++m) { v[2 * m] = a[m]; v[2 * m + 1] = b[m]; }
}

// ---------------------------------------------------------------- radix-8/16/32 kernels
// (also the per-lane DFTs of the register FFT, wig_rfft.cuh)
// cos(pi j / 16) for any integer j
__host__ __device__ constexpr double cospi16(int j) {
  j = ((j % 32) + 32) % 32;
  if (j > 16) j = 32 - j;
  const bool neg = j > 8;
  if (neg) j = 16 - j;
  double c = 0.;
  switch (j) {
    case 0: c = 1.; break;
    case 1: c = 0.98078528040323044912618223613424; break;
    case 2: c = 0.92387953251128675612818318939679; break;
    case 3: c = 0.83146961230254523707878837761791; break;
    case 4: c = 0.70710678118654752440084436210485; break;
    case 5: c = 0.55557023301960222474283081394853; break;
    case 6: c = 0.38268343236508977172845998403040; break;
    case 7: c = 0.19509032201612826784828486847702; break;
    default: c = 0.; break;
  }
  return neg ? -c : c;
}

// u * c for a compile-time constant c.  In FP32 the constant is applied as a
// compensated pair hi + lo (hi = c rounded, lo = the rounding error), so the
// product carries only the rounding of the arithmetic: a constant rounded to
// float alone has |w|^2 != 1 by up to 6e-8, and a forward/inverse pair of FFTs
// would then scale some spectral components by a fixed factor every step.
__device__ __forceinline__ float mulk(float u, double c) {
  const float hi = (float)c, lo = (float)(c - (double)hi);
  return fmaf(u, hi, u * lo);
}
__device__ __forceinline__ double mulk(double u, double c) { return u * c; }
// u * c + v * s (c, s compile-time constants)
__device__ __forceinline__ float mulk2(float u, double c, float v, double s) {
  const float ch = (float)c, cl = (float)(c - (double)ch), sh = (float)s, sl = (float)(s - (double)sh);
  return fmaf(u, ch, fmaf(v, sh, fmaf(u, cl, v * sl)));
}
__device__ __forceinline__ double mulk2(double u, double c, double v, double s) { return fma(u, c, v * s); }

// v * W_32^j, W_32 = exp(-2 pi i / 32) (forward) or its conjugate (inverse);
// j is a compile-time constant after unrolling.
template <bool INV, class C>
__device__ __forceinline__ C twc32(C v, int j) {
  j &= 31;
  if (j == 0) return v;
  if (j == 16) { v.x = -v.x; v.y = -v.y; return v; }
  if (j == 8) return mul_mi<INV>(v);
  if (j == 24) return mul_mi<!INV>(v);
  const double c = cospi16(j), s = cospi16(8 - j);   // cos, sin of 2 pi j / 32
  C r;
  if ((j & 7) == 4) {   // |c| = |s| = sqrt(1/2): one product per component
    const double h = 0.70710678118654752440084436210485;
    const auto cx = c > 0. ? v.x : -v.x, cy = c > 0. ? v.y : -v.y;   // v c / h
    const auto sx = s > 0. ? v.x : -v.x, sy = s > 0. ? v.y : -v.y;   // v s / h
    if (INV) { r.x = mulk(cx - sy, h); r.y = mulk(sx + cy, h); }
    else     { r.x = mulk(cx + sy, h); r.y = mulk(cy - sx, h); }
    return r;
  }
  if (INV) { r.x = mulk2(v.x, c, v.y, -s); r.y = mulk2(v.x, s, v.y, c); }
  else     { r.x = mulk2(v.x, c, v.y, s);  r.y = mulk2(v.y, c, v.x, -s); }
  return r;
}

// 8-point DFT (radix-2 over two 4-point DFTs), constants through twc32.
template <bool INV, class C> __device__ __forceinline__ void dft8c(C* v) {
  C a[4], b[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) { a[k] = padd(v[k], v[k + 4]); b[k] = psub(v[k], v[k + 4]); }
  b[1] = twc32<INV>(b[1], 4);
  b[2] = mul_mi<INV>(b[2]);
  b[3] = twc32<INV>(b[3], 12);
  dft4<INV>(a[0], a[1], a[2], a[3]);
  dft4<INV>(b[0], b[1], b[2], b[3]);
#pragma unroll
  for (int m = 0; m < 4; ++m) { v[2 * m] = a[m]; v[2 * m + 1] = b[m]; }
}

// 16-point DFT as 4 x 4 (n = 4 a + b): radix-4 over a, twiddles W_16^{b k1},
// radix-4 over b.  Natural order in and out.
template <bool INV, class C> __device__ __forceinline__ void dft16(C* v) {
  C t[16];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    C a0 = v[b], a1 = v[b + 4], a2 = v[b + 8], a3 = v[b + 12];
    dft4<INV>(a0, a1, a2, a3);
    t[b] = a0; t[b + 4] = a1; t[b + 8] = a2; t[b + 12] = a3;   // t[4 k1 + b]
  }
#pragma unroll
  for (int k1 = 1; k1 < 4; ++k1)
#pragma unroll
    for (int b = 1; b < 4; ++b) t[4 * k1 + b] = twc32<INV>(t[4 * k1 + b], 2 * b * k1);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C a0 = t[4 * k1], a1 = t[4 * k1 + 1], a2 = t[4 * k1 + 2], a3 = t[4 * k1 + 3];
    dft4<INV>(a0, a1, a2, a3);
    v[k1] = a0; v[k1 + 4] = a1; v[k1 + 8] = a2; v[k1 + 12] = a3;   // X[k1 + 4 k2]
  }
}

// 16-point DFT of the inputs v[4 a + b] w4^a w1^b (w4[a - 1], w1[b - 1] given): w4^a before the
// radix-4 over a, w1^b after it.
template <bool INV, class C> __device__ __forceinline__ void dft16_tw(C* v, const C* w4, const C* w1) {
  C t[16];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    C a0 = v[b], a1 = cmul(v[b + 4], w4[0]), a2 = cmul(v[b + 8], w4[1]), a3 = cmul(v[b + 12], w4[2]);
    dft4<INV>(a0, a1, a2, a3);
    t[b] = a0; t[b + 4] = a1; t[b + 8] = a2; t[b + 12] = a3;   // t[4 k1 + b]
  }
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int b = 1; b < 4; ++b) t[4 * k1 + b] = twc32<INV>(cmul(t[4 * k1 + b], w1[b - 1]), 2 * b * k1);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C a0 = t[4 * k1], a1 = t[4 * k1 + 1], a2 = t[4 * k1 + 2], a3 = t[4 * k1 + 3];
    dft4<INV>(a0, a1, a2, a3);
    v[k1] = a0; v[k1 + 4] = a1; v[k1 + 8] = a2; v[k1 + 12] = a3;   // X[k1 + 4 k2]
  }
}

// 32-point DFT: radix-2 decimation in time over two 16-point DFTs.
template <bool INV, class C> __device__ __forceinline__ void dft32(C* v) {
  C e[16], o[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) { e[k] = v[2 * k]; o[k] = v[2 * k + 1]; }
  dft16<INV>(e);
  dft16<INV>(o);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const C t = twc32<INV>(o[k], k);
    v[k] = padd(e[k], t);
    v[k + 16] = psub(e[k], t);
  }
}

template <int R, bool INV, class C> __device__ __forceinline__ void dft_r(C* v) {
  if constexpr (R == 32) dft32<INV>(v);
  else if constexpr (R == 16) dft16<INV>(v);
  else if constexpr (R == 8) dft8c<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 2) dft2<INV>(v[0], v[1]);
}

template <int R, bool INV, class C> __device__ __forceinline__ void dft(C* v) {
  if constexpr (R == 2) dft2<INV>(v[0], v[1]);
  else if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 8) dft8<INV>(v);
  else dft16<INV>(v);
}

// ---------------------------------------------------------------- layouts
// Shared-memory layouts.  Both are a linear order plus one padding slot every
// 8 elements (phys = lin + lin/8), which spreads the stride-R accesses of the
// first Stockham stage over distinct 16-byte bank groups.
__device__ __forceinline__ int pad8(int lin) { return lin + (lin >> 3); }
__host__ __device__ constexpr int padded_size(int n) { return n + (n >> 3); }

// Contiguous rows: sequence b, element k at lin = b*N + k; consecutive
// butterflies walk along a row.
template <int N> struct RowMap {
  __device__ __forceinline__ static int idx(int b, int k) { return pad8(b * N + k); }
  template <int NBF> __device__ __forceinline__ static void split(int q, int& b, int& j) { b = q / NBF; j = q % NBF; }
};

// Column tile stored row-major: sequence (column) b, element k at lin = k*NB + b;
// consecutive butterflies walk across the columns first.
template <int NB> struct ColMap {
  __device__ __forceinline__ static int idx(int b, int k) { return pad8(k * NB + b); }
  template <int NBF> __device__ __forceinline__ static void split(int q, int& b, int& j) { b = q % NB; j = q / NB; }
};

// Largest radix <= MAXR that fits the remaining length.  MAXR = 16 takes fewer
// shared-memory round trips (256 = 16 16, 1024 = 16 16 4) but needs about twice the
// registers of MAXR = 8, so it is a per-call-site choice.
template <int N, int NS, int MAXR = 8> struct Radix {
  static constexpr int rem = N / NS;
  static constexpr int value = (MAXR >= 16 && rem >= 16) ? 16 : (rem >= 8 ? 8 : (rem >= 4 ? 4 : 2));
};

// One Stockham stage over all NB sequences.  Phase 1 reads each butterfly's R
// inputs from shared memory and its R-1 twiddles from the (L1-resident) table,
// so the twiddle latency overlaps the barrier; phase 2 computes and writes.
template <class C, int N, int NS, int NB, int NT, bool INV, class Map, int MAXR = 8>
__device__ __forceinline__ void fft_stage(C* s, const C* __restrict__ tw) {
  constexpr int R = Radix<N, NS, MAXR>::value;
  constexpr int NBF = N / R;                 // butterflies per sequence
  constexpr int TOT = NB * NBF;              // butterflies per stage
  constexpr int PER = (TOT + NT - 1) / NT;   // per thread
  constexpr int TWS = N / (NS * R);          // twiddle-table stride of this stage
  const int tid = threadIdx.x;
  C v[PER][R];
  C w[PER][R > 1 ? R - 1 : 1];
#pragma unroll
  for (int m = 0; m < PER; ++m) {
    const int q = tid + m * NT;
    if ((TOT % NT) == 0 || q < TOT) {
      int b, j;
      Map::template split<NBF>(q, b, j);
#pragma unroll
      for (int r = 0; r < R; ++r) v[m][r] = s[Map::idx(b, j + r * NBF)];
      if (NS > 1) {
        const int k = j & (NS - 1);
#pragma unroll
        for (int r = 1; r < R; ++r) w[m][r - 1] = __ldg(&tw[(k * r) * TWS]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < PER; ++m) {
    const int q = tid + m * NT;
    if ((TOT % NT) == 0 || q < TOT) {
      int b, j;
      Map::template split<NBF>(q, b, j);
      const int k = j & (NS - 1);
      if (NS > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[m][r] = cmul(v[m][r], INV ? cconj(w[m][r - 1]) : w[m][r - 1]);
      }
      dft<R, INV>(v[m]);
      const int d = (j - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) s[Map::idx(b, d + r * NS)] = v[m][r];
    }
  }
  __syncthreads();
}

template <class C, int N, int NS, int NB, int NT, bool INV, class Map, int MAXR> struct FftRun {
  __device__ __forceinline__ static void run(C* s, const C* __restrict__ tw) {
    fft_stage<C, N, NS, NB, NT, INV, Map, MAXR>(s, tw);
    FftRun<C, N, NS * Radix<N, NS, MAXR>::value, NB, NT, INV, Map, MAXR>::run(s, tw);
  }
};
template <class C, int N, int NB, int NT, bool INV, class Map, int MAXR> struct FftRun<C, N, N, NB, NT, INV, Map, MAXR> {
  __device__ __forceinline__ static void run(C*, const C* __restrict__) {}
};

// Batched FFT of NB sequences of length N in shared memory (caller has
// synchronised before; the CTA is synchronised on return).
template <class C, int N, int NB, int NT, bool INV, class Map, int MAXR = 8>
__device__ __forceinline__ void cta_fft(C* s, const C* __restrict__ tw) {
  FftRun<C, N, 1, NB, NT, INV, Map, MAXR>::run(s, tw);
}

// ---------------------------------------------------------------- register-blocked FFT
// Stockham transform of one sequence of N elements held in the registers of
// T = N / E threads: thread t holds v[m] = x[t + T m], on input and on output
// (natural order both ways), so pointwise factors apply between transforms
// without touching shared memory.  Only the stage boundaries go through shared
// memory: one store and one load per element and boundary, against a store and a
// load per stage and per pointwise factor of cta_fft.
//
// Every stage has radix E but one, which takes what is left: the second of three or
// more (1024 = 16 4 16, 512 = 16 2 16 or 8 8 8, 256 = 8 4 8 or 4 4 4 4), where its
// E / R butterflies share their twiddles, or the first of two (128 = 8 16).
//
// Twiddles.  The input r of a radix-16 butterfly carries w^{k r}, w = exp(-2 pi i /
// (16 NS)); with r = 4 a + b the factor w^{4 k a} is applied before the butterfly's
// first four 4-point DFTs (over a) and w^{k b} after them, so 6 table entries serve
// a butterfly instead of 15: the passes wait for loads, boundaries and dependent
// chains rather than for the FP64 pipe (44 % busy in the 1024^2 damped p-pass).
// Table (host: wighost::block_twiddles), stage after stage (NS > 1), NS entries
// each: radix 16: w^{4 k a}, a = 1..3, then w^{k b}, b = 1..3; radix R < 16: w^{k r},
// r = 1..R - 1, w = exp(-2 pi i / (R NS)).  Entry k of one factor is next to k + 1:
// the lanes of a warp read consecutive entries.  The inverse conjugates.
//
// Boundary after a stage (sub-length NS, radix R): consecutive threads store runs of
// NS elements, NS R apart.  Element i lies at i + NS (i / (NS R)), which puts the runs
// on distinct 16-byte bank groups (runs of 8 or more need no padding; below 8
// elements a group, one pad per 8 does it; 4 elements' radix-2 stage is left
// unpadded, its pads would be half the region); the loads stay consecutive.  The
// indices of a boundary differ in disjoint bits, so slot(i + j) = slot(i) + slot(j):
// one address and constant offsets.
template <class C, int N, int E> struct BlockFft {
  static constexpr int T = N / E;
  static constexpr int REGION = N + N / (E < 8 ? E : 8);
  static_assert(E >= 4 && E <= 16 && T >= 1 && (N & (N - 1)) == 0 && (E & (E - 1)) == 0, "BlockFft: powers of two");
  // radix of the stage of sub-length ns
  __host__ __device__ static constexpr int radix(int ns) {
    int shrt = N;
    while (shrt > E) shrt /= E;
    const int at = N <= E * E ? 1 : E;   // the short stage's sub-length
    return ns == at ? shrt : E;
  }
  // entries of the twiddle table
  __host__ __device__ static constexpr int table() {
    int n = 0;
    for (int ns = 1; ns < N; ns *= radix(ns))
      if (ns > 1) n += (radix(ns) == 16 ? 6 : radix(ns) - 1) * ns;
    return n;
  }
  template <int NS, int R> __device__ __forceinline__ static int slot(int i) {
    if (NS >= 8 || (NS > 1 && R < 4)) return i;
    return NS * R < 8 ? i + (i >> 3) : i + NS * (i / (NS * R));   // at most N / min(R, 8) pads
  }

  // s: the sequence's exchange region; sync() orders the T threads' accesses to it.
  template <bool INV, class Sync>
  __device__ __forceinline__ static void run(C (&v)[E], C* s, const C* __restrict__ tw, int t, const Sync& sync) {
    stage<1, INV, 1>(reinterpret_cast<C(&)[1][E]>(v), s, tw, t, sync);
  }
  // NC sequences held by the same T threads, transformed together (each stage's twiddles are
  // loaded once, its boundary costs one pair of barriers); s: NC regions, one after another
  template <bool INV, int NC, class Sync>
  __device__ __forceinline__ static void run_many(C (&v)[NC][E], C* s, const C* __restrict__ tw, int t,
                                                  const Sync& sync) {
    stage<1, INV, NC>(v, s, tw, t, sync);
  }

  // the stage of sub-length NS: butterflies t + T q, q < E / R
  template <int NS, bool INV, int NC, class Sync>
  __device__ __forceinline__ static void stage(C (&v)[NC][E], C* s, const C* __restrict__ tw, int t,
                                               const Sync& sync) {
    constexpr int R = radix(NS), Q = E / R;
    static_assert(T % NS == 0, "a stage's butterflies share their twiddles");
    const int k = t & (NS - 1);
    if constexpr (NS > 1 && R == 16) {
      C w4[3], w1[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        w4[a] = __ldg(tw + a * NS + k);
        w1[a] = __ldg(tw + (3 + a) * NS + k);
        if (INV) { w4[a] = cconj(w4[a]); w1[a] = cconj(w1[a]); }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) dft16_tw<INV>(v[c], w4, w1);
    } else {
      C w[R];
      if constexpr (NS > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
          w[r] = __ldg(tw + (r - 1) * NS + k);
          if (INV) w[r] = cconj(w[r]);
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          C u[R];
#pragma unroll
          for (int r = 0; r < R; ++r) u[r] = NS > 1 && r > 0 ? cmul(v[c][q + r * Q], w[r]) : v[c][q + r * Q];
          dft_r<R, INV>(u);
#pragma unroll
          for (int r = 0; r < R; ++r) v[c][q + r * Q] = u[r];
        }
    }
    if constexpr (NS * R < N) {
      sync();   // the region's previous contents have been read
      C* d = s + slot<NS, R>((t - k) * R + k);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
          for (int r = 0; r < R; ++r)
            d[c * REGION + slot<NS, R>(T * q * R) + slot<NS, R>(r * NS)] = v[c][q + r * Q];
      sync();
      const C* g = s + slot<NS, R>(t);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int m = 0; m < E; ++m) v[c][m] = g[c * REGION + slot<NS, R>(T * m)];
      stage<NS * R, INV, NC>(v, s, tw + (NS > 1 ? (R == 16 ? 6 : R - 1) * NS : 0), t, sync);
    }
  }
};

// Barriers over the threads that share an exchange region.
struct SyncWarp {
  __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
struct SyncCta {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// NTH threads (a multiple of 32) of the CTA, on a hardware barrier of their own
template <int NTH> struct SyncGroup {
  int id;
  __device__ __forceinline__ void operator()() const {
#ifdef __CUDA_ARCH__
    asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(NTH) : "memory");
#else
    __syncthreads();   // host execution: one barrier for the block
#endif
  }
};
// The barrier of a sequence of T threads, `per_cta` sequences in the CTA (consecutive threads).  A CTA has
// 16 hardware barriers, the first of them __syncthreads': 15 sequences of more than a warp.
__host__ __device__ constexpr int seq_max(int t) { return t <= 32 ? 1024 : 15; }
template <int T, int PER_CTA> struct SeqSync {
  static_assert(PER_CTA <= seq_max(T), "a hardware barrier for every sequence");
  __device__ __forceinline__ static auto make(int seq) {
    if constexpr (T <= 32) return SyncWarp{};
    else if constexpr (PER_CTA == 1) return SyncCta{};
    else return SyncGroup<T>{seq};
  }
};

// The pointer, opaque to the optimiser: loads through it are not moved out of the
// loop that takes it (a rolled loop of transforms would otherwise keep every
// twiddle and factor of an iteration in registers, and spill them).
template <class P> __device__ __forceinline__ P* fresh(P* p) {
#ifdef __CUDA_ARCH__
  asm volatile("" : "+l"(p));
#endif
  return p;
}

// Tensor memory as a per-thread register file: NR 32-bit registers a thread, thread
// l of warp w in lane 32 (w % 4) + l, columns from (w / 4) NR.  Used to keep the
// Caldeira-Leggett base of a column out of registers and of the shared-memory
// pipe, which bounds the pass.  alloc / release by every thread of the CTA (warp 0
// acts); NR WARPS / 4 columns, a power of two in [32, 512]; the holders of an
// allocation never wait for another CTA, so an alloc that finds the columns taken
// waits for CTAs that run on.
#if defined(WIG_TMEM) && defined(__CUDA_ARCH__)
template <int NR, int WARPS> struct Tmem {
  static constexpr int COLS = NR * ((WARPS + 3) / 4);
  static_assert(NR % 16 == 0 && COLS >= 32 && COLS <= 512 && (COLS & (COLS - 1)) == 0, "tensor-memory columns");
  unsigned base, mine;
  __device__ __forceinline__ void alloc(unsigned* slot) {
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(slot)),
                   "n"(COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    base = *slot;
    const unsigned w = threadIdx.x >> 5;
    mine = base + ((w & 3u) << 21) + (w >> 2) * NR;
  }
  __device__ __forceinline__ void release() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x < 32)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS) : "memory");
  }
  // four double2 (16 registers) from column 16 q of the thread's slice
  __device__ __forceinline__ void put(int q, const double2* v) const {
    unsigned r[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[4 * i] = (unsigned)__double2loint(v[i].x);
      r[4 * i + 1] = (unsigned)__double2hiint(v[i].x);
      r[4 * i + 2] = (unsigned)__double2loint(v[i].y);
      r[4 * i + 3] = (unsigned)__double2hiint(v[i].y);
    }
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(mine + 16 * q),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
  }
  __device__ __forceinline__ static void put_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
  __device__ __forceinline__ void get(int q, double2* v) const {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(mine + 16 * q)
        : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = make_double2(__hiloint2double((int)r[4 * i + 1], (int)r[4 * i]),
                          __hiloint2double((int)r[4 * i + 3], (int)r[4 * i + 2]));
  }
};
#endif

// Programmatic dependent launch: a kernel launched with the attribute may start
// while its predecessor drains.  grid_wait() returns once the predecessor's
// memory is visible (at once without the attribute); every thread calls it
// before its first access to anything an earlier kernel writes.
__device__ __forceinline__ void grid_wait() {
#ifdef __CUDA_ARCH__
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}
__device__ __forceinline__ void grid_launch_next() {
#ifdef __CUDA_ARCH__
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

}  // namespace wig
