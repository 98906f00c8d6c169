// Register DFTs of the radices that the pass kernels use beside the ones of fft_device.cuh,
// and the in-place mixed-radix stages of one CTA (several transforms of one runtime length in
// shared memory).
#pragma once
#include "fft_device.cuh"

namespace fdr {

// DFT of an odd prime length from the sums and differences of the mirrored inputs:
// X[q], X[R-q] = (v0 + sum_m cos(2 pi q m / R) (v[m] + v[R-m]))
//                +- i sign (sum_m sin(2 pi q m / R) (v[m] - v[R-m])).
template <int R, class Table>
struct DftPrime {
  __device__ __forceinline__ static void run(float2* v, int sign) {
    constexpr int H = (R - 1) / 2;
    constexpr Table tab{};
    float2 t[H], d[H];
    float2 x0 = v[0];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      t[m] = cadd(v[m + 1], v[R - 1 - m]);
      d[m] = csub(v[m + 1], v[R - 1 - m]);
      x0 = cadd(x0, t[m]);
    }
    const float2 v0 = v[0];
    v[0] = x0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      float2 a = v0, b = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const float c = tab.c[(q * (m + 1)) % R], s = tab.s[(q * (m + 1)) % R];
        a = make_float2(fmaf(c, t[m].x, a.x), fmaf(c, t[m].y, a.y));
        b = make_float2(fmaf(s, d[m].x, b.x), fmaf(s, d[m].y, b.y));
      }
      const float2 ib = cmul_i(b, sign);
      v[q] = cadd(a, ib);
      v[R - q] = csub(a, ib);
    }
  }
};

// DFT of R1 * R2 points: R2-point DFTs over r = r1 + R1 * r2, the twiddles, R1-point DFTs.
template <int R1, int R2, class Table>
struct DftComposite {
  __device__ __forceinline__ static void run(float2* v, int sign) {
    constexpr Table tab{};
    float2 y[R1][R2];
#pragma unroll
    for (int r1 = 0; r1 < R1; ++r1) {
      float2 t[R2];
#pragma unroll
      for (int r2 = 0; r2 < R2; ++r2) t[r2] = v[r1 + R1 * r2];
      Dft<R2>::run(t, sign);
#pragma unroll
      for (int m2 = 0; m2 < R2; ++m2)
        y[r1][m2] = (r1 * m2) == 0 ? t[m2]
                                   : cmul(t[m2], make_float2(tab.c[r1 * m2], (float)sign * tab.s[r1 * m2]));
    }
#pragma unroll
    for (int m2 = 0; m2 < R2; ++m2) {
      float2 t[R1];
#pragma unroll
      for (int r1 = 0; r1 < R1; ++r1) t[r1] = y[r1][m2];
      Dft<R1>::run(t, sign);
#pragma unroll
      for (int m1 = 0; m1 < R1; ++m1) v[m2 + R2 * m1] = t[m1];
    }
  }
};

// DFT of R1 * R2 points, R1 and R2 coprime, without twiddles (Good's mapping): inputs R2 n1 + R1 n2,
// outputs E1 k1 + E2 k2 (mod R1 R2) with E1 = 1 mod R1 and 0 mod R2, E2 = 0 mod R1 and 1 mod R2.
template <int R1, int R2, int E1, int E2>
struct DftCoprime {
  static_assert(E1 % R1 == 1 && E1 % R2 == 0 && E2 % R1 == 0 && E2 % R2 == 1, "output mapping");
  __device__ __forceinline__ static void run(float2* v, int sign) {
    float2 y[R1][R2];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) y[n1][n2] = v[(R2 * n1 + R1 * n2) % (R1 * R2)];
      Dft<R2>::run(y[n1], sign);
    }
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      float2 t[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) t[n1] = y[n1][k2];
      Dft<R1>::run(t, sign);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) v[(E1 * k1 + E2 * k2) % (R1 * R2)] = t[k1];
    }
  }
};

// cos and sin of 2 pi m / n
struct CosSin7 {
  float c[7] = {
      1.00000000000000000f, 0.62348980185873359f, -0.22252093395631434f, -0.90096886790241903f,
      -0.90096886790241915f, -0.22252093395631459f, 0.62348980185873337f};
  float s[7] = {
      0.00000000000000000f, 0.78183148246802980f, 0.97492791218182362f, 0.43388373911755823f,
      -0.43388373911755801f, -0.97492791218182362f, -0.78183148246802991f};
};
struct CosSin9 {
  float c[9] = {
      1.00000000000000000f, 0.76604444311897801f, 0.17364817766693041f, -0.49999999999999978f,
      -0.93969262078590832f, -0.93969262078590843f, -0.50000000000000044f, 0.17364817766692997f,
      0.76604444311897779f};
  float s[9] = {
      0.00000000000000000f, 0.64278760968653925f, 0.98480775301220802f, 0.86602540378443871f,
      0.34202014332566888f, -0.34202014332566866f, -0.86602540378443837f, -0.98480775301220813f,
      -0.64278760968653958f};
};
struct CosSin11 {
  float c[11] = {
      1.00000000000000000f, 0.84125353283118121f, 0.41541501300188644f, -0.14231483827328500f,
      -0.65486073394528499f, -0.95949297361449737f, -0.95949297361449748f, -0.65486073394528521f,
      -0.14231483827328523f, 0.41541501300188605f, 0.84125353283118121f};
  float s[11] = {
      0.00000000000000000f, 0.54064081745559756f, 0.90963199535451833f, 0.98982144188093280f,
      0.75574957435425827f, 0.28173255684142967f, -0.28173255684142939f, -0.75574957435425816f,
      -0.98982144188093268f, -0.90963199535451855f, -0.54064081745559744f};
};
struct CosSin13 {
  float c[13] = {
      1.00000000000000000f, 0.88545602565320991f, 0.56806474673115592f, 0.12053668025532301f,
      -0.35460488704253545f, -0.74851074817110119f, -0.97094181742605201f, -0.97094181742605212f,
      -0.74851074817110130f, -0.35460488704253590f, 0.12053668025532320f, 0.56806474673115481f,
      0.88545602565321002f};
  float s[13] = {
      0.00000000000000000f, 0.46472317204376851f, 0.82298386589365635f, 0.99270887409805397f,
      0.93501624268541483f, 0.66312265824079519f, 0.23931566428755768f, -0.23931566428755743f,
      -0.66312265824079497f, -0.93501624268541472f, -0.99270887409805397f, -0.82298386589365702f,
      -0.46472317204376840f};
};

template <> struct Dft<6> : DftCoprime<2, 3, 3, 4> {};
template <> struct Dft<7> : DftPrime<7, CosSin7> {};
template <> struct Dft<9> : DftComposite<3, 3, CosSin9> {};
template <> struct Dft<10> : DftCoprime<2, 5, 5, 6> {};
template <> struct Dft<11> : DftPrime<11, CosSin11> {};
template <> struct Dft<13> : DftPrime<13, CosSin13> {};

// ------------------------------------------------------------------------------------
// In-place stages over `bpc` transforms of one length L = R_0 R_1 ... in shared memory, at most
// kStageElems points in all (decimation in frequency).  Stage s transforms R_s elements n_s / R_s
// apart of every block of n_s = L / (R_0 .. R_{s-1}) elements and leaves output m, times
// exp(-+ 2 pi i jj m / n_s), in the place of input m, so that a butterfly reads and writes the
// same places: one buffer, one barrier a stage, a loop over butterflies whose code is one
// butterfly long.  (Stages that first take all of a thread's butterflies into registers spent
// most of their time on instruction fetches: their code ran once per CTA.)  The first stage takes
// its inputs straight from global memory; the last one, whose butterfly j in digit order
// m_0 + R_0 m_1 + ... holds the outputs j + m L / R, hands them to global memory.
// Element (m_0, rest) of transform i is at i * SS + m_0 * pitch + rest with pitch odd and
// SS = 16 / bpc (mod 16) (1 from bpc = 16 on): a half-warp of neighbouring transforms (lanes over
// i) and one of neighbouring butterflies both meet 16 different 8-byte banks.
// ------------------------------------------------------------------------------------
constexpr int kStageThreads = 256;
constexpr int kStageCtas = 3;  // per SM: up to 85 registers a thread, 72 KB of shared memory
constexpr int kStageElems = 32 * kStageThreads;
constexpr int kStageMax = 8;

struct StageDesc {
  int L, nst, bpc, bpc_log2, SS, pitch;
  int radix[kStageMax];
  int nbf[kStageMax];              // L / radix: butterflies of one transform
  int Ns[kStageMax];               // product of the earlier radices
  int step[kStageMax];             // n_s / radix: distance of a butterfly's elements
  int digit[kStageMax];            // place value of digit m_s of a position
  unsigned radix_magic[kStageMax]; // of div_magic
  unsigned nbf_magic[kStageMax];
  const float2* roots;             // exp(-2 pi i m / L), m < L
};

// n / d for n < 2^13 from magic = ceil(2^32 / d) (0 stands for d = 1): the excess of the
// product, below 2^13 / 2^32, is less than the 1 / d that separates it from the next integer.
__device__ __forceinline__ int div_magic(int n, unsigned magic) {
  return magic ? (int)__umulhi((unsigned)n, magic) : n;
}

// Position of butterfly j of stage s (j in digit order, the element jj within the block last);
// *jj receives that element.
__device__ __forceinline__ int stage_pos(const StageDesc& d, int s, int j, int* jj) {
  int pos = 0;
  for (int t = 0; t < s; ++t) {
    const int q = div_magic(j, d.radix_magic[t]);
    pos += (j - q * d.radix[t]) * d.digit[t];
    j = q;
  }
  *jj = j;
  return pos + j;
}

// exp(SIGN 2 pi i jj m / n_s) on the elements m of a butterfly of stage s.
template <int R, int SIGN>
__device__ __forceinline__ void stage_twiddle(const StageDesc& d, int s, int jj, float2* v) {
  const int step = jj * d.Ns[s];
#pragma unroll
  for (int m = 1; m < R; ++m) {
    float2 t = __ldg(d.roots + m * step);
    if (SIGN > 0) t.y = -t.y;
    v[m] = cmul(v[m], t);
  }
}

// First stage.  get(i)(l): element l of transform i.  lane_i: neighbouring threads take
// neighbouring transforms (else neighbouring elements).
template <int R, int SIGN, class Get>
__device__ __forceinline__ void stage_first(const StageDesc& d, bool lane_i, float2* sm, Get get) {
  const int nbf = d.nbf[0], total = nbf << d.bpc_log2;
  for (int j = threadIdx.x; j < total; j += blockDim.x) {
    const int i = lane_i ? j & (d.bpc - 1) : div_magic(j, d.nbf_magic[0]);
    const int jj = lane_i ? j >> d.bpc_log2 : j - i * nbf;
    float2 v[R];
    auto row = get(i);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = row(jj + r * nbf);
    Dft<R>::run(v, SIGN);
    if (d.nst > 1) stage_twiddle<R, SIGN>(d, 0, jj, v);
    float2* o = sm + i * d.SS + jj;
#pragma unroll
    for (int m = 0; m < R; ++m) o[m * d.pitch] = v[m];
  }
}

// A stage within shared memory.  TIME: the mirrored stage of a transform that takes its input in
// the order this one leaves (decimation in time: twiddles before the butterfly).
template <int R, int SIGN, bool TIME>
__device__ __forceinline__ void stage_mid(const StageDesc& d, int s, float2* sm) {
  const int total = d.nbf[s] << d.bpc_log2;
  const int step = s == 0 ? d.pitch : d.step[s];
  for (int j = threadIdx.x; j < total; j += blockDim.x) {
    int jj;
    float2* const o = sm + (j & (d.bpc - 1)) * d.SS + stage_pos(d, s, j >> d.bpc_log2, &jj);
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = o[r * step];
    if (TIME) stage_twiddle<R, SIGN>(d, s, jj, v);
    Dft<R>::run(v, SIGN);
    if (!TIME) stage_twiddle<R, SIGN>(d, s, jj, v);
#pragma unroll
    for (int r = 0; r < R; ++r) o[r * step] = v[r];
  }
}

// Last stage.  put(i)(l, v) takes output l of transform i.
template <int R, int SIGN, class Put>
__device__ __forceinline__ void stage_last(const StageDesc& d, bool lane_i, const float2* sm, Put put) {
  const int s = d.nst - 1, nbf = d.nbf[s], total = nbf << d.bpc_log2;
  const int step = s == 0 ? d.pitch : 1;
  for (int j = threadIdx.x; j < total; j += blockDim.x) {
    const int i = lane_i ? j & (d.bpc - 1) : div_magic(j, d.nbf_magic[s]);
    const int jj = lane_i ? j >> d.bpc_log2 : j - i * nbf;
    int within;
    const float2* const o = sm + i * d.SS + stage_pos(d, s, jj, &within);
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = o[r * step];
    Dft<R>::run(v, SIGN);
    auto row = put(i);
#pragma unroll
    for (int m = 0; m < R; ++m) row(jj + m * nbf, v[m]);
  }
}

// Last forward stage, the product with factor(i)(l) and the first backward stage.
template <int R, class Factor>
__device__ __forceinline__ void stage_turn(const StageDesc& d, float2* sm, Factor factor) {
  const int s = d.nst - 1, nbf = d.nbf[s], total = nbf << d.bpc_log2;
  const int step = s == 0 ? d.pitch : 1;
  for (int j = threadIdx.x; j < total; j += blockDim.x) {
    const int i = j & (d.bpc - 1), jj = j >> d.bpc_log2;
    auto row = factor(i);
    float2 f[R], v[R];
#pragma unroll
    for (int m = 0; m < R; ++m) f[m] = row(jj + m * nbf);
    int within;
    float2* const o = sm + i * d.SS + stage_pos(d, s, jj, &within);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = o[r * step];
    Dft<R>::run(v, -1);
#pragma unroll
    for (int m = 0; m < R; ++m) v[m] = cmul(v[m], f[m]);
    Dft<R>::run(v, +1);
#pragma unroll
    for (int r = 0; r < R; ++r) o[r * step] = v[r];
  }
}

#define FDR_FOR_RADIX(X) X(16) X(13) X(11) X(10) X(9) X(8) X(7) X(6) X(5) X(4) X(3) X(2)

// All stages of d (nst >= 2: a single stage passes through shared memory all the same); the
// block must be synchronised before if shared memory is still being read.
template <int SIGN, class Get, class Put>
__device__ __forceinline__ void stages_run(const StageDesc& d, bool first_lane_i, bool last_lane_i,
                                           float2* sm, Get get, Put put) {
  if (d.nst == 1) {  // L <= 16: the butterfly is the transform
    for (int e = threadIdx.x; e < d.L << d.bpc_log2; e += blockDim.x)
      sm[(e & (d.bpc - 1)) * d.SS + (e >> d.bpc_log2) * d.pitch] = get(e & (d.bpc - 1))(e >> d.bpc_log2);
  } else {
    switch (d.radix[0]) {
#define FDR_STAGE(R) case R: stage_first<R, SIGN>(d, first_lane_i, sm, get); break;
      FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
    }
  }
  __syncthreads();
  for (int s = 1; s + 1 < d.nst; ++s) {
    switch (d.radix[s]) {
#define FDR_STAGE(R) case R: stage_mid<R, SIGN, false>(d, s, sm); break;
      FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
    }
    __syncthreads();
  }
  switch (d.radix[d.nst - 1]) {
#define FDR_STAGE(R) case R: stage_last<R, SIGN>(d, last_lane_i, sm, put); break;
    FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
  }
}

// Place of element l of a transform in shared memory.
__device__ __forceinline__ int stage_place(const StageDesc& d, int l) {
  const int m0 = div_magic(l, d.nbf_magic[0] /* n_1 = L / R_0 */);
  return l + m0 * (d.pitch - d.nbf[0]);
}

// Circular convolution of the transforms in shared memory (element l of transform i at
// i * SS + stage_place(l)) with the spectrum factor(i)(l), unnormalised.
template <class Factor>
__device__ __forceinline__ void convolve_smem(const StageDesc& d, float2* sm, Factor factor) {
  for (int s = 0; s + 1 < d.nst; ++s) {
    switch (d.radix[s]) {
#define FDR_STAGE(R) case R: stage_mid<R, -1, false>(d, s, sm); break;
      FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
    }
    __syncthreads();
  }
  switch (d.radix[d.nst - 1]) {
#define FDR_STAGE(R) case R: stage_turn<R>(d, sm, factor); break;
    FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
  }
  __syncthreads();
  for (int s = d.nst - 2; s >= 0; --s) {
    switch (d.radix[s]) {
#define FDR_STAGE(R) case R: stage_mid<R, +1, true>(d, s, sm); break;
      FDR_FOR_RADIX(FDR_STAGE)
#undef FDR_STAGE
    }
    __syncthreads();
  }
}

// Tables of the four-step twiddles (TwiddleTables below): log2 of the outputs l that share a coarse
// factor, rows of coarse factors and bytes.
__host__ __device__ constexpr int tw_fine(int L) {
  int lg = 0;
  while ((32 << lg) <= L && lg < 5) ++lg;
  return lg;
}
__host__ __device__ constexpr int tw_rows(int L) { return ((L + (1 << tw_fine(L)) - 1) >> tw_fine(L)) | 1; }
__host__ __device__ inline size_t tw_bytes(int L, int bpc) {
  return 16 + (size_t)bpc * (sizeof(float4) * tw_rows(L) + sizeof(float2) * ((1 << tw_fine(L)) + 1));
}

// Fills d for `groups` sets of `nb` transforms of length L, neighbouring transforms of a set at
// neighbouring addresses (rows: CTAs then take at least 8 of them, 64 bytes a row); false if L
// has a prime factor above 13 or exceeds kStageElems.  `twiddles`: the pass keeps twiddle tables
// beside its transforms; both stay within kStageSmem.
constexpr size_t kStageSmem = 112 * 1024;  // two CTAs per SM
bool stage_plan(int64_t L, int64_t nb, int64_t groups, bool rows, bool twiddles, StageDesc* d);
size_t stage_smem_bytes(const StageDesc& d);
int stage_threads(const StageDesc& d);

// Four-step twiddle exp(SIGN 2 pi i l b / N) of the CTA's transforms b, as the product of a coarse
// factor for l >> lg (rounded value and its residue) and a fine one for the rest of l (its difference
// from 1), 2^lg of them, lg = tw_fine(L) with 2^lg <= L / 16: the fine angles stay below 2 pi / 16.
// All values come from float64, once per CTA, eight of a table from one sincospi and the float64
// powers of another.  Error in units of a rounded value's rms: 1.00 to 1.05 (1.05 to 1.5 for L < 512
// with 32 fine factors whatever L; finer tables of L = 400 brought a CTA above 64 KB, and the pass from
// 58 to 67 us).
struct TwiddleTables {
  int hi, lo;  // where they start in shared memory, in float4 and float2
  int nh, lg;  // rows of coarse factors per transform; lg
};

inline TwiddleTables twiddle_tables(const StageDesc& d) {
  TwiddleTables t;
  t.nh = tw_rows(d.L);
  t.lg = tw_fine(d.L);
  t.hi = (d.bpc * d.SS + 1) / 2;
  t.lo = 2 * (t.hi + d.bpc * t.nh);
  return t;
}

template <int SIGN>
__device__ __forceinline__ void fill_twiddles(const TwiddleTables& t, float4* sm4, int bpc, int L, long long b1_0,
                                              double inv2N) {
  const int nl = 1 << t.lg, nh = (L + nl - 1) >> t.lg, gh = (nh + 7) / 8, groups = gh + (nl + 7) / 8;
  float4* const hi = sm4 + t.hi;
  float2* const lo = reinterpret_cast<float2*>(sm4) + t.lo;
  for (int e = threadIdx.x; e < bpc * groups; e += blockDim.x) {
    const int i = e / groups, g = e - i * groups;
    const bool fine = g >= gh;
    const int m0 = 8 * (fine ? g - gh : g), n = min(8, (fine ? nl : nh) - m0);
    const long long b = (b1_0 + i) << (fine ? 0 : t.lg);
    double c, s, wc, ws;
    sincospi((double)(m0 * b) * inv2N, &s, &c);
    sincospi((double)b * inv2N, &ws, &wc);
    for (int u = 0; u < n; ++u) {
      const double ss = SIGN * s;
      if (fine) {
        lo[i * (nl + 1) + m0 + u] = make_float2((float)(c - 1.0), (float)ss);
      } else {
        const float x = (float)c, y = (float)ss;
        hi[i * t.nh + m0 + u] = make_float4(x, y, (float)(c - x), (float)(ss - y));
      }
      const double cn = c * wc - s * ws;
      s = c * ws + s * wc;
      c = cn;
    }
  }
}

// Factor of output l from a transform's rows of the tables.
__device__ __forceinline__ float2 twiddle_at(const float4* hi, const float2* lo, int lg, int l) {
  const float4 h = hi[l >> lg];
  const float2 e = lo[l & ((1 << lg) - 1)];
  return make_float2(h.x + fmaf(h.x, e.x, fmaf(-h.y, e.y, h.z)), h.y + fmaf(h.x, e.y, fmaf(h.y, e.x, h.w)));
}

}  // namespace fdr
