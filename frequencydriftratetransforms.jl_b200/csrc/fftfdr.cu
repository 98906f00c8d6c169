// Fourier-domain shift FDR (src/fftfdr.jl of FrequencyDriftRateTransforms.jl):
// fftfdr_workspace (:39-59), fftfdr_workspace! (:69-84), fdshiftsum! (:86-96),
// fdshift! (:104-111), fftfdr! (:126-134).
//
// The phasor of time step t and channel-bin k is cispi(2*k*t*r/Nf) with the argument
// formed in Float32 exactly as the reference does (fftfdr.jl:10-12): Float32(2*k*t) * r,
// then / Float32(Nf), each rounded once.  The sum over t runs in time order from zero in
// complex float32, as Base's sum! over dims=2 accumulates.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "fft_engine.cuh"

struct fdr_fft_ws {
  int64_t Nf = 0, Nt = 0, K = 0;
  float2* F = nullptr;        // dest_rfft (K x Nt)
  float2* P = nullptr;        // dest_phasor (K x Nt)
  float2* S = nullptr;        // per-rate sums (K x kRateChunk)
  float2* rscratch = nullptr;
  int64_t rscratch_pairs = 0;
};

namespace fdr {

constexpr int kRateChunk = 32;

struct RateParams {
  float r[kRateChunk];
};

__device__ __forceinline__ float2 phasor_ref(long long k, long long t, float r, float Nf_f) {
  float x = __fdiv_rn(__fmul_rn(__ll2float_rn(2 * k * t), r), Nf_f);
  return cispif(x);
}

// S[k + jj*K] = sum_t F[k, t] * phasor(k, t, r_jj).  A thread takes one bin and RPT
// rates, two per packed operation, so F is read once for all of them; the time goes to the phasors,
// one for each (k, t, r).  Their arguments are formed by the same rounded operations as in
// phasor_ref, with cheaper instructions where they give the same value: for MULT (2k and t exact in
// Float32) the rounded product Float32(2k) * Float32(t) is Float32(2kt), and for a power-of-two Nf
// the quotient is the product with 1 / Nf.  For a small rate (every |argument| < 2^19 half-turns) the
// nearest quarter turn is the sum with 1.5 * 2^23 rounded, its low bits the quadrant, and the rest
// is exact; the other rates, if any (LARGE: the bits of `large`), take cispif.  Each rate is decided
// by itself, so that a column does not depend on the rates beside it.  At Nf = 2^20, Nt = 16, 21
// rates: 440 us with a thread per sum and sincospif, 246 us with 8 rates per thread, 201 us with
// packed polynomials (179 us without EXACT, whose error was above that of sincospif).
// RPT is 8 where that fills the GPU; a grid of less than one CTA an SM takes a pair per
// thread, a quarter of the chain (calls of 16 rates at Nf = 10,200: 149 -> 132 us, 131 with a thread per
// sum; 8 rates and 64 steps at Nf = 4096: 42 -> 27 us, 68 with a thread per sum).
constexpr int kRatesPerThread = 8;

template <int RPT, bool MULT, bool POW2, bool LARGE>
__global__ void __launch_bounds__(256) phasor_sum_kernel(const float2* __restrict__ F, long long K, int Nt,
                                                         long long Nf, int nr, unsigned large,
                                                         float2* __restrict__ S,
                                                         const __grid_constant__ RateParams rp) {
  const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= K) return;
  const int j0 = blockIdx.y * RPT;
  const float Nf_f = __ll2float_rn(Nf), inv = 1.f / Nf_f, k2 = __ll2float_rn(2 * k);
  float2 ax[RPT / 2], ay[RPT / 2];  // lanes: rates 2q and 2q + 1
#pragma unroll
  for (int q = 0; q < RPT / 2; ++q) ax[q] = ay[q] = make_float2(0.f, 0.f);
  for (int t = 0; t < Nt; ++t) {
    const float2 f = __ldg(F + k + t * K);
    const float2 fx = pk_set(f.x), fy = pk_set(f.y);
    const float kt = MULT ? __fmul_rn(k2, (float)t) : __ll2float_rn(2 * k * t);
#pragma unroll
    for (int q = 0; q < RPT / 2; ++q) {
      if (j0 + 2 * q < nr) {  // uniform; rates past the last are zero
        const float2 x = pk_mul(pk_set(kt), make_float2(rp.r[j0 + 2 * q], rp.r[j0 + 2 * q + 1]));
        const float2 h = POW2 ? pk_mul(x, pk_set(inv)) : make_float2(__fdiv_rn(x.x, Nf_f), __fdiv_rn(x.y, Nf_f));
        const float2 h2 = pk_add(h, h);
        const float2 m = pk_add(h2, pk_set(12582912.f));
        const float2 rest = csub(h2, pk_add(m, pk_set(-12582912.f)));
        float2 c, s;
        cis_quarter_pk<true>(rest, __float_as_uint(m.x), __float_as_uint(m.y), c, s);
        if (LARGE) {
          const unsigned two = large >> (j0 + 2 * q);  // uniform
          if (two & 1) {
            const float2 p = cispif(h.x);
            c.x = p.x;
            s.x = p.y;
          }
          if (two & 2) {
            const float2 p = cispif(h.y);
            c.y = p.x;
            s.y = p.y;
          }
        }
        // cmul_rn and a rounded sum, for both rates
        ax[q] = pk_add(ax[q], csub(pk_mul(fx, c), pk_mul(fy, s)));
        ay[q] = pk_add(ay[q], pk_add(pk_mul(fx, s), pk_mul(fy, c)));
      }
    }
  }
#pragma unroll
  for (int q = 0; q < RPT / 2; ++q) {
    if (j0 + 2 * q < nr) S[k + (j0 + 2 * q) * K] = make_float2(ax[q].x, ay[q].x);
    if (j0 + 2 * q + 1 < nr) S[k + (j0 + 2 * q + 1) * K] = make_float2(ax[q].y, ay[q].y);
  }
}

// P[k, t] = F[k, t] * phasor(k, t, r)
__global__ void phasor_kernel(const float2* __restrict__ F, long long K, long long Nt, long long Nf,
                              float r, float2* __restrict__ P) {
  const long long total = K * Nt;
  const float Nf_f = __ll2float_rn(Nf);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long t = e / K, k = e - t * K;
    P[e] = cmul_rn(F[e], phasor_ref(k, t, r, Nf_f));
  }
}

static unsigned grid_1d(long long total) {
  long long b = cdiv(total, 256);
  long long cap = (long long)sm_count() * 16;
  return (unsigned)std::max(1LL, std::min(b, cap));
}

static void release(fdr_fft_ws* ws) {
  if (!ws) return;
  cudaFree(ws->F);
  cudaFree(ws->P);
  cudaFree(ws->S);
  cudaFree(ws->rscratch);
  delete ws;
}

}  // namespace fdr

using namespace fdr;

extern "C" {

int fdr_fftfdr_workspace(fdr_fft_ws** out, const float* spectrogram, int64_t Nf, int64_t Nt,
                         fdr_stream_t stream) {
  FDR_CHECK_ARG(out && spectrogram, "fftfdr_workspace: NULL argument");
  FDR_CHECK_ARG(Nf >= 1 && Nt >= 1, "fftfdr_workspace: bad sizes");
  *out = nullptr;
  fdr_fft_ws* ws = new fdr_fft_ws();
  ws->Nf = Nf; ws->Nt = Nt; ws->K = Nf / 2 + 1;
  const int64_t K = ws->K;
  const int64_t per = real_fft_scratch_per_pair(Nf);
  int64_t pairs = cdiv(std::max<int64_t>(Nt, kRateChunk), 2);
  const int64_t cap = std::max<int64_t>(1, (int64_t(256) << 20) / (int64_t)(per * sizeof(float2)));
  ws->rscratch_pairs = std::min(pairs, cap);
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMalloc(&ws->F, sizeof(float2) * K * Nt);
  if (e == cudaSuccess) e = cudaMalloc(&ws->P, sizeof(float2) * K * Nt);
  if (e == cudaSuccess) e = cudaMalloc(&ws->S, sizeof(float2) * K * kRateChunk);
  if (e == cudaSuccess) e = cudaMalloc(&ws->rscratch, sizeof(float2) * per * ws->rscratch_pairs);
  if (e != cudaSuccess) {
    int st = cuda_status(e, "fftfdr_workspace allocation");
    release(ws);
    return st;
  }
  int st = fdr_fftfdr_workspace_update(ws, spectrogram, Nf, Nt, stream);
  if (st != FDR_OK) { release(ws); return st; }
  *out = ws;
  return FDR_OK;
}

int fdr_fftfdr_workspace_update(fdr_fft_ws* ws, const float* spectrogram, int64_t Nf, int64_t Nt,
                                fdr_stream_t stream) {
  FDR_CHECK_ARG(ws && spectrogram, "fftfdr_workspace!: NULL argument");
  // fftfdr.jl:71-76
  FDR_CHECK_ARG(Nf == ws->Nf && Nt == ws->Nt, "input spectrogram has unexpected size");
  return rfft_columns(spectrogram, Nf, Nt, Nf, ws->F, ws->K, ws->rscratch, ws->rscratch_pairs,
                      (cudaStream_t)stream);
}

int fdr_fftfdr_destroy(fdr_fft_ws* ws) {
  if (ws) {
    cudaDeviceSynchronize();
    release(ws);
  }
  return FDR_OK;
}

int fdr_fftfdr_rfft_buffer(fdr_fft_ws* ws, void** F) {
  FDR_CHECK_ARG(ws && F, "NULL argument");
  *F = ws->F;
  return FDR_OK;
}

int fdr_fdshiftsum(fdr_fft_ws* ws, float rate, float* dest, fdr_stream_t stream) {
  FDR_CHECK_ARG(ws && dest, "fdshiftsum!: NULL argument");
  return fdr_fftfdr(ws, &rate, 1, dest, stream);
}

int fdr_fdshift(fdr_fft_ws* ws, float rate, float* dest, fdr_stream_t stream) {
  FDR_CHECK_ARG(ws && dest, "fdshift!: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  phasor_kernel<<<grid_1d(ws->K * ws->Nt), 256, 0, s>>>(ws->F, ws->K, ws->Nt, ws->Nf, rate, ws->P);
  FDR_LAUNCH_CHECK("phasor_kernel");
  return irfft_columns(ws->P, ws->K, ws->Nt, ws->Nf, dest, ws->Nf, ws->rscratch,
                       ws->rscratch_pairs, s);
}

int fdr_fftfdr(fdr_fft_ws* ws, const float* rates, int64_t Nr, float* fdr, fdr_stream_t stream) {
  FDR_CHECK_ARG(ws && fdr, "fftfdr!: NULL argument");
  FDR_CHECK_ARG(Nr >= 0 && (Nr == 0 || rates), "fftfdr!: bad rates");
  cudaStream_t s = (cudaStream_t)stream;
  RateParams rp;
  for (int64_t j0 = 0; j0 < Nr; j0 += kRateChunk) {
    const int nr = (int)std::min<int64_t>(kRateChunk, Nr - j0);
    memset(&rp, 0, sizeof(rp));
    for (int i = 0; i < nr; ++i) rp.r[i] = rates[j0 + i];
    const bool mult = 2 * ws->K < (1LL << 24) && ws->Nt < (1LL << 24), pow2 = is_pow2(ws->Nf);
    unsigned large = 0;  // rates with |argument| = 2 k t |r| / Nf possibly 2^19 or more, NaN among them
    static_assert(kRateChunk == 32, "one bit per rate");
    for (int i = 0; i < nr; ++i)
      if (!((double)fabsf(rp.r[i]) * (double)ws->Nt < (double)(1 << 19))) large |= 1u << i;
    auto launch = [&](auto rpt) {
      constexpr int RPT = decltype(rpt)::value;
      auto pick = [&](auto m, auto p2) {
        constexpr bool M = decltype(m)::value, P = decltype(p2)::value;
        return large ? phasor_sum_kernel<RPT, M, P, true> : phasor_sum_kernel<RPT, M, P, false>;
      };
      const std::true_type yes;
      const std::false_type no;
      auto kernel = mult ? (pow2 ? pick(yes, yes) : pick(yes, no)) : (pow2 ? pick(no, yes) : pick(no, no));
      const dim3 grid((unsigned)cdiv(ws->K, 256), (unsigned)cdiv(nr, RPT));
      kernel<<<grid, 256, 0, s>>>(ws->F, ws->K, (int)ws->Nt, ws->Nf, nr, large, ws->S, rp);
    };
    const bool full = cdiv(ws->K, 256) * cdiv(nr, kRatesPerThread) >= sm_count();
    if (full) launch(std::integral_constant<int, kRatesPerThread>());
    else launch(std::integral_constant<int, 2>());
    FDR_LAUNCH_CHECK("phasor_sum_kernel");
    FDR_TRY(irfft_columns(ws->S, ws->K, nr, ws->Nf, fdr + j0 * ws->Nf, ws->Nf, ws->rscratch,
                          ws->rscratch_pairs, s));
  }
  return FDR_OK;
}

}  // extern "C"
