// Generic batched FFT engine: see fft_engine.cuh.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "fft_engine.cuh"
#include "fft_stages.cuh"

namespace fdr {

// ------------------------------------------------------------------------------------
// Planning
// ------------------------------------------------------------------------------------
bool plan_radices(long long L, int* radix, int* nst) {
  int n = 0;
  long long m = L;
  while (m % 8 == 0 && n < kMaxStages) { radix[n++] = 8; m /= 8; }
  while (m % 4 == 0 && n < kMaxStages) { radix[n++] = 4; m /= 4; }
  while (m % 2 == 0 && n < kMaxStages) { radix[n++] = 2; m /= 2; }
  for (int p = 3; p <= kMaxRadixPrime && m > 1; p += 2) {
    while (m % p == 0 && n < kMaxStages) { radix[n++] = p; m /= p; }
  }
  *nst = n;
  return m == 1;
}

int get_roots(long long L, const float2** roots) {
  static std::mutex mu;
  static std::map<std::pair<int, long long>, float2*> cache;
  int dev = 0;
  FDR_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto key = std::make_pair(dev, L);
  auto it = cache.find(key);
  if (it != cache.end()) { *roots = it->second; return FDR_OK; }
  std::vector<float2> h((size_t)L);
  for (long long m = 0; m < L; ++m) {
    // exp(-2*pi*i*m/L) with the angle reduced to the first half-turn pair in double
    double a = -2.0 * (double)m / (double)L;  // half-turns
    double c = cos(M_PI * a), sn = sin(M_PI * a);
    h[(size_t)m] = make_float2((float)c, (float)sn);
  }
  float2* d = nullptr;
  FDR_CUDA(cudaMalloc(&d, sizeof(float2) * (size_t)L));
  FDR_CUDA(cudaMemcpy(d, h.data(), sizeof(float2) * (size_t)L, cudaMemcpyHostToDevice));
  cache[key] = d;
  *roots = d;
  return FDR_OK;
}

// ------------------------------------------------------------------------------------
// Small DFT kernels on register arrays.  sign: -1 forward, +1 backward.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float2 root_at(const float2* roots, int m, int sign) {
  float2 w = __ldg(roots + m);
  return sign > 0 ? cconj(w) : w;
}

// One Stockham stage of radix R over bpc transforms of length L held in shared memory.
template <int R>
__device__ __forceinline__ void stage_fixed(const float2* __restrict__ A, float2* __restrict__ B,
                                            int L, int bpc, int Ns, int sign,
                                            const float2* roots) {
  const int nbf = L / R;
  const int total = nbf * bpc;
  const int stride = L / (Ns * R);
  for (int j = threadIdx.x; j < total; j += blockDim.x) {
    const int i = j / nbf;
    const int jj = j - i * nbf;
    const int k = jj % Ns;
    const float2* a = A + (size_t)i * L;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = a[jj + r * nbf];
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], root_at(roots, r * k * stride, sign));
    }
    Dft<R>::run(v, sign);
    const int base = (jj / Ns) * Ns * R + k;
    float2* b = B + (size_t)i * L;
#pragma unroll
    for (int r = 0; r < R; ++r) b[base + r * Ns] = v[r];
  }
}

// Direct DFT stage for any radix R <= kMaxRadixPrime (one output per thread iteration).
__device__ void stage_generic(const float2* __restrict__ A, float2* __restrict__ B, int L,
                              int bpc, int Ns, int R, int sign, const float2* roots) {
  const int nbf = L / R;
  const int total = nbf * bpc * R;
  const int stride = L / (Ns * R);
  const int rstep = L / R;  // roots[q*rstep] = exp(-2*pi*i*q/R)
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int m = e % R;
    const int j = e / R;
    const int i = j / nbf;
    const int jj = j - i * nbf;
    const int k = jj % Ns;
    const float2* a = A + (size_t)i * L;
    float2 acc = make_float2(0.f, 0.f);
    for (int r = 0; r < R; ++r) {
      float2 v = a[jj + r * nbf];
      if (Ns > 1 && r > 0) v = cmul(v, root_at(roots, r * k * stride, sign));
      int q = (r * m) % R;
      acc = cadd(acc, cmul(v, root_at(roots, q * rstep, sign)));
    }
    const int base = (jj / Ns) * Ns * R + k;
    B[(size_t)i * L + base + m * Ns] = acc;
  }
}

__global__ void __launch_bounds__(256) fft_pass_kernel(PassDesc d) {
  extern __shared__ float2 sm[];
  const int L = d.L, bpc = d.bpc;
  const long long b1_0 = (long long)blockIdx.x * bpc;
  const int nb = (int)min((long long)bpc, d.nb1 - b1_0);
  const int total = L * bpc;
  for (long long b0 = blockIdx.y; b0 < d.nb0; b0 += gridDim.y) {
    float2* A = sm;
    float2* B = sm + (size_t)L * bpc;
    // load
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      int i, l;
      if (d.ld_b1_fast) { i = e % bpc; l = e / bpc; } else { l = e % L; i = e / L; }
      float2 v = make_float2(0.f, 0.f);
      if (i < nb) v = d.in[b0 * d.is0 + (b1_0 + i) * d.is1 + (long long)l * d.isl];
      A[(size_t)i * L + l] = v;
    }
    __syncthreads();
    int Ns = 1;
    for (int s = 0; s < d.nst; ++s) {
      const int R = d.radix[s];
      switch (R) {
        case 2: stage_fixed<2>(A, B, L, bpc, Ns, d.sign, d.roots); break;
        case 3: stage_fixed<3>(A, B, L, bpc, Ns, d.sign, d.roots); break;
        case 4: stage_fixed<4>(A, B, L, bpc, Ns, d.sign, d.roots); break;
        case 5: stage_fixed<5>(A, B, L, bpc, Ns, d.sign, d.roots); break;
        case 8: stage_fixed<8>(A, B, L, bpc, Ns, d.sign, d.roots); break;
        default: stage_generic(A, B, L, bpc, Ns, R, d.sign, d.roots); break;
      }
      __syncthreads();
      float2* t = A; A = B; B = t;
      Ns *= R;
    }
    // store
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      int i, l;
      if (d.st_b1_fast) { i = e % bpc; l = e / bpc; } else { l = e % L; i = e / L; }
      if (i >= nb) continue;
      float2 v = A[(size_t)i * L + l];
      const long long b1 = b1_0 + i;
      if (d.tw_n) {
        const long long b = d.tw_dim == 1 ? b1 : b0;
        const long long m = ((long long)l * b) % d.tw_n;
        double sn, cs;
        sincospi(2.0 * (double)m / (double)d.tw_n, &sn, &cs);
        v = cmul(v, make_float2((float)cs, (float)(d.sign * sn)));
      }
      if (d.mul) v = cmul(v, d.mul[b0 * d.ms0 + b1 * d.ms1 + (long long)l * d.msl]);
      v = cscale(v, d.scale);
      d.out[b0 * d.os0 + b1 * d.os1 + (long long)l * d.osl] = v;
    }
    __syncthreads();
  }
}

int launch_pass(PassDesc d, cudaStream_t s) {
  if (!plan_radices(d.L, d.radix, &d.nst)) {
    set_error(FDR_ERR_UNSUPPORTED_SIZE, "FFT length %d has a prime factor > %d", d.L,
              kMaxRadixPrime);
    return FDR_ERR_UNSUPPORTED_SIZE;
  }
  FDR_TRY(get_roots(d.L, &d.roots));
  static bool attr_set[64] = {false};
  int dev = 0;
  FDR_CUDA(cudaGetDevice(&dev));
  const size_t smem = sizeof(float2) * 2 * (size_t)d.L * d.bpc;
  if (dev < 64 && !attr_set[dev]) {
    FDR_CUDA(cudaFuncSetAttribute(fft_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(float2) * 2 * kMaxCtaElems)));
    attr_set[dev] = true;
  }
  if (d.nb0 <= 0 || d.nb1 <= 0) return FDR_OK;
  dim3 grid((unsigned)cdiv(d.nb1, d.bpc), (unsigned)min(d.nb0, 65535LL));
  fft_pass_kernel<<<grid, 256, smem, s>>>(d);
  FDR_LAUNCH_CHECK("fft_pass_kernel");
  return FDR_OK;
}

static int pick_bpc(long long L, long long nb1) {
  long long b = kMaxCtaElems / L;
  if (b < 1) b = 1;
  long long p = 1;
  while (p * 2 <= b && p * 2 <= 64) p *= 2;
  if (p > nb1) {
    p = 1;
    while (p * 2 <= nb1) p *= 2;
  }
  return (int)p;
}

static PassDesc blank_pass() {
  PassDesc d;
  memset(&d, 0, sizeof(d));
  d.scale = 1.f;
  d.nb0 = 1;
  return d;
}


// ------------------------------------------------------------------------------------
// Passes over lengths whose prime factors are at most 13 (in-place stages of fft_stages.cuh).
// ------------------------------------------------------------------------------------
namespace {

// Radices of a plan of n with `left` stages, none above `top`, into r; the sum of the best (least; of
// equal ones the larger first radix), or 0.
int least_radices(int n, int left, int top, int* r) {
  static const int radices[] = {16, 13, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  int best = 0, rest[kStageMax];
  for (int x : radices) {
    int64_t most = 1;
    for (int k = 0; k < left; ++k) most *= x;
    if (most < n) break;  // nor do smaller radices reach n
    if (x > top || n % x) continue;
    int sum = left == 1 ? (x == n ? x : 0) : least_radices(n / x, left - 1, x, rest);
    if (sum == 0) continue;
    if (left > 1) sum += x;
    if (best && sum >= best) continue;
    best = sum;
    r[0] = x;
    for (int k = 1; k < left; ++k) r[k] = rest[k - 1];
  }
  return best;
}

unsigned magic_of(int d) { return d == 1 ? 0u : (unsigned)(((1ULL << 32) + d - 1) / d); }

}  // namespace

bool stage_plan(int64_t L, int64_t nb, int64_t groups, bool rows, bool twiddles, StageDesc* d) {
  if (L < 2 || L > kStageElems) return false;
  int64_t smooth = L;
  for (int p : {2, 3, 5, 7, 11, 13})
    while (smooth % p == 0) smooth /= p;
  if (smooth > 1) return false;
  memset(d, 0, sizeof(*d));
  d->L = (int)L;
  // fewest stages, then the least sum of radices
  while (++d->nst <= kStageMax && least_radices((int)L, d->nst, 16, d->radix) == 0) {}
  if (d->nst > kStageMax) return false;
  // the largest radix second: of the orders tried the least error at nearly every length (2^20: 0.99 of
  // that of radices 8, 8, 8, 2 in time order; largest first 1.01, and 3.7% less time)
  if (d->nst >= 3) std::swap(d->radix[0], d->radix[1]);
  int Ns = 1;
  for (int s = 0; s < d->nst; ++s) {
    const int R = d->radix[s];
    d->nbf[s] = d->L / R;
    d->Ns[s] = Ns;
    d->step[s] = d->L / (Ns * R);
    d->digit[s] = d->step[s];
    d->radix_magic[s] = magic_of(R);
    d->nbf_magic[s] = magic_of(d->nbf[s]);
    Ns *= R;
  }
  d->pitch = d->digit[0] = d->nbf[0] | 1;
  // as many transforms as the buffer holds, fewer when the grid would not reach two CTAs an SM
  int lg = 0;
  while ((L << (lg + 1)) <= kStageElems && lg < 8 && (int64_t(1) << lg) < nb) ++lg;
  while (lg > (rows ? 3 : 0) && cdiv(nb, int64_t(1) << lg) * groups < 2LL * sm_count()) --lg;
  // (the padding and the twiddle tables can take more than the elements do: L = 52, 128 transforms)
  for (;; --lg) {
    d->bpc_log2 = lg;
    d->bpc = 1 << lg;
    d->SS = (d->radix[0] * d->pitch + 15) / 16 * 16 + (d->bpc >= 16 ? 1 : 16 / d->bpc);
    const size_t bytes = stage_smem_bytes(*d) + (twiddles ? tw_bytes(d->L, d->bpc) : 0);
    if (bytes <= kStageSmem) return true;
    if (lg == 0) return false;
  }
}

// Threads of a CTA: two rounds of butterflies of the widest stage, up to kStageThreads.
int stage_threads(const StageDesc& d) {
  const int want = (d.nbf[d.nst - 1] << d.bpc_log2) / 2;
  return std::max(64, std::min(kStageThreads, (want + 31) / 32 * 32));
}
size_t stage_smem_bytes(const StageDesc& d) { return sizeof(float2) * (size_t)d.bpc * d.SS; }

namespace {

enum { kInComplex, kInRealPair, kInHalfPair };
enum { kOutComplex, kOutTwiddle, kOutRealPair };

struct StageArgs {
  StageDesc d;
  TwiddleTables tw;
  const void* in;
  void* out;
  const float2* mul;  // kOutComplex: pointwise factor addressed like the output, or NULL
  long long is0, is1, isl, os0, os1, osl;
  long long nb0, nb1;
  long long N, K;     // transform length of the columns and N/2 + 1
  long long p0, ncol;   // column pairs: first pair, columns in all
  long long ldi, ldo;   // column strides of the real columns or half spectra
  int pair_b1;        // the pair index is b1 (whole column in one CTA), else b0
  int in_lane_i, out_lane_i;
  float scale;
};

// One pass: several transforms of length L per CTA in shared memory (64 KB, three CTAs per SM at 80
// registers), the first stage reading and the last writing device memory.  Passes of Nf = 200,000,
// 81 columns back: 59 and 51 us (99 and 80 with the butterflies of a thread in registers across the
// stage, which spilled and ran into instruction fetches; the four Stockham kernels before both: over
// 400).  Bound by instruction issue (55 to 62%), a good part of it integer addressing of the runtime
// lengths, then by the latency of the loads.
template <int SIGN, int IN, int OUT>
__global__ void __launch_bounds__(kStageThreads, kStageCtas) fft_stage_kernel(const __grid_constant__ StageArgs a) {
  extern __shared__ float4 sm4[];
  float2* const sm = reinterpret_cast<float2*>(sm4);
  const StageDesc& d = a.d;
  const long long b1_0 = (long long)blockIdx.x << d.bpc_log2;
  const int nb = (int)min((long long)d.bpc, a.nb1 - b1_0);
  if (OUT == kOutTwiddle)  // the first stage's barrier follows
    fill_twiddles<SIGN>(a.tw, sm4, d.bpc, d.L, b1_0, 2.0 / (double)a.N);
  for (long long b0 = blockIdx.y; b0 < a.nb0; b0 += gridDim.y) {
    const float2* const in = static_cast<const float2*>(a.in) + b0 * a.is0 + b1_0 * a.is1;
    float2* const out = static_cast<float2*>(a.out) + b0 * a.os0 + b1_0 * a.os1;
    const float2* const mul = a.mul ? a.mul + b0 * a.os0 + b1_0 * a.os1 : nullptr;
    // rows past the last transform read the last one's values and write nothing
    auto get = [&](int i0) {
      const int i = min(i0, nb - 1);
      const long long c = 2 * (a.p0 + (a.pair_b1 ? b1_0 + i : b0));
      const int n0 = a.pair_b1 ? 0 : (int)b1_0 + i, N = (int)a.N, K = (int)a.K, isl = (int)a.isl;
      const bool has1 = c + 1 < a.ncol;
      const float2* const row = in + i * a.is1;
      const float* const ra = static_cast<const float*>(a.in) + c * a.ldi;
      const float* const rb = has1 ? ra + a.ldi : ra;
      const float2* const sa = static_cast<const float2*>(a.in) + c * a.ldi;
      const float2* const sb = has1 ? sa + a.ldi : sa;
      return [=](int l) -> float2 {
        if (IN == kInComplex) return row[l * (long long)isl];
        const int n = n0 + l * isl;
        if (IN == kInRealPair) {
          const float x = __ldg(ra + n), y = __ldg(rb + n);
          return make_float2(x, has1 ? y : 0.f);
        }
        // S_a + i S_b of bin n, from the conjugates of bin N - n above K; the imaginary parts
        // of bin 0 and, for even N, bin N/2 do not enter
        const bool upper = n >= K;
        const int k = upper ? N - n : n;
        const float2 u = __ldg(sa + k), w = __ldg(sb + k);
        const bool real = k == 0 || 2 * k == N;
        const float uy = real ? 0.f : (upper ? -u.y : u.y);
        const float wy = real || !has1 ? 0.f : (upper ? -w.y : w.y);
        return make_float2(u.x - wy, uy + (has1 ? w.x : 0.f));
      };
    };
    auto put = [&](int i) {
      const bool live = i < nb;
      const long long c = 2 * (a.p0 + (a.pair_b1 ? b1_0 + i : b0));
      const int n0 = a.pair_b1 ? 0 : (int)b1_0 + i, osl = (int)a.osl;
      const bool has1 = live && c + 1 < a.ncol;
      float2* const row = out + i * a.os1;
      const float2* const mrow = mul ? mul + i * a.os1 : nullptr;
      float* const ra = static_cast<float*>(a.out) + c * a.ldo;
      const float scale = a.scale;
      const float4* const hi = sm4 + a.tw.hi + i * a.tw.nh;
      const float2* const lo = sm + a.tw.lo + (i << a.tw.lg) + i;
      const int lg = a.tw.lg;
      return [=](int l, float2 v) {
        if (OUT == kOutRealPair) {
          v = cscale(v, scale);
          if (live) ra[n0 + l * osl] = v.x;
          if (has1) ra[n0 + l * osl + a.ldo] = v.y;
          return;
        }
        if (OUT == kOutTwiddle) {
          v = cmul(v, twiddle_at(hi, lo, lg, l));
        } else {
          if (mrow && live) v = cmul(v, __ldg(mrow + l * (long long)osl));
          v = cscale(v, scale);
        }
        if (live) row[l * (long long)osl] = v;
      };
    };
    stages_run<SIGN>(d, a.in_lane_i, a.out_lane_i, sm, get, put);
    if (b0 + gridDim.y < a.nb0) __syncthreads();  // the last stage has read shared memory
  }
}

template <int SIGN, int IN, int OUT>
int launch_stages(StageArgs& a, cudaStream_t s) {
  if (a.nb0 <= 0 || a.nb1 <= 0) return FDR_OK;
  FDR_TRY(get_roots(a.d.L, &a.d.roots));
  static bool attr_set[64] = {false};
  int dev = 0;
  FDR_CUDA(cudaGetDevice(&dev));
  if (dev >= 64 || !attr_set[dev]) {
    FDR_CUDA(cudaFuncSetAttribute(fft_stage_kernel<SIGN, IN, OUT>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageSmem));
    if (dev < 64) attr_set[dev] = true;
  }
  a.tw = twiddle_tables(a.d);
  const size_t smem = stage_smem_bytes(a.d) + (OUT == kOutTwiddle ? tw_bytes(a.d.L, a.d.bpc) : 0);
  const dim3 grid((unsigned)cdiv(a.nb1, a.d.bpc), (unsigned)std::min(a.nb0, 65535LL));
  fft_stage_kernel<SIGN, IN, OUT><<<grid, stage_threads(a.d), smem, s>>>(a);
  FDR_LAUNCH_CHECK("fft_stage_kernel");
  return FDR_OK;
}

StageArgs blank_stages() {
  StageArgs a;
  memset(&a, 0, sizeof(a));
  a.nb0 = 1;
  a.scale = 1.f;
  return a;
}

}  // namespace

int fft_strided_inplace(float2* buf, long long L, long long sl, long long nb, long long sb,
                        int sign, float scale, const float2* mul, cudaStream_t s) {
  if (L > kMaxCtaElems) {
    set_error(FDR_ERR_UNSUPPORTED_SIZE, "strided FFT length %lld exceeds %d", L, kMaxCtaElems);
    return FDR_ERR_UNSUPPORTED_SIZE;
  }
  StageArgs a = blank_stages();
  if (stage_plan(L, nb, 1, true, false, &a.d)) {
    a.in = a.out = buf;
    a.mul = mul;
    a.nb1 = nb;
    a.is1 = a.os1 = sb;
    a.isl = a.osl = sl;
    a.in_lane_i = a.out_lane_i = 1;
    a.scale = scale;
    return sign < 0 ? launch_stages<-1, kInComplex, kOutComplex>(a, s)
                    : launch_stages<+1, kInComplex, kOutComplex>(a, s);
  }
  PassDesc d = blank_pass();
  d.in = buf; d.out = buf; d.mul = mul;
  d.L = (int)L;
  d.nb0 = 1; d.nb1 = nb;
  d.is1 = sb; d.isl = sl; d.os1 = sb; d.osl = sl; d.ms1 = sb; d.msl = sl;
  d.sign = sign; d.scale = scale;
  d.bpc = pick_bpc(L, nb);
  d.ld_b1_fast = d.st_b1_fast = (sb == 1) ? 1 : 0;
  return launch_pass(d, s);
}

static void split_len(long long N, long long* L1, long long* L2) {
  // N = L1 * L2 with both <= kMaxCtaElems, L2 (the contiguous inner length) near sqrt(N).
  long long best1 = 0, best2 = 0;
  for (long long a = 2; a <= kMaxCtaElems; ++a) {
    if (N % a) continue;
    long long b = N / a;
    if (b > kMaxCtaElems) continue;
    if (best1 == 0 || llabs(a - b) < llabs(best1 - best2)) { best1 = a; best2 = b; }
  }
  *L1 = best1;
  *L2 = best2;
}

int fft_contig(const float2* in, long long ldin, float2* out, long long ldout, long long N,
               long long ncol, int sign, float scale, float2* tmp, cudaStream_t s) {
  if (N <= kMaxCtaElems) {
    PassDesc d = blank_pass();
    d.in = in; d.out = out;
    d.L = (int)N;
    d.nb0 = 1; d.nb1 = ncol;
    d.is1 = ldin; d.isl = 1; d.os1 = ldout; d.osl = 1;
    d.sign = sign; d.scale = scale;
    d.bpc = pick_bpc(N, ncol);
    d.ld_b1_fast = d.st_b1_fast = 0;
    return launch_pass(d, s);
  }
  long long L1, L2;
  split_len(N, &L1, &L2);
  if (L1 == 0) {
    set_error(FDR_ERR_UNSUPPORTED_SIZE, "FFT length %lld cannot be split into two factors <= %d",
              N, kMaxCtaElems);
    return FDR_ERR_UNSUPPORTED_SIZE;
  }
  FDR_CHECK_ARG(tmp != nullptr, "four-step FFT needs scratch");
  // Pass 1: n = n2 + L2*n1; DFT over n1 (stride L2) for each n2; twiddle exp(sign*2pi i k1 n2/N)
  PassDesc d = blank_pass();
  d.in = in; d.out = tmp;
  d.L = (int)L1;
  d.nb0 = ncol; d.nb1 = L2;
  d.is0 = ldin; d.is1 = 1; d.isl = L2;
  d.os0 = N; d.os1 = 1; d.osl = L2;
  d.sign = sign; d.scale = 1.f;
  d.tw_n = N; d.tw_dim = 1;
  d.bpc = pick_bpc(L1, L2);
  d.ld_b1_fast = d.st_b1_fast = 1;
  FDR_TRY(launch_pass(d, s));
  // Pass 2: for each k1, DFT over n2 (contiguous) -> out[k1 + L1*k2]
  PassDesc e = blank_pass();
  e.in = tmp; e.out = out;
  e.L = (int)L2;
  e.nb0 = ncol; e.nb1 = L1;
  e.is0 = N; e.is1 = L2; e.isl = 1;
  e.os0 = ldout; e.os1 = 1; e.osl = L1;
  e.sign = sign; e.scale = scale;
  e.bpc = pick_bpc(L2, L1);
  e.ld_b1_fast = 0; e.st_b1_fast = 1;
  return launch_pass(e, s);
}

long long real_fft_scratch_per_pair(long long N) {
  return N <= kMaxCtaElems ? N : 2 * N;
}

// z[p][n] = in[n, 2p] + i*in[n, 2p+1]
__global__ void pack_real_pairs(const float* __restrict__ in, long long ldin, long long ncol,
                                long long N, long long p0, long long np, float2* __restrict__ z) {
  const long long total = N * np;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long p = e / N, n = e - p * N;
    const long long c0 = 2 * (p0 + p), c1 = c0 + 1;
    float a = in[n + c0 * ldin];
    float b = c1 < ncol ? in[n + c1 * ldin] : 0.f;
    z[e] = make_float2(a, b);
  }
}

// F[k, 2p] = (Z[k] + conj Z[-k]) / 2, F[k, 2p+1] = (Z[k] - conj Z[-k]) / (2i)
__global__ void unpack_r2c(const float2* __restrict__ Z, long long N, long long K, long long ncol,
                           long long p0, long long np, float2* __restrict__ F, long long ldF) {
  const long long total = K * np;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long p = e / K, k = e - p * K;
    const float2* z = Z + p * N;
    float2 a = z[k];
    float2 b = cconj(z[k == 0 ? 0 : N - k]);
    const long long c0 = 2 * (p0 + p), c1 = c0 + 1;
    F[k + c0 * ldF] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
    if (c1 < ncol) {
      // (a - b) / (2i) = -i (a - b) / 2
      float2 d = csub(a, b);
      F[k + c1 * ldF] = make_float2(0.5f * d.y, -0.5f * d.x);
    }
  }
}

// C[p][k] = S_a[k] + i S_b[k] for k <= N/2, conj(S_a[N-k]) + i conj(S_b[N-k]) above.
__global__ void pack_c2r(const float2* __restrict__ S, long long ldS, long long ncol, long long N,
                         long long K, long long p0, long long np, float2* __restrict__ C) {
  const long long total = N * np;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long p = e / N, k = e - p * N;
    const long long c0 = 2 * (p0 + p), c1 = c0 + 1;
    const bool upper = k >= K;
    const long long kk = upper ? N - k : k;
    float2 a = S[kk + c0 * ldS];
    float2 b = c1 < ncol ? S[kk + c1 * ldS] : make_float2(0.f, 0.f);
    const bool real_bin = (kk == 0) || ((N % 2 == 0) && kk == N / 2);
    if (real_bin) { a.y = 0.f; b.y = 0.f; }
    if (upper) { a = cconj(a); b = cconj(b); }
    C[e] = make_float2(a.x - b.y, a.y + b.x);  // a + i b
  }
}

__global__ void unpack_c2r(const float2* __restrict__ z, long long N, long long ncol, long long p0,
                           long long np, float* __restrict__ out, long long ldout) {
  const long long total = N * np;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long p = e / N, n = e - p * N;
    const long long c0 = 2 * (p0 + p), c1 = c0 + 1;
    float2 v = z[e];
    out[n + c0 * ldout] = v.x;
    if (c1 < ncol) out[n + c1 * ldout] = v.y;
  }
}

static unsigned grid_for(long long total) {
  long long b = cdiv(total, 256);
  long long cap = (long long)sm_count() * 32;
  return (unsigned)max(1LL, min(b, cap));
}

// The two passes of a real transform of `np` column pairs starting at pair p0 whose packing
// and unpacking happen in the passes' own loads and stores (rfft: real columns -> the packed
// spectra Z in `z`, tmp in between; irfft: half spectra -> real columns, tmp in between).
// *done is false when a factor of N has a prime above 13: the caller takes the generic passes.
static int real_stages(bool forward, const void* in, long long ldin, void* out, long long ldout,
                       long long N, long long ncol, long long p0, long long np, float2* tmp,
                       cudaStream_t s, bool* done) {
  *done = false;
  StageArgs a = blank_stages();
  a.in = in;
  a.N = N;
  a.K = N / 2 + 1;
  a.p0 = p0;
  a.ncol = ncol;
  a.ldi = ldin;
  a.ldo = ldout;
  if (N <= kMaxCtaElems) {
    if (!stage_plan(N, np, 1, false, false, &a.d)) return FDR_OK;
    a.nb1 = np;
    a.isl = a.osl = 1;
    a.pair_b1 = 1;
    a.out = out;
    *done = true;
    if (forward) {
      a.os1 = N;
      return launch_stages<-1, kInRealPair, kOutComplex>(a, s);
    }
    a.scale = 1.f / (float)N;
    return launch_stages<+1, kInHalfPair, kOutRealPair>(a, s);
  }
  long long L1, L2;
  split_len(N, &L1, &L2);
  StageArgs b = a;
  if (L1 == 0 || !stage_plan(L1, L2, np, true, true, &a.d) || !stage_plan(L2, L1, np, true, false, &b.d))
    return FDR_OK;
  *done = true;
  // Pass 1: n = n2 + L2*n1, DFT over n1 for each n2, twiddle, tmp[k1*L2 + n2]
  a.out = tmp;
  a.nb0 = np;
  a.nb1 = L2;
  a.is1 = 1;
  a.isl = L2;
  a.os0 = N;
  a.os1 = 1;
  a.osl = L2;
  a.in_lane_i = a.out_lane_i = 1;
  FDR_TRY((forward ? launch_stages<-1, kInRealPair, kOutTwiddle>(a, s)
                   : launch_stages<+1, kInHalfPair, kOutTwiddle>(a, s)));
  // Pass 2: for each k1, DFT over n2 (contiguous), bin or channel k1 + L1*k2
  b.in = tmp;
  b.out = out;
  b.nb0 = np;
  b.nb1 = L1;
  b.is0 = N;
  b.is1 = L2;
  b.isl = 1;
  b.os0 = N;
  b.os1 = 1;
  b.osl = L1;
  b.out_lane_i = 1;
  if (forward) return launch_stages<-1, kInComplex, kOutComplex>(b, s);
  b.scale = 1.f / (float)N;
  return launch_stages<+1, kInComplex, kOutRealPair>(b, s);
}

int rfft_columns(const float* in, long long ldin, long long ncol, long long N, float2* F,
                 long long ldF, float2* scratch, long long pairs_per_chunk, cudaStream_t s) {
  const long long K = N / 2 + 1;
  const long long npairs = cdiv(ncol, 2);
  const long long per = real_fft_scratch_per_pair(N);
  for (long long p0 = 0; p0 < npairs; p0 += pairs_per_chunk) {
    const long long np = min(pairs_per_chunk, npairs - p0);
    // packed pairs in z; the four-step's first pass runs in place on z, the second
    // writes zo
    float2* z = scratch;
    float2* zo = (N <= kMaxCtaElems) ? scratch : scratch + N * np;
    float2* tmp = z;
    (void)per;
    bool done;
    FDR_TRY(real_stages(true, in, ldin, zo, N, N, ncol, p0, np, tmp, s, &done));
    if (!done) {
      pack_real_pairs<<<grid_for(N * np), 256, 0, s>>>(in, ldin, ncol, N, p0, np, z);
      FDR_LAUNCH_CHECK("pack_real_pairs");
      FDR_TRY(fft_contig(z, N, zo, N, N, np, -1, 1.f, tmp, s));
    }
    unpack_r2c<<<grid_for(K * np), 256, 0, s>>>(zo, N, K, ncol, p0, np, F, ldF);
    FDR_LAUNCH_CHECK("unpack_r2c");
  }
  return FDR_OK;
}

int irfft_columns(const float2* S, long long ldS, long long ncol, long long N, float* out,
                  long long ldout, float2* scratch, long long pairs_per_chunk, cudaStream_t s) {
  const long long K = N / 2 + 1;
  const long long npairs = cdiv(ncol, 2);
  for (long long p0 = 0; p0 < npairs; p0 += pairs_per_chunk) {
    const long long np = min(pairs_per_chunk, npairs - p0);
    float2* c = scratch;
    float2* co = (N <= kMaxCtaElems) ? scratch : scratch + N * np;
    float2* tmp = c;
    bool done;
    FDR_TRY(real_stages(false, S, ldS, out, ldout, N, ncol, p0, np, tmp, s, &done));
    if (done) continue;
    pack_c2r<<<grid_for(N * np), 256, 0, s>>>(S, ldS, ncol, N, K, p0, np, c);
    FDR_LAUNCH_CHECK("pack_c2r");
    FDR_TRY(fft_contig(c, N, co, N, N, np, +1, 1.f / (float)N, tmp, s));
    unpack_c2r<<<grid_for(N * np), 256, 0, s>>>(co, N, ncol, p0, np, out, ldout);
    FDR_LAUNCH_CHECK("unpack_c2r");
  }
  return FDR_OK;
}

}  // namespace fdr
