// Learned drift-rate window proposal: a small 1-D convolutional network that reads the
// 256-channel-summed power of a coarse channel (nbins x Nt) and predicts which of `nwin`
// drift-rate windows hold proto-hits, so that zdtfdr! runs only over those windows
// (rate batches through the r0 iterator, zdtfdr.jl:354).  The reference has no learned
// component; this is the training/serving extension of its batched-rate search
// (batchrates.jl:22-60).
//
// Network (all convolutions along the bin axis, zero padded to keep the length):
//   x [B][Nt][X] -> conv(Nt->C, K) ReLU -> conv(C->C, K) ReLU -> conv(C->C, K) ReLU
//                -> conv(C->nwin, 1) -> max over bins -> logits [B][nwin]
// Loss: mean binary cross-entropy with logits.  Optimiser: Adam on float32 master weights;
// the forward pass uses their float16 rounding ("FP16 weights").  Every reduction runs in a
// fixed order (per-block partial sums, then an ordered sum), so results are deterministic
// and a resumed training run matches an uninterrupted one bit for bit.
#include <cuda_fp16.h>
#include <limits.h>
#include <math.h>
#include <string.h>

#include "fdr_internal.cuh"

namespace fdr {

constexpr int kConvTile = 256;  // bins per CTA

struct Layer {
  int cin, cout, k;
  int64_t woff, boff;  // offsets (floats) into the parameter vector
};

}  // namespace fdr

struct fdr_propose_net {
  int nbins, nt, width, ksize, nwin;
  fdr::Layer L[4];
  int64_t nparams = 0;
  float* params = nullptr;   // float32 master weights (w then b per layer)
  __half* wh = nullptr;      // float16 copy used by both passes
  float* wt = nullptr;       // its values, each layer as [input channel][tap][output channel]
  float* m = nullptr;        // Adam moments
  float* v = nullptr;
  float* grad = nullptr;
  int64_t step = 0;
  uint64_t seed = 0;
  // for backward (allocated for max batch)
  int maxb = 0;
  float* act[3] = {nullptr, nullptr, nullptr};  // outputs of layers 1..3
  float* tile_max = nullptr;                    // per (sample, tile, window): largest logit,
  int* tile_arg = nullptr;                      //   its bin
  int* odd = nullptr;                           // taps that meet a non-finite input, see conv_fwd_kernel
  int* argmax = nullptr;
  float* dlogit = nullptr;                      // gradient of the loss wrt the logits
  float* gact = nullptr;                        // per sample: SparseGrad
  float* partial = nullptr;                     // per sample: gradient of every parameter
  float* loss = nullptr;                                  // device scalar
};

namespace fdr {

// --------------------------------------------------------------------------------------
// Network input, one pass over the spectrogram.  For bin b (channels n = b*factor + i,
// i < factor) and x = s - 1 (zero mean for an exponential(1) background):
//   power[t][b] = sum_i x[n, t] / sqrt(factor)
//   lag[l + ML][b] = sum_i sum_{t < Nt-1} x[n, t] * x[(n + l) mod Nf, t+1] / sqrt(factor*(Nt-1))
// each optionally compressed to sign(v)*log1p(|v|).  One CTA of 256 threads per bin; the
// bin's channels plus a halo of ML either side are staged in shared memory for `chunk`+1
// steps at a time (all loads of a chunk in flight together); every block reduction runs in
// a fixed order.
// --------------------------------------------------------------------------------------
constexpr int kFeatThreads = 256;
constexpr int kFeatMaxNt = 64;

__device__ __forceinline__ float compress_value(float v, int compress) {
  return compress ? copysignf(log1pf(fabsf(v)), v) : v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <int ML>
__global__ void __launch_bounds__(kFeatThreads)
proposal_input_kernel(const float* __restrict__ spec, long long Nf, int Nt, int factor, int nbins,
                      int chunk, float pscale, float lscale, int compress,
                      float* __restrict__ pow_out, float* __restrict__ lag_out) {
  constexpr int NL = 2 * ML + 1;
  constexpr int NW = kFeatThreads / 32;
  extern __shared__ float tile[];  // (chunk + 1) rows of W floats
  __shared__ float red_p[kFeatMaxNt][NW];
  __shared__ float red_l[NL][NW];
  const int W = factor + 2 * ML;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bin = blockIdx.x;
  const long long n0 = (long long)bin * factor;
  float lacc[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) lacc[l] = 0.f;
  for (int t0 = 0; t0 < Nt; t0 += chunk) {
    const int tc = min(chunk, Nt - t0);       // steps summed in this chunk
    const int rows = min(tc + 1, Nt - t0);    // plus the next step for the lag products
    __syncthreads();                          // the tile is free
    for (int r = 0; r < rows; ++r) {
      const float* col = spec + (long long)(t0 + r) * Nf;
      for (int i = tid; i < W; i += kFeatThreads) {
        long long n = n0 - ML + i;
        n = n < 0 ? n + Nf : (n >= Nf ? n - Nf : n);
        tile[r * W + i] = __ldg(col + n) - 1.f;
      }
    }
    __syncthreads();
    for (int r = 0; r < tc; ++r) {
      const float* xr = tile + r * W + ML;
      if (pow_out) {
        float ps = 0.f;
        for (int i = tid; i < factor; i += kFeatThreads) ps += xr[i];
        ps = warp_sum(ps);
        if (lane == 0) red_p[t0 + r][warp] = ps;
      }
      if (lag_out && r + 1 < rows) {
        const float* xn = tile + (r + 1) * W;  // channel n0 - ML + i of step t+1
        for (int i = tid; i < factor; i += kFeatThreads) {
          const float a = xr[i];
#pragma unroll
          for (int l = 0; l < NL; ++l) lacc[l] = fmaf(a, xn[i + l], lacc[l]);
        }
      }
    }
  }
  if (lag_out) {
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const float v = warp_sum(lacc[l]);
      if (lane == 0) red_l[l][warp] = v;
    }
  }
  __syncthreads();
  if (pow_out && tid < Nt) {
    float v = 0.f;
    for (int w = 0; w < NW; ++w) v += red_p[tid][w];
    pow_out[(long long)tid * nbins + bin] = compress_value(v * pscale, compress);
  }
  if (lag_out && tid < NL) {
    float v = 0.f;
    for (int w = 0; w < NW; ++w) v += red_l[tid][w];
    lag_out[(long long)tid * nbins + bin] = compress_value(v * lscale, compress);
  }
}

static int launch_input(const float* spec, int64_t Nf, int64_t Nt, int factor, int maxlag,
                        int compress, float* pow_out, float* lag_out, cudaStream_t s,
                        const char* who) {
  FDR_CHECK_ARG(spec != nullptr && (pow_out || lag_out), "%s: NULL argument", who);
  FDR_CHECK_ARG(maxlag == 8, "%s: this build supports maxlag 8", who);
  FDR_CHECK_ARG(factor >= 1 && factor <= 4096 && Nf % factor == 0 && Nf >= 2 * maxlag + 1 &&
                Nf / factor <= 0x7fffffff,
                "%s: Nf must be a multiple of factor (<= 4096) and >= %d", who, 2 * maxlag + 1);
  FDR_CHECK_ARG(Nt >= 1 && Nt <= kFeatMaxNt && (lag_out == nullptr || Nt >= 2),
                "%s: Nt must be in [1, %d] (>= 2 for lag products)", who, kFeatMaxNt);
  const int nbins = (int)(Nf / factor);
  const int W = factor + 2 * maxlag;
  const int chunk = std::max(1, std::min(16, (int)((48 * 1024 / sizeof(float)) / W) - 1));
  const size_t sm = sizeof(float) * (size_t)(chunk + 1) * W;
  const float pscale = 1.f / sqrtf((float)factor);
  const float lscale = Nt >= 2 ? 1.f / sqrtf((float)factor * (float)(Nt - 1)) : 0.f;
  proposal_input_kernel<8><<<nbins, kFeatThreads, sm, s>>>(spec, Nf, (int)Nt, factor, nbins, chunk,
                                                           pscale, lscale, compress, pow_out, lag_out);
  FDR_LAUNCH_CHECK("proposal_input_kernel");
  return FDR_OK;
}

// --------------------------------------------------------------------------------------
// Convolution forward: y[b][co][x] = b[co] + sum_{ci,k} w[co][ci][k] * in[b][ci][x+k-pad], ReLU.
// grid (X/kConvTile, B), kConvTile / 2 threads: a thread takes two bins and all 32 output
// channels, two channels per packed multiply-add, so that a 16-byte broadcast load of weights
// feeds four of them (one scalar weight load per multiply-add bound the scalar form: 190 us a
// layer at 64 x 4096 bins, 33 channels; now 83 us, FMA pipe 57%, the weights' loads behind it).
// Every output sums over (ci, k) in order from its bias.
// HEAD: the last hidden layer also forms the 16 window logits of its bins (the 1x1 layer, same
// order of sums) and their maximum over the tile's bins, the first bin on ties.
// odd: per (sample, tile, input channel) the taps that meet an infinity or NaN (bit k), for HEAD
// also per (sample, tile) the output channels that hold an infinity: the gradient's sums over all
// bins multiply these by zeros, which the sparse kernels below leave out, so that they turn the
// sums that these would meet into NaN.
// --------------------------------------------------------------------------------------
constexpr int kWidth = 32, kWin = 16, kTaps = 5, kPad = kTaps / 2;
constexpr int kConvThreads = kConvTile / 2;

template <bool HEAD>
__global__ void __launch_bounds__(kConvThreads, 4)
conv_fwd_kernel(const float* __restrict__ in, int cin, int X, const float* __restrict__ wt,
                const float* __restrict__ bias, float* __restrict__ out, const float* __restrict__ wt3,
                const float* __restrict__ bias3, float* __restrict__ tile_max, int* __restrict__ tile_arg,
                int* __restrict__ odd, int* __restrict__ odd_head) {
  extern __shared__ float4 sm4[];
  constexpr int TW = kConvTile + kTaps - 1;
  float* const wsm = reinterpret_cast<float*>(sm4);  // [ci][k][co]
  float* const w3sm = wsm + cin * kTaps * kWidth;     // HEAD: [ci][window]
  float* const xs = w3sm + (HEAD ? kWidth * kWin : 0);  // [ci][TW]
  const int b = blockIdx.y, x0 = blockIdx.x * kConvTile, tid = threadIdx.x;
  const float* const inb = in + (long long)b * cin * X;
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll 2
  for (int ci = warp; ci < cin; ci += kConvThreads / 32) {  // a warp per row: loads in flight together
    const float* const row = inb + (long long)ci * X;
    bool any = false;
#pragma unroll
    for (int j = 0; j < (TW + 31) / 32; ++j) {
      const int i = lane + 32 * j, xx = x0 - kPad + i;
      if (i < TW) {
        const float v = (xx >= 0 && xx < X) ? __ldg(row + xx) : 0.f;
        xs[ci * TW + i] = v;
        any |= !(fabsf(v) < INFINITY);
      }
    }
    int taps = 0;
    if (__any_sync(0xffffffffu, any)) {
      for (int i = lane; i < TW; i += 32)
        if (!(fabsf(xs[ci * TW + i]) < INFINITY))
          for (int k = 0; k < kTaps; ++k)
            if (i >= k && i - k < kConvTile) taps |= 1 << k;  // tap k takes it to bin i - k of the tile
      taps = __reduce_or_sync(0xffffffffu, taps);
    }
    if (lane == 0) odd[((long long)b * gridDim.x + blockIdx.x) * cin + ci] = taps;
  }
#pragma unroll 4
  for (int i = tid; i < cin * kTaps * kWidth; i += kConvThreads) wsm[i] = __ldg(wt + i);
  if (HEAD)
    for (int i = tid; i < kWidth * kWin; i += kConvThreads) w3sm[i] = __ldg(wt3 + i);
  __syncthreads();
  float2 acc[2][kWidth / 2];
#pragma unroll
  for (int p = 0; p < kWidth / 2; ++p) acc[0][p] = acc[1][p] = make_float2(bias[2 * p], bias[2 * p + 1]);
  for (int ci = 0; ci < cin; ++ci) {
    const float* const xr = xs + ci * TW + tid;
#pragma unroll
    for (int k = 0; k < kTaps; ++k) {
      const float v0 = xr[k], v1 = xr[kConvThreads + k];
      const float2 a0 = make_float2(v0, v0), a1 = make_float2(v1, v1);
      const float4* const wr = sm4 + (ci * kTaps + k) * (kWidth / 4);
#pragma unroll
      for (int q = 0; q < kWidth / 4; ++q) {
        const float4 wv = wr[q];
        acc[0][2 * q] = __ffma2_rn(make_float2(wv.x, wv.y), a0, acc[0][2 * q]);
        acc[0][2 * q + 1] = __ffma2_rn(make_float2(wv.z, wv.w), a0, acc[0][2 * q + 1]);
        acc[1][2 * q] = __ffma2_rn(make_float2(wv.x, wv.y), a1, acc[1][2 * q]);
        acc[1][2 * q + 1] = __ffma2_rn(make_float2(wv.z, wv.w), a1, acc[1][2 * q + 1]);
      }
    }
  }
  float* const ob = out + (long long)b * kWidth * X;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int x = x0 + tid + h * kConvThreads;
#pragma unroll
    for (int p = 0; p < kWidth / 2; ++p) {
      acc[h][p] = make_float2(fmaxf(acc[h][p].x, 0.f), fmaxf(acc[h][p].y, 0.f));
      if (x < X) {
        ob[(long long)(2 * p) * X + x] = acc[h][p].x;
        ob[(long long)(2 * p + 1) * X + x] = acc[h][p].y;
      }
    }
  }
  if constexpr (!HEAD) return;
  __shared__ int inf_channels[kConvThreads / 32];
  {
    float top = 0.f;
#pragma unroll
    for (int p = 0; p < kWidth / 2; ++p)
      top = fmaxf(top, fmaxf(fmaxf(acc[0][p].x, acc[0][p].y), fmaxf(acc[1][p].x, acc[1][p].y)));
    int m = 0;
    if (__any_sync(0xffffffffu, top == INFINITY)) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < kWidth / 2; ++p)
          if (x0 + tid + h * kConvThreads < X)
            m |= ((acc[h][p].x == INFINITY) << (2 * p)) | ((int)((unsigned)(acc[h][p].y == INFINITY) << (2 * p + 1)));
      m = __reduce_or_sync(0xffffffffu, m);
    }
    if (lane == 0) inf_channels[warp] = m;
  }
  __shared__ float rv[kConvThreads / 32][kWin];
  __shared__ int ri[kConvThreads / 32][kWin];
#pragma unroll
  for (int half = 0; half < 2; ++half) {  // 8 windows at a time
    float best[kWin / 2];
    int at[kWin / 2];
#pragma unroll
    for (int j = 0; j < kWin / 2; ++j) {
      best[j] = -INFINITY;
      at[j] = 0;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 z[kWin / 4];
#pragma unroll
      for (int p = 0; p < kWin / 4; ++p)
        z[p] = make_float2(bias3[8 * half + 2 * p], bias3[8 * half + 2 * p + 1]);
#pragma unroll
      for (int ci = 0; ci < kWidth; ++ci) {
        const float v = ci & 1 ? acc[h][ci / 2].y : acc[h][ci / 2].x;
        const float2 vv = make_float2(v, v);
        const float4* const wr = reinterpret_cast<const float4*>(w3sm + ci * kWin + 8 * half);
        const float4 wa = wr[0], wb = wr[1];
        z[0] = __ffma2_rn(make_float2(wa.x, wa.y), vv, z[0]);
        z[1] = __ffma2_rn(make_float2(wa.z, wa.w), vv, z[1]);
        z[2] = __ffma2_rn(make_float2(wb.x, wb.y), vv, z[2]);
        z[3] = __ffma2_rn(make_float2(wb.z, wb.w), vv, z[3]);
      }
      const int x = x0 + tid + h * kConvThreads;
#pragma unroll
      for (int j = 0; j < kWin / 2; ++j) {
        const float v = j & 1 ? z[j / 2].y : z[j / 2].x;
        if (x < X && v > best[j]) {
          best[j] = v;
          at[j] = x;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kWin / 2; ++j) {
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_down_sync(0xffffffffu, best[j], o);
        const int oi = __shfl_down_sync(0xffffffffu, at[j], o);
        if (ov > best[j] || (ov == best[j] && oi < at[j])) {
          best[j] = ov;
          at[j] = oi;
        }
      }
      if (lane == 0) {
        rv[warp][8 * half + j] = best[j];
        ri[warp][8 * half + j] = at[j];
      }
    }
  }
  __syncthreads();
  if (tid < kWin) {
    float v = rv[0][tid];
    int i = ri[0][tid];
    for (int q = 1; q < kConvThreads / 32; ++q)
      if (rv[q][tid] > v || (rv[q][tid] == v && ri[q][tid] < i)) {
        v = rv[q][tid];
        i = ri[q][tid];
      }
    const long long o = ((long long)b * gridDim.x + blockIdx.x) * kWin + tid;
    tile_max[o] = v;
    tile_arg[o] = i;
    if (tid == 0) {
      int m = 0;
      for (int q = 0; q < kConvThreads / 32; ++q) m |= inf_channels[q];
      odd_head[(long long)b * gridDim.x + blockIdx.x] = m;
    }
  }
}

// logits[b][w] = the largest logit over the tiles (first bin on ties), argmax its bin.
__global__ void maxpool_kernel(const float* __restrict__ tile_max, const int* __restrict__ tile_arg, int tiles, int n,
                               float* __restrict__ logits, int* __restrict__ argmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long at = (long long)(i / kWin) * tiles * kWin + i % kWin;
  float v = tile_max[at];
  int bi = tile_arg[at];
  for (int t = 1; t < tiles; ++t) {
    const float tv = tile_max[at + (long long)t * kWin];
    const int ti = tile_arg[at + (long long)t * kWin];
    if (tv > v || (tv == v && ti < bi)) {
      v = tv;
      bi = ti;
    }
  }
  logits[i] = v;
  argmax[i] = bi;
}

// Mean BCE with logits (single block, fixed order) and its gradient wrt the logits.
__global__ void bce_kernel(const float* __restrict__ logits, const float* __restrict__ labels, int n,
                           float* __restrict__ dlogit, float* __restrict__ loss) {
  __shared__ float part[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float z = logits[i], y = labels[i];
    s += fmaxf(z, 0.f) - z * y + log1pf(expf(-fabsf(z)));
    const float p = 1.f / (1.f + expf(-z));
    dlogit[i] = (p - y) / (float)n;
  }
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < blockDim.x; ++i) t += part[i];
    *loss = t / (float)n;
  }
}

// --------------------------------------------------------------------------------------
// Backward.  The maximum over bins passes a window's gradient to one bin, so at most 16 bins of
// a sample's last hidden layer have one, 5 bins around each of them in the layer below and 9 in
// the first: 16, 80 and 144 of the (4096) bins.  Everything else is zero and is not touched (the
// dense form multiplied it out: 3.4 of a training step's 4.1 ms).  The bins of a layer are listed
// in ascending order, those around the selected ones merged; bins outside [0, X) stay in the list
// with zero gradient so that five neighbouring bins are neighbours in the list below.
// --------------------------------------------------------------------------------------
constexpr int kMaxBins = kWin * 9;       // listed bins of the first layer
constexpr int kMaxInBins = kWin * 13;    // and of its input

struct SparseGrad {                 // of one sample
  int n[3];                         // listed bins of layers 1, 2, 3 (index 0, 1, 2)
  int bins[3][kMaxBins];
  float g[3][kMaxBins * kWidth];    // [bin][channel], masked by the layer's ReLU
};

// The selected bins of a sample, sorted and distinct, and lists of the bins around them.
struct BinSet {
  int sel[kWin], n;
  int start[kWin + 1];
  // by all threads of the block, from the 16 bins in `raw` (shared memory, visible)
  __device__ __forceinline__ void sort(const int* raw) {
    const int t = threadIdx.x;
    if (t < kWin) {
      int rank = 0, distinct = 0;
      bool repeat = false;
      for (int w = 0; w < kWin; ++w) {
        bool seen = false;  // raw[w] occurs before w
        for (int v = 0; v < w; ++v) seen |= raw[v] == raw[w];
        repeat |= w < t && raw[w] == raw[t];
        if (!seen) {
          ++distinct;
          rank += raw[w] < raw[t];
        }
      }
      if (!repeat) sel[rank] = raw[t];
      if (t == 0) n = distinct;
    }
    __syncthreads();
  }
  // the bins within `radius` of a selected one, ascending, without repeats; their number
  __device__ __forceinline__ int list(int radius, int* out) {
    const int t = threadIdx.x, w = 2 * radius + 1;
    if (t <= kWin) {
      int s = 0;
      for (int i = 0; i < n && i < t; ++i) s += i == 0 ? w : min(w, sel[i] - sel[i - 1]);
      start[t] = s;
    }
    __syncthreads();
    const int i = t / 16, j = t % 16;  // w <= 13
    const int total = start[n];        // before the barrier: the next call overwrites start after it
    if (i < n && j < start[i + 1] - start[i]) out[start[i] + j] = sel[i] + radius + 1 - (start[i + 1] - start[i]) + j;
    __syncthreads();
    return total;
  }
};
// Index in the ascending list of bin x, or `none` if it is not there.
__device__ __forceinline__ int find_bin(const int* list, int n, int x, int none) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (list[mid] < x) lo = mid + 1; else hi = mid;
  }
  return list[lo] == x ? lo : none;
}

// Gradients of a sample's hidden layers at the listed bins.  grid B, kSparseThreads threads.
// At 64 samples: 43 us (56 with the lists built by one thread), one CTA on 64 of the SMs, bound by
// the chain of three layers and its barriers; with the kernel below it replaced 3.4 ms of dense
// backward kernels.
constexpr int kSparseThreads = 512;

__global__ void __launch_bounds__(kSparseThreads)
sparse_grad_kernel(const float* __restrict__ dlogit, const int* __restrict__ argmax,
                   const float* __restrict__ act0, const float* __restrict__ act1, const float* __restrict__ act2,
                   int X, const float* __restrict__ wt1, const float* __restrict__ wt2, const __half* __restrict__ w3,
                   SparseGrad* __restrict__ out) {
  extern __shared__ float4 sm4[];
  float* const wsm = reinterpret_cast<float*>(sm4);          // [k][co][ci] of a 32 x 32 layer
  float* const ga = wsm + kTaps * kWidth * kWidth;           // [bin][channel]; a row of zeros after the last
  float* const gb = ga + (kMaxBins + 1) * kWidth;
  __shared__ BinSet set;
  __shared__ int raw[kWin], bins[3][kMaxBins], slot[kMaxBins][kTaps];
  const int b = blockIdx.x, tid = threadIdx.x;
  SparseGrad& o = out[b];
  if (tid < kWin) raw[tid] = argmax[b * kWin + tid];
  __syncthreads();
  set.sort(raw);
  int nb[3];
  for (int l = 0; l < 3; ++l) {
    nb[l] = set.list(4 - 2 * l, bins[l]);
    if (tid == 0) o.n[l] = nb[l];
    if (tid < nb[l]) o.bins[l][tid] = bins[l][tid];
  }
  // last hidden layer: the 1x1 layer's weights of the windows whose bin this is, in window order
  for (int i = tid; i < nb[2] * kWidth; i += kSparseThreads) {
    const int x = bins[2][i / kWidth], c = i % kWidth;
    const float relu = act2[((long long)b * kWidth + c) * X + x];
    float g = 0.f;
    for (int w = 0; w < kWin; ++w)
      if (raw[w] == x) g = fmaf(__half2float(w3[w * kWidth + c]), dlogit[b * kWin + w], g);
    if (relu <= 0.f) g = 0.f;
    ga[i] = g;
    o.g[2][i] = g;
  }
  float* from = ga;
  float* to = gb;
  for (int l = 1; l >= 0; --l) {  // layer l + 1 from the layer above it
    const float* const w = l == 1 ? wt2 : wt1;  // [ci][k][co]
    const float* const act = l == 1 ? act1 : act0;
    for (int i = tid; i < kTaps * kWidth * kWidth; i += kSparseThreads) {
      const int co = i / (kWidth * kTaps), r = i - co * kWidth * kTaps, k = r / kWidth, ci = r - k * kWidth;
      wsm[(k * kWidth + co) * kWidth + ci] = __ldg(w + (ci * kTaps + k) * kWidth + co);
    }
    for (int i = tid; i < nb[l] * kTaps; i += kSparseThreads) {
      const int s = i / kTaps, k = i - s * kTaps;
      slot[s][k] = find_bin(bins[l + 1], nb[l + 1], bins[l][s] + kPad - k, nb[l + 1]);
    }
    if (tid < kWidth) from[nb[l + 1] * kWidth + tid] = 0.f;
    __syncthreads();
    // d_in[x] = sum over k, co of w[co][ci][k] g[x + pad - k]: a thread takes channel ci of four
    // bins, so that its four weights feed 16 multiply-adds
    const int ci = tid % kWidth;
    for (int s0 = 4 * (tid / kWidth); s0 < nb[l]; s0 += 4 * (kSparseThreads / kWidth)) {
      float g[4] = {0.f, 0.f, 0.f, 0.f}, relu[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int x = bins[l][min(s0 + q, nb[l] - 1)];
        relu[q] = x >= 0 && x < X ? act[((long long)b * kWidth + ci) * X + x] : 0.f;
      }
      for (int k = 0; k < kTaps; ++k) {
        const float4* gr[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          gr[q] = reinterpret_cast<const float4*>(from + slot[min(s0 + q, nb[l] - 1)][k] * kWidth);
        const float* const wr = wsm + k * kWidth * kWidth + ci;
#pragma unroll
        for (int c4 = 0; c4 < kWidth / 4; ++c4) {
          const float w0 = wr[(4 * c4) * kWidth], w1 = wr[(4 * c4 + 1) * kWidth], w2 = wr[(4 * c4 + 2) * kWidth],
                      w3v = wr[(4 * c4 + 3) * kWidth];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 v = gr[q][c4];
            g[q] = fmaf(w3v, v.w, fmaf(w2, v.z, fmaf(w1, v.y, fmaf(w0, v.x, g[q]))));
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (s0 + q < nb[l]) {
          if (relu[q] <= 0.f) g[q] = 0.f;
          to[(s0 + q) * kWidth + ci] = g[q];
          o.g[l][(s0 + q) * kWidth + ci] = g[q];
        }
    }
    __syncthreads();
    float* const t = from;
    from = to;
    to = t;
  }
}

// Flags of conv_fwd_kernel for the inputs of the four layers.
struct OddInputs {
  const int* at[4];
  int tiles;
};

// A sample's gradient of one layer's parameters: grid (4 layers, B).  Layers 1 to 3: a thread
// takes four output channels, an input channel and the five taps; the layer's input at the listed
// bins and two either side sits in shared memory in list order.  Layer 4 (1x1): its selected bins.
// At 64 samples: 40 us (55 with serial lists), bound by the latency of the gathered loads.
__global__ void __launch_bounds__(kSparseThreads)
sparse_weight_grad_kernel(const SparseGrad* __restrict__ sg, const float* __restrict__ x0,
                          const float* __restrict__ act0, const float* __restrict__ act1,
                          const float* __restrict__ act2, const float* __restrict__ dlogit,
                          const int* __restrict__ argmax, int cin0, int X, Layer L0, Layer L1, Layer L2, Layer L3,
                          float* __restrict__ partial, long long nparams, OddInputs odd) {
  extern __shared__ float4 sm4[];
  const int l = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  float* const pb = partial + b * nparams;
  if (l == 3) {
    int inf = 0;
    for (int t = 0; t < odd.tiles; ++t) inf |= odd.at[3][(long long)b * odd.tiles + t];
    for (int i = tid; i < kWin * kWidth; i += kSparseThreads) {
      const int w = i / kWidth, c = i % kWidth;
      const float v = dlogit[b * kWin + w] * act2[((long long)b * kWidth + c) * X + argmax[b * kWin + w]];
      pb[L3.woff + i] = (inf >> c & 1) && fabsf(v) < INFINITY ? NAN : v;
    }
    for (int w = tid; w < kWin; w += kSparseThreads) pb[L3.boff + w] = dlogit[b * kWin + w];
    return;
  }
  const Layer& L = l == 0 ? L0 : l == 1 ? L1 : L2;
  const int cin = l == 0 ? cin0 : kWidth;
  const float* const in = (l == 0 ? x0 : l == 1 ? act0 : act1) + (long long)b * cin * X;
  const SparseGrad& s = sg[b];
  const int n = s.n[l];
  float* const gsm = reinterpret_cast<float*>(sm4);          // [bin][channel]
  float* const xsm = gsm + kMaxBins * kWidth;             // [ci][kMaxInBins]: bins within two of the list
  __shared__ BinSet set;
  __shared__ int raw[kWin], first[kMaxBins], ext[kMaxInBins];
  if (tid < kWin) raw[tid] = argmax[b * kWin + tid];
  for (int i = tid; i < n * kWidth; i += kSparseThreads) gsm[i] = s.g[l][i];
  __syncthreads();
  set.sort(raw);
  const int ne = set.list(6 - 2 * l, ext);  // the input's bins: two either side of the layer's
  for (int i = tid; i < n; i += kSparseThreads) first[i] = find_bin(ext, ne, s.bins[l][i] - kPad, 0);
  for (int i = tid; i < cin * ne; i += kSparseThreads) {
    const int ci = i / ne, e = i - ci * ne, x = ext[e];
    xsm[ci * kMaxInBins + e] = (x >= 0 && x < X) ? in[(long long)ci * X + x] : 0.f;
  }
  __syncthreads();
  for (int u = tid; u < (kWidth / 4) * cin; u += kSparseThreads) {
    const int cg = u % (kWidth / 4), ci = u / (kWidth / 4);
    const float* const xr = xsm + ci * kMaxInBins;
    float a[4][kTaps];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int k = 0; k < kTaps; ++k) a[q][k] = 0.f;
    for (int i = 0; i < n; ++i) {
      const float4 g = sm4[i * (kWidth / 4) + cg];
      const float* const xe = xr + first[i];
#pragma unroll
      for (int k = 0; k < kTaps; ++k) {
        const float v = xe[k];
        a[0][k] = fmaf(g.x, v, a[0][k]);
        a[1][k] = fmaf(g.y, v, a[1][k]);
        a[2][k] = fmaf(g.z, v, a[2][k]);
        a[3][k] = fmaf(g.w, v, a[3][k]);
      }
    }
    int taps = 0;
    for (int t = 0; t < odd.tiles; ++t) taps |= __ldg(odd.at[l] + ((long long)b * odd.tiles + t) * cin + ci);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int k = 0; k < kTaps; ++k)
        pb[L.woff + ((long long)(4 * cg + q) * cin + ci) * kTaps + k] =
            (taps >> k & 1) && fabsf(a[q][k]) < INFINITY ? NAN : a[q][k];
  }
  for (int c = tid; c < kWidth; c += kSparseThreads) {
    float a = 0.f;
    for (int i = 0; i < n; ++i) a += gsm[i * kWidth + c];
    pb[L.boff + c] = a;
  }
}

// grad[i] = sum over samples (in order) of partial[b][i]
__global__ void reduce_partials_kernel(const float* __restrict__ partial, int B, long long n,
                                       float* __restrict__ grad) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < B; ++k) s += partial[k * n + i];
  grad[i] = s;
}

// Where weight i of the layers goes in their [ci][k][co] order (biases keep their place).
struct LayerOrder {
  Layer L[4];
};
__device__ __forceinline__ long long transposed_place(const LayerOrder& o, long long i) {
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const Layer& L = o.L[l];
    if (i >= L.woff && i < L.boff) {
      const int r = (int)(i - L.woff), per = L.cin * L.k;
      return L.woff + (long long)(r % per) * L.cout + r / per;
    }
  }
  return i;
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, __half* __restrict__ wh, float* __restrict__ wt, LayerOrder order,
                            long long n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  const __half h = __float2half_rn(pi);
  wh[i] = h;
  wt[transposed_place(order, i)] = __half2float(h);
}

__global__ void to_half_kernel(const float* __restrict__ p, __half* __restrict__ wh, float* __restrict__ wt,
                               LayerOrder order, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const __half h = __float2half_rn(p[i]);
  wh[i] = h;
  wt[transposed_place(order, i)] = __half2float(h);
}

// ---- host helpers ---------------------------------------------------------------------
static LayerOrder layer_order(const fdr_propose_net* n) {
  LayerOrder o;
  for (int i = 0; i < 4; ++i) o.L[i] = n->L[i];
  return o;
}

static uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

static int set_attrs() {
  static bool done[64] = {false};
  int dev = 0;
  FDR_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && done[dev]) return FDR_OK;
  const int big = 160 * 1024;  // conv layers with up to 64 input channels need <= 110 KB
  FDR_CUDA(cudaFuncSetAttribute(conv_fwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  FDR_CUDA(cudaFuncSetAttribute(conv_fwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  FDR_CUDA(cudaFuncSetAttribute(sparse_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  FDR_CUDA(cudaFuncSetAttribute(sparse_weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  if (dev < 64) done[dev] = true;
  return FDR_OK;
}

static OddInputs odd_inputs(const fdr_propose_net* n) {
  OddInputs o;
  o.tiles = (int)cdiv(n->nbins, kConvTile);
  const int cin[3] = {n->nt, kWidth, kWidth};
  const int* p = n->odd;
  for (int l = 0; l < 3; ++l) {
    o.at[l] = p;
    p += (size_t)n->maxb * o.tiles * cin[l];
  }
  o.at[3] = p;
  return o;
}

static int net_forward(fdr_propose_net* n, const float* x, int B, float* logits, cudaStream_t s) {
  FDR_CHECK_ARG(B >= 1 && B <= n->maxb, "proposal net: batch %d exceeds the maximum %d", B, n->maxb);
  const float* in = x;
  const int X = n->nbins, tiles = (int)cdiv(X, kConvTile);
  const dim3 grid((unsigned)tiles, (unsigned)B);
  const OddInputs odd = odd_inputs(n);
  for (int li = 0; li < 3; ++li) {
    const Layer& L = n->L[li];
    const size_t sm = sizeof(float) * (L.cin * (kConvTile + kTaps - 1) + kWidth * L.cin * kTaps +
                                       (li == 2 ? kWidth * kWin : 0));
    auto kernel = li == 2 ? conv_fwd_kernel<true> : conv_fwd_kernel<false>;
    kernel<<<grid, kConvThreads, sm, s>>>(in, L.cin, X, n->wt + L.woff, n->params + L.boff, n->act[li],
                                          n->wt + n->L[3].woff, n->params + n->L[3].boff, n->tile_max, n->tile_arg,
                                          const_cast<int*>(odd.at[li]), const_cast<int*>(odd.at[3]));
    FDR_LAUNCH_CHECK("conv_fwd_kernel");
    in = n->act[li];
  }
  maxpool_kernel<<<(unsigned)cdiv(B * n->nwin, 64), 64, 0, s>>>(n->tile_max, n->tile_arg, tiles, B * n->nwin, logits,
                                                               n->argmax);
  FDR_LAUNCH_CHECK("maxpool_kernel");
  return FDR_OK;
}

// Forward + loss + backward into n->grad.  logits: device [B][nwin] scratch.
static int net_grad(fdr_propose_net* n, const float* x, const float* labels, int B, float* logits,
                    cudaStream_t s) {
  FDR_TRY(net_forward(n, x, B, logits, s));
  const int X = n->nbins;
  bce_kernel<<<1, 256, 0, s>>>(logits, labels, B * n->nwin, n->dlogit, n->loss);
  FDR_LAUNCH_CHECK("bce_kernel");
  SparseGrad* const sg = reinterpret_cast<SparseGrad*>(n->gact);
  const size_t sm1 = sizeof(float) * (kTaps * kWidth * kWidth + 2 * (kMaxBins + 1) * kWidth);
  sparse_grad_kernel<<<B, kSparseThreads, sm1, s>>>(n->dlogit, n->argmax, n->act[0], n->act[1], n->act[2], X,
                                                    n->wt + n->L[1].woff, n->wt + n->L[2].woff,
                                                    n->wh + n->L[3].woff, sg);
  FDR_LAUNCH_CHECK("sparse_grad_kernel");
  const size_t sm2 = sizeof(float) * (kMaxBins * kWidth + std::max(n->nt, kWidth) * kMaxInBins);
  sparse_weight_grad_kernel<<<dim3(4, B), kSparseThreads, sm2, s>>>(
      sg, x, n->act[0], n->act[1], n->act[2], n->dlogit, n->argmax, n->nt, X, n->L[0], n->L[1], n->L[2], n->L[3],
      n->partial, n->nparams, odd_inputs(n));
  FDR_LAUNCH_CHECK("sparse_weight_grad_kernel");
  reduce_partials_kernel<<<(unsigned)cdiv(n->nparams, 128), 128, 0, s>>>(n->partial, B, n->nparams, n->grad);
  FDR_LAUNCH_CHECK("reduce_partials_kernel");
  return FDR_OK;
}

static void net_release(fdr_propose_net* n) {
  if (!n) return;
  cudaFree(n->params);
  cudaFree(n->wh);
  cudaFree(n->wt);
  cudaFree(n->m);
  cudaFree(n->v);
  cudaFree(n->grad);
  for (auto* a : n->act) cudaFree(a);
  cudaFree(n->tile_max);
  cudaFree(n->tile_arg);
  cudaFree(n->odd);
  cudaFree(n->argmax);
  cudaFree(n->dlogit);
  cudaFree(n->gact);
  cudaFree(n->partial);
  cudaFree(n->loss);
  delete n;
}

}  // namespace fdr

using namespace fdr;

extern "C" {

int fdr_propose_create(fdr_propose_net** out, int nbins, int nt, int width, int ksize, int nwin,
                       int max_batch, uint64_t seed) {
  FDR_CHECK_ARG(out != nullptr, "fdr_propose_create: NULL handle");
  FDR_CHECK_ARG(nbins >= 1 && nt >= 1 && nt <= 64 && nwin >= 1 && max_batch >= 1,
                "fdr_propose_create: bad sizes");
  FDR_CHECK_ARG(width == 32 && ksize == 5 && nwin == 16,
                "fdr_propose_create: this build supports width 32, kernel 5, 16 windows");
  *out = nullptr;
  FDR_TRY(set_attrs());
  fdr_propose_net* n = new fdr_propose_net();
  n->nbins = nbins; n->nt = nt; n->width = width; n->ksize = ksize; n->nwin = nwin;
  n->maxb = max_batch;
  n->seed = seed;
  const int cins[4] = {nt, width, width, width}, couts[4] = {width, width, width, nwin};
  const int ks[4] = {ksize, ksize, ksize, 1};
  int64_t off = 0;
  for (int i = 0; i < 4; ++i) {
    n->L[i] = {cins[i], couts[i], ks[i], off, off + (int64_t)couts[i] * cins[i] * ks[i]};
    off = n->L[i].boff + couts[i];
  }
  n->nparams = off;
  // He-uniform initialisation from a seeded splitmix64 stream; zero biases.
  std::vector<float> h((size_t)off, 0.f);
  uint64_t st = seed;
  for (int i = 0; i < 4; ++i) {
    const float bound = sqrtf(6.f / (float)(n->L[i].cin * n->L[i].k));
    for (int64_t j = 0; j < (int64_t)n->L[i].cout * n->L[i].cin * n->L[i].k; ++j) {
      const double u = (double)(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
      h[(size_t)(n->L[i].woff + j)] = (float)((2.0 * u - 1.0) * bound);
    }
  }
  const size_t act_elems = (size_t)max_batch * width * nbins;
  const size_t tile_elems = (size_t)cdiv(nbins, kConvTile) * max_batch * nwin;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMalloc(&n->params, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->wh, sizeof(__half) * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->wt, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->m, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->v, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->grad, sizeof(float) * off);
  for (int i = 0; i < 3 && e == cudaSuccess; ++i) e = cudaMalloc(&n->act[i], sizeof(float) * act_elems);
  if (e == cudaSuccess) e = cudaMalloc(&n->tile_max, sizeof(float) * tile_elems);
  if (e == cudaSuccess) e = cudaMalloc(&n->tile_arg, sizeof(int) * tile_elems);
  if (e == cudaSuccess)
    e = cudaMalloc(&n->odd, sizeof(int) * tile_elems / kWin * ((size_t)n->nt + 2 * kWidth + 1));
  if (e == cudaSuccess) e = cudaMalloc(&n->dlogit, sizeof(float) * (size_t)max_batch * nwin);
  if (e == cudaSuccess) e = cudaMalloc(&n->gact, sizeof(SparseGrad) * (size_t)max_batch);
  if (e == cudaSuccess) e = cudaMalloc(&n->argmax, sizeof(int) * (size_t)max_batch * nwin);
  if (e == cudaSuccess) e = cudaMalloc(&n->partial, sizeof(float) * (size_t)max_batch * off);
  if (e == cudaSuccess) e = cudaMalloc(&n->loss, sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(n->params, h.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(n->m, 0, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMemset(n->v, 0, sizeof(float) * off);
  if (e != cudaSuccess) {
    int st2 = cuda_status(e, "fdr_propose_create");
    net_release(n);
    return st2;
  }
  to_half_kernel<<<(unsigned)cdiv(off, 256), 256>>>(n->params, n->wh, n->wt, layer_order(n), off);
  e = cudaDeviceSynchronize();
  if (e != cudaSuccess) { int st2 = cuda_status(e, "fdr_propose_create"); net_release(n); return st2; }
  count_launch();
  *out = n;
  return FDR_OK;
}

int fdr_propose_destroy(fdr_propose_net* n) {
  if (n) { cudaDeviceSynchronize(); net_release(n); }
  return FDR_OK;
}

int fdr_propose_num_params(const fdr_propose_net* n, int64_t* count) {
  FDR_CHECK_ARG(n && count, "NULL argument");
  *count = n->nparams;
  return FDR_OK;
}

int fdr_propose_features(const float* spec, int64_t Nf, int64_t Nt, int factor, int compress,
                         float* out, fdr_stream_t stream) {
  return launch_input(spec, Nf, Nt, factor, 8, compress, out, nullptr, (cudaStream_t)stream,
                      "fdr_propose_features");
}

int fdr_propose_lag_features(const float* spec, int64_t Nf, int64_t Nt, int factor, int maxlag,
                             int compress, float* out, fdr_stream_t stream) {
  return launch_input(spec, Nf, Nt, factor, maxlag, compress, nullptr, out, (cudaStream_t)stream,
                      "fdr_propose_lag_features");
}

int fdr_propose_input(const float* spec, int64_t Nf, int64_t Nt, int factor, int maxlag,
                      int compress, float* out, fdr_stream_t stream) {
  FDR_CHECK_ARG(out != nullptr, "fdr_propose_input: NULL argument");
  return launch_input(spec, Nf, Nt, factor, maxlag, compress, out,
                      out + Nt * (Nf / std::max(factor, 1)), (cudaStream_t)stream, "fdr_propose_input");
}

int fdr_propose_forward(fdr_propose_net* n, const float* x, int batch, float* logits,
                        fdr_stream_t stream) {
  FDR_CHECK_ARG(n && x && logits, "fdr_propose_forward: NULL argument");
  return net_forward(n, x, batch, logits, (cudaStream_t)stream);
}

int fdr_propose_gradients(fdr_propose_net* n, const float* x, const float* labels, int batch,
                          float* logits, float* grad_out, float* loss_out, fdr_stream_t stream) {
  FDR_CHECK_ARG(n && x && labels && logits, "fdr_propose_gradients: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  FDR_TRY(net_grad(n, x, labels, batch, logits, s));
  if (grad_out) FDR_CUDA(cudaMemcpyAsync(grad_out, n->grad, sizeof(float) * n->nparams, cudaMemcpyDeviceToDevice, s));
  if (loss_out) FDR_CUDA(cudaMemcpyAsync(loss_out, n->loss, sizeof(float), cudaMemcpyDeviceToDevice, s));
  return FDR_OK;
}

int fdr_propose_train_step(fdr_propose_net* n, const float* x, const float* labels, int batch,
                           float lr, float* logits, float* loss_out, fdr_stream_t stream) {
  FDR_CHECK_ARG(n && x && labels && logits, "fdr_propose_train_step: NULL argument");
  cudaStream_t s = (cudaStream_t)stream;
  FDR_TRY(net_grad(n, x, labels, batch, logits, s));
  n->step += 1;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - powf(b1, (float)n->step), c2 = 1.f - powf(b2, (float)n->step);
  adam_kernel<<<(unsigned)cdiv(n->nparams, 256), 256, 0, s>>>(n->params, n->grad, n->m, n->v, n->wh, n->wt,
                                                               layer_order(n), n->nparams, lr, b1, b2, eps, c1, c2);
  FDR_LAUNCH_CHECK("adam_kernel");
  if (loss_out) FDR_CUDA(cudaMemcpyAsync(loss_out, n->loss, sizeof(float), cudaMemcpyDeviceToDevice, s));
  return FDR_OK;
}

// Checkpoint state: params, m, v (host float arrays of num_params) and the step count.
int fdr_propose_get_state(fdr_propose_net* n, float* params, float* m, float* v, int64_t* step) {
  FDR_CHECK_ARG(n != nullptr, "NULL net");
  FDR_CUDA(cudaDeviceSynchronize());
  if (params) FDR_CUDA(cudaMemcpy(params, n->params, sizeof(float) * n->nparams, cudaMemcpyDeviceToHost));
  if (m) FDR_CUDA(cudaMemcpy(m, n->m, sizeof(float) * n->nparams, cudaMemcpyDeviceToHost));
  if (v) FDR_CUDA(cudaMemcpy(v, n->v, sizeof(float) * n->nparams, cudaMemcpyDeviceToHost));
  if (step) *step = n->step;
  return FDR_OK;
}

int fdr_propose_set_state(fdr_propose_net* n, const float* params, const float* m, const float* v,
                          int64_t step) {
  FDR_CHECK_ARG(n && params, "NULL argument");
  FDR_CUDA(cudaDeviceSynchronize());
  FDR_CUDA(cudaMemcpy(n->params, params, sizeof(float) * n->nparams, cudaMemcpyHostToDevice));
  if (m) FDR_CUDA(cudaMemcpy(n->m, m, sizeof(float) * n->nparams, cudaMemcpyHostToDevice));
  if (v) FDR_CUDA(cudaMemcpy(n->v, v, sizeof(float) * n->nparams, cudaMemcpyHostToDevice));
  n->step = step;
  to_half_kernel<<<(unsigned)cdiv(n->nparams, 256), 256>>>(n->params, n->wh, n->wt, layer_order(n), n->nparams);
  FDR_LAUNCH_CHECK("to_half_kernel");
  FDR_CUDA(cudaDeviceSynchronize());
  return FDR_OK;
}

}  // extern "C"
