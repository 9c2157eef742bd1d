// Convolution and pooling kernels (NCHW): im2col / col2im for the GEMM-lowered convolution, direct
// fp32 convolution forward / input gradient / weight gradient / bias gradient (groups supported, so
// depthwise convolutions run here too), transposed convolution through the same kernels, max pooling
// with saved arg-max positions and average pooling, each with a deterministic backward.
//
// The reference has a one-thread-per-output max-pool and direct-convolution forward on the device
// (legacy/src/momijo/tensor/gpu/runtime.mojo:122-200) and host loops for the rest; its max-pool
// backward adds `gy` at the arg-max with a plain `+=`, which races when windows overlap
// (legacy/src/momijo/learn/nn/conv.mojo:342-405). Every backward here is written in gather form:
// one thread owns one gradient element and sums the contributions that reach it in a fixed order,
// so there are no atomics and results are bitwise reproducible.
#include "common.cuh"

namespace mmj {

struct ConvGeom {
  int N, C, H, W;        // input
  int OC, kH, kW;        // filters
  int OH, OW;            // output
  int sh, sw, ph, pw, dh, dw;
  int groups;
};

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// ---- im2col: cols[(n, oh, ow), c * kH * kW + kh * kW + kw], row pitch ldc >= C*kH*kW (pad columns = 0) ----
// Small matrices (up to 131072 elements), an element to a thread: 49 x 72 bf16 in 1.5 us, where the kernel below has a
// chain of gathers and stores (2.9 with 16 columns to a warp, 5.1 with 64).
template <typename T>
__global__ void __launch_bounds__(256) im2col_small_kernel(const T* __restrict__ x, T* __restrict__ cols, ConvGeom g, int ldc) {
  const int i = blockIdx.x * 256 + threadIdx.x, r = i / ldc, k = i - r * ldc;
  if (r >= g.N * g.OH * g.OW) return;
  T v = from_f<T>(0.f);
  if (k < g.C * g.kH * g.kW) {
    const int t = k / g.kW, kw = k - t * g.kW, c = t / g.kH, kh = t - c * g.kH;
    const int q = r / g.OW, ow = r - q * g.OW, n = q / g.OH, oh = q - n * g.OH;
    const int h = oh * g.sh - g.ph + kh * g.dh, w = ow * g.sw - g.pw + kw * g.dw;
    if (h >= 0 && h < g.H && w >= 0 && w < g.W) v = x[(((long long)n * g.C + c) * g.H + h) * g.W + w];
  }
  cols[i] = v;
}

// A warp owns 32 output positions and KT columns: it gathers with the positions along its lanes (contiguous in the image
// rows, one tap for the whole warp, stepped without divisions), turns the tile through shared memory and stores rows of
// KT columns. One element per thread, consecutive threads along a row of cols, took two 64-bit divisions each and
// gathered 32 sectors with every load: 504 us for 100352 x 576 bf16, 82 now with 64 columns. Smaller matrices have too few
// warps of 64 columns, whose gathers follow one another: 3136 x 144 in 7.0 us with an element per thread, 5.4 with 64
// columns to a warp, 3.6 with 16; 25088 x 64 17.5 / 6.5 / 5.4.
template <typename T, int KT>
__global__ void __launch_bounds__(128) im2col_kernel(const T* __restrict__ x, T* __restrict__ cols, ConvGeom g,
                                                     long long ldc, int vec) {
  constexpr int V = 16 / sizeof(T);             // elements per 16-byte store
  constexpr int kPitch = KT + V;                // rows stay 16-byte aligned
  __shared__ __align__(16) T tile[4][32 * kPitch];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* st = tile[warp];
  const long long rows = (long long)g.N * g.OH * g.OW;
  const int K = g.C * g.kH * g.kW;
  const int k_tiles = (int)((ldc + KT - 1) / KT);
  const long long units = (rows + 31) / 32 * k_tiles;
  for (long long u = blockIdx.x * 4LL + warp; u < units; u += gridDim.x * 4LL) {
    const long long r0 = u / k_tiles * 32;
    const int k0 = (int)(u % k_tiles) * KT;
    const long long r = r0 + lane;
    int h0 = -(1 << 29), w0 = 0;                // a position past the end reads nothing
    const T* xp = x;
    if (r < rows) {
      const int ow = (int)(r % g.OW);
      const long long q = r / g.OW;
      const int oh = (int)(q % g.OH);
      h0 = oh * g.sh - g.ph;
      w0 = ow * g.sw - g.pw;
      xp = x + (q / g.OH) * g.C * g.H * g.W + (long long)h0 * g.W + w0;
    }
    int c = k0 / (g.kH * g.kW), t = k0 - c * g.kH * g.kW;
    int kh = t / g.kW, kw = t - kh * g.kW;
#pragma unroll 8
    for (int j = 0; j < KT; ++j) {
      const int dh = kh * g.dh, dw = kw * g.dw;
      T v = from_f<T>(0.f);
      if (k0 + j < K && (unsigned)(h0 + dh) < (unsigned)g.H && (unsigned)(w0 + dw) < (unsigned)g.W)
        v = xp[(long long)c * g.H * g.W + dh * g.W + dw];
      st[lane * kPitch + j] = v;
      if (++kw == g.kW) {
        kw = 0;
        if (++kh == g.kH) { kh = 0; ++c; }
      }
    }
    __syncwarp();
    const int n = (int)(ldc - k0 < KT ? ldc - k0 : KT);
    if (vec) {
      constexpr int kLanes = KT / V;            // lanes per row
      for (int i = lane; i < 32 * kLanes; i += 32) {
        const int rr = i / kLanes, cc = (i % kLanes) * V;
        if (r0 + rr < rows && cc < n)
          *reinterpret_cast<uint4*>(cols + (r0 + rr) * ldc + k0 + cc) = *reinterpret_cast<const uint4*>(st + rr * kPitch + cc);
      }
    } else {
      for (int i = lane; i < 32 * KT; i += 32) {
        const int rr = i / KT, cc = i % KT;
        if (r0 + rr < rows && cc < n) cols[(r0 + rr) * ldc + k0 + cc] = st[rr * kPitch + cc];
      }
    }
    __syncwarp();
  }
}

// ---- col2im (gather form): dx[n, c, h, w] = sum over the window positions that read this element ----
template <typename T>
__global__ void col2im_kernel(const T* __restrict__ cols, T* __restrict__ dx, ConvGeom g, long long ldc) {
  const long long total = (long long)g.N * g.C * g.H * g.W;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(i % g.W);
    const int h = (int)((i / g.W) % g.H);
    const int c = (int)((i / ((long long)g.W * g.H)) % g.C);
    const int n = (int)(i / ((long long)g.W * g.H * g.C));
    float acc = 0.f;
    for (int kh = 0; kh < g.kH; ++kh) {
      const int hh = h + g.ph - kh * g.dh;
      if (hh < 0 || hh % g.sh) continue;
      const int oh = hh / g.sh;
      if (oh >= g.OH) continue;
      for (int kw = 0; kw < g.kW; ++kw) {
        const int ww = w + g.pw - kw * g.dw;
        if (ww < 0 || ww % g.sw) continue;
        const int ow = ww / g.sw;
        if (ow >= g.OW) continue;
        const long long r = ((long long)n * g.OH + oh) * g.OW + ow;
        acc += to_f<T>(cols[r * ldc + ((long long)c * g.kH + kh) * g.kW + kw]);
      }
    }
    dx[i] = from_f<T>(acc);
  }
}

// ---- direct convolution, fp32 accumulate; weight [OC, C/groups, kH, kW] --------------------------------
template <typename T>
__global__ void conv2d_fwd_kernel(const T* __restrict__ x, const T* __restrict__ wt, const T* __restrict__ bias,
                                  T* __restrict__ y, ConvGeom g) {
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  const long long total = (long long)g.N * g.OC * g.OH * g.OW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ow = (int)(i % g.OW);
    const int oh = (int)((i / g.OW) % g.OH);
    const int oc = (int)((i / ((long long)g.OW * g.OH)) % g.OC);
    const int n = (int)(i / ((long long)g.OW * g.OH * g.OC));
    const int c0 = (oc / ocg) * cg;
    float acc = (bias != nullptr) ? to_f<T>(bias[oc]) : 0.f;
    for (int c = 0; c < cg; ++c) {
      const T* xp = x + ((long long)n * g.C + c0 + c) * g.H * g.W;
      const T* wp = wt + ((long long)oc * cg + c) * g.kH * g.kW;
      for (int kh = 0; kh < g.kH; ++kh) {
        const int h = oh * g.sh - g.ph + kh * g.dh;
        if (h < 0 || h >= g.H) continue;
        for (int kw = 0; kw < g.kW; ++kw) {
          const int w = ow * g.sw - g.pw + kw * g.dw;
          if (w < 0 || w >= g.W) continue;
          acc = fmaf(to_f<T>(xp[(long long)h * g.W + w]), to_f<T>(wp[kh * g.kW + kw]), acc);
        }
      }
    }
    y[i] = from_f<T>(acc);
  }
}

// dx[n, c, h, w] = sum_{oc in group, kh, kw} dy[n, oc, oh, ow] * wt[oc, c - c0, kh, kw]  (gather form).
// Run on (x = input of a transposed convolution, weight [Cin, Cout/groups, kH, kW]) this is also the
// forward pass of the transposed convolution; `bias` (per output channel here = per c) is added then.
template <typename T>
__global__ void conv2d_dx_kernel(const T* __restrict__ dy, const T* __restrict__ wt, const T* __restrict__ bias,
                                 T* __restrict__ dx, ConvGeom g) {
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  const long long total = (long long)g.N * g.C * g.H * g.W;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(i % g.W);
    const int h = (int)((i / g.W) % g.H);
    const int c = (int)((i / ((long long)g.W * g.H)) % g.C);
    const int n = (int)(i / ((long long)g.W * g.H * g.C));
    const int grp = c / cg, cl = c - grp * cg;
    float acc = (bias != nullptr) ? to_f<T>(bias[c]) : 0.f;
    for (int o = 0; o < ocg; ++o) {
      const int oc = grp * ocg + o;
      const T* dyp = dy + ((long long)n * g.OC + oc) * g.OH * g.OW;
      const T* wp = wt + ((long long)oc * cg + cl) * g.kH * g.kW;
      for (int kh = 0; kh < g.kH; ++kh) {
        const int hh = h + g.ph - kh * g.dh;
        if (hh < 0 || hh % g.sh) continue;
        const int oh = hh / g.sh;
        if (oh >= g.OH) continue;
        for (int kw = 0; kw < g.kW; ++kw) {
          const int ww = w + g.pw - kw * g.dw;
          if (ww < 0 || ww % g.sw) continue;
          const int ow = ww / g.sw;
          if (ow >= g.OW) continue;
          acc = fmaf(to_f<T>(dyp[(long long)oh * g.OW + ow]), to_f<T>(wp[kh * g.kW + kw]), acc);
        }
      }
    }
    dx[i] = from_f<T>(acc);
  }
}

__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float x = (lane < 8) ? red[lane] : 0.f;
  x = warp_sum(x);
  __syncthreads();
  return x;
}

// dw[oc, cl, kh, kw] = sum_{n, oh, ow} dy[n, oc, oh, ow] * x[n, c0 + cl, h, w]: one block per weight
// element, threads stride over (n, oh, ow), fixed-order block reduction.
template <typename T>
__global__ void __launch_bounds__(256) conv2d_dw_kernel(const T* __restrict__ x, const T* __restrict__ dy,
                                                        T* __restrict__ dwt, ConvGeom g) {
  __shared__ float red[8];
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  const long long e = blockIdx.x;
  const int kw = (int)(e % g.kW);
  const int kh = (int)((e / g.kW) % g.kH);
  const int cl = (int)((e / ((long long)g.kW * g.kH)) % cg);
  const int oc = (int)(e / ((long long)g.kW * g.kH * cg));
  const int c = (oc / ocg) * cg + cl;
  const long long spatial = (long long)g.OH * g.OW;
  const long long total = (long long)g.N * spatial;
  float acc = 0.f;
  for (long long i = threadIdx.x; i < total; i += blockDim.x) {
    const int ow = (int)(i % g.OW);
    const int oh = (int)((i / g.OW) % g.OH);
    const int n = (int)(i / spatial);
    const int h = oh * g.sh - g.ph + kh * g.dh;
    const int w = ow * g.sw - g.pw + kw * g.dw;
    if (h < 0 || h >= g.H || w < 0 || w >= g.W) continue;
    acc = fmaf(to_f<T>(dy[((long long)n * g.OC + oc) * spatial + (long long)oh * g.OW + ow]),
               to_f<T>(x[(((long long)n * g.C + c) * g.H + h) * g.W + w]), acc);
  }
  acc = block_sum_256(acc, red);
  if (threadIdx.x == 0) dwt[e] = from_f<T>(acc);
}

// ---- tiled convolution: a register-blocked fp32 product whose second operand is gathered from the image ----
//
// Forward and input gradient are one kernel: out[m, p] = bias[m] + sum_k w(m, k) * src(k, p), where p runs over
// output positions and k over (channel, tap); only the affine maps of taps and positions differ. A strided input
// gradient is cut into stride x stride classes of pixels that meet the same taps (blockIdx.z), so that no product
// is spent on taps that fall between the strides.
//
// What bounds it: fp32 multiply-adds (74 TFLOP/s on 148 SMs at 1.965 GHz; bytes are 20 times below that at 64
// channels). The one-thread-per-output kernels above load two operands per multiply-add and spent their time on
// the load pipe (1.8 TFLOP/s forward, 0.7 input gradient, 0.4 weight gradient at N32 C64 56x56 OC64 k3). A 64 x 128
// tile on 128 threads keeps 8 x 8 sums per thread, so that 64 multiply-adds take four 16-byte shared-memory reads;
// they are issued as fma.rn.f32x2, which halves the issue slots and rounds like two scalar FMAs. Positions lie
// along the lanes: gathers of one tap are contiguous in the image rows. Each chunk of 16 k has its tap table
// (offset, row and column shift, weight offset) computed once per block by 16 threads, two chunks ahead.
// Measured at that shape, before -> now: forward 4121 -> 217 us (34 TFLOP/s), input gradient 10160 -> 216 us; three
// blocks per SM (168 registers, no spills) against four: 217 / 224 us.
// Taps outside the image are multiplied as zeros. An infinite weight would make a NaN of those, where the tap does not
// exist: results that come out as NaN are computed again by skip_sum, without such taps.
struct GatherGeom {
  int SH, SW;                      // image that is gathered from
  int cls_h, cls_w;                // pixel classes (strides of an input gradient; 1 x 1 in a forward pass)
  int PHf, PWf;                    // full grid of output positions; class (a, b) owns rows a, a + cls_h, ...
  int pos_s_h, pos_s_w;            // source row of position i = i * pos_s + pos_o (forward: stride, -pad)
  int pos_o_h, pos_o_w;
  int kH, kW, dh, dw, ph, pw;
  int transposed;                  // 1: input gradient
  int channels;                    // contraction channels per group
  int M, groups, N;                // output channels per group
  long long src_n, src_g;          // image / group strides of the source (elements)
  long long w_m, w_ch, w_g;        // weight strides: output channel, contraction channel, group
  long long dst_n, dst_m, dst_g;
};

// taps of one axis that a pixel class meets: t = first + i * step, i < count; source shift = e0 + i * es
struct AxisTaps {
  int first, step, count, e0, es;
};
__device__ __forceinline__ AxisTaps axis_taps(int transposed, int cls, int stride, int k, int dil, int pad) {
  AxisTaps r;
  if (!transposed) {
    r.first = 0; r.step = 1; r.count = k; r.e0 = 0; r.es = dil;
    return r;
  }
  // taps t with (cls + pad - t * dil) divisible by the stride: an arithmetic progression
  int a = stride, b = dil;
  while (b) { const int c = a % b; a = b; b = c; }
  const int step = stride / a;
  int first = -1;
  for (int t = 0; t < step && t < k; ++t)
    if ((cls + pad - t * dil) % stride == 0) { first = t; break; }
  r.first = first; r.step = step;
  r.count = first < 0 ? 0 : (k - first + step - 1) / step;
  r.e0 = first < 0 ? 0 : (cls + pad - first * dil) / stride;
  r.es = -(step * dil) / stride;
  return r;
}

constexpr int kGatherBN = 128, kGatherBK = 16, kGatherThreads = 128;

// One result of the tiled product, in its order, over the taps inside the image only; false where every tap is inside.
// `sp` points at the position's source pixel (h0, w0), `wp` at the output channel's weights.
template <typename T>
__device__ bool skip_sum(const T* sp, const T* wp, const GatherGeom& g, const AxisTaps& vh, const AxisTaps& vw, int h0,
                         int w0, float& sum) {
  bool outside = false;
  float s = 0.f;
  for (int ch = 0; ch < g.channels; ++ch)
    for (int ih = 0; ih < vh.count; ++ih)
      for (int iw = 0; iw < vw.count; ++iw) {
        const int eh = vh.e0 + ih * vh.es, ew = vw.e0 + iw * vw.es;
        if ((unsigned)(h0 + eh) >= (unsigned)g.SH || (unsigned)(w0 + ew) >= (unsigned)g.SW) {
          outside = true;
          continue;
        }
        if (ch > 0 && !outside) return false;
        s = fmaf(to_f<T>(wp[ch * (int)g.w_ch + (vh.first + ih * vh.step) * g.kW + (vw.first + iw * vw.step)]),
                 to_f<T>(sp[ch * g.SH * g.SW + eh * g.SW + ew]), s);
      }
  sum = s;
  return outside;
}
// The NaNs among one thread's results, in a function of its own so that the product's registers don't know of it.
template <typename T, int TM, int TN>
__device__ __noinline__ void skip_nan_results(const T* src, const T* wt, const T* bias, T* dst, const long long* out_off,
                                              const GatherGeom& g, long long p0, int grp, int mt, int tx, int ca, int cb) {
  const int PH = (g.PHf - ca + g.cls_h - 1) / g.cls_h, PW = (g.PWf - cb + g.cls_w - 1) / g.cls_w;
  const AxisTaps vh = axis_taps(g.transposed, ca, g.cls_h, g.kH, g.dh, g.ph);
  const AxisTaps vw = axis_taps(g.transposed, cb, g.cls_w, g.kW, g.dw, g.pw);
  for (int i = 0; i < TM * TN; ++i) {
    const int m = mt + i / TN, jj = i % TN;
    const int p = (jj >> 2) * (kGatherBN * 4 / TN) + tx * 4 + (jj & 3);
    if (m >= g.M || out_off[p] < 0) continue;
    T* o = dst + (long long)m * g.dst_m + out_off[p];
    if (to_f<T>(*o) == to_f<T>(*o)) continue;
    const long long pos = p0 + p, q = pos / PW;
    const int h = (int)(q % PH) * g.pos_s_h + g.pos_o_h, w = (int)(pos % PW) * g.pos_s_w + g.pos_o_w;
    float v;
    if (skip_sum<T>(src + q / PH * g.src_n + grp * g.src_g + (long long)h * g.SW + w, wt + grp * g.w_g + m * g.w_m, g, vh,
                    vw, h, w, v))
      *o = from_f<T>(v + ((bias != nullptr) ? to_f<T>(bias[grp * g.M + m]) : 0.f));
  }
}

template <typename T, int BM, int TM, int TN>
__global__ void __launch_bounds__(kGatherThreads, 3)
    conv_gather_kernel(const T* __restrict__ src, const T* __restrict__ wt, const T* __restrict__ bias,
                       T* __restrict__ dst, const __grid_constant__ GatherGeom g) {
  constexpr int BN = kGatherBN, BK = kGatherBK;
  constexpr int TX = BN / TN, TY = BM / TM;
  static_assert(TX * TY == kGatherThreads, "tile and thread count disagree");
  constexpr int LA = BM * BK / kGatherThreads;   // weights each thread fetches per chunk
  constexpr int ldA = BM + 4;
  __shared__ __align__(16) float As[2][BK][ldA];
  __shared__ __align__(16) float Bs[2][BK][BN];
  __shared__ int4 tab[3][BK];
  __shared__ long long out_off[BN];

  const int t = threadIdx.x, tx = t % TX, ty = t / TX;
  const int ca = (int)blockIdx.z / g.cls_w, cb = (int)blockIdx.z % g.cls_w;
  const int PH = (g.PHf - ca + g.cls_h - 1) / g.cls_h, PW = (g.PWf - cb + g.cls_w - 1) / g.cls_w;
  const long long P = (long long)g.N * PH * PW;
  const long long p0 = (long long)blockIdx.x * BN;
  if (p0 >= P) return;                           // classes differ by a row or a column
  bool nan = false;
  const int m_tiles = (g.M + BM - 1) / BM;
  const int grp = (int)blockIdx.y / m_tiles, m0 = ((int)blockIdx.y % m_tiles) * BM;
  const AxisTaps vh = axis_taps(g.transposed, ca, g.cls_h, g.kH, g.dh, g.ph);
  const AxisTaps vw = axis_taps(g.transposed, cb, g.cls_w, g.kW, g.dw, g.pw);
  const int taps = vh.count * vw.count;
  const int K = g.channels * taps;
  const int chunks = (K + BK - 1) / BK;

  // this thread's position: it fetches column t of every chunk
  int h0 = -(1 << 29), w0 = 0;                   // a position past the end meets no valid tap
  const T* sp = src;
  {
    const long long p = p0 + t;
    long long off = -1;
    if (p < P) {
      const int j = (int)(p % PW);
      const long long q = p / PW;
      const int i = (int)(q % PH);
      const long long n = q / PH;
      h0 = i * g.pos_s_h + g.pos_o_h;
      w0 = j * g.pos_s_w + g.pos_o_w;
      sp = src + n * g.src_n + grp * g.src_g + (long long)h0 * g.SW + w0;
      off = n * g.dst_n + grp * g.dst_g + (long long)(ca + i * g.cls_h) * g.PWf + (cb + j * g.cls_w);
    }
    out_off[t] = off;
  }
  const T* wp = wt + grp * g.w_g + (long long)m0 * g.w_m;

  auto make_tab = [&](int c) {
    if (t < BK) {
      const int k = c * BK + t;
      int4 e = make_int4(0, -(1 << 29), 0, -1);
      if (k < K) {
        const int ch = k / taps, r = k - ch * taps;
        const int ih = r / vw.count, iw = r - ih * vw.count;
        const int eh = vh.e0 + ih * vh.es, ew = vw.e0 + iw * vw.es;
        e.x = ch * g.SH * g.SW + eh * g.SW + ew;
        e.y = eh;
        e.z = ew;
        e.w = ch * (int)g.w_ch + (vh.first + ih * vh.step) * g.kW + (vw.first + iw * vw.step);
      }
      tab[c % 3][t] = e;
    }
  };
  // widened when they are staged: here the conversion waits for its load before the products of this chunk (bf16,
  // N4 C64 28x28, 8 filters, k11: 489 us, 334 now)
  T ra[LA], rb[BK];
  auto fetch = [&](int c) {
    const int4* tb = tab[c % 3];
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int id = t + i * kGatherThreads;
      const int kk = id % BK, m = id / BK;
      const int off = tb[kk].w;
      ra[i] = (off >= 0 && m0 + m < g.M) ? wp[(long long)m * g.w_m + off] : from_f<T>(0.f);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const int4 e = tb[kk];
      const bool ok = ((unsigned)(h0 + e.y) < (unsigned)g.SH) & ((unsigned)(w0 + e.z) < (unsigned)g.SW);
      rb[kk] = ok ? sp[e.x] : from_f<T>(0.f);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int id = t + i * kGatherThreads;
      As[buf][id % BK][id / BK] = to_f<T>(ra[i]);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) Bs[buf][kk][t] = to_f<T>(rb[kk]);
  };

  f32x2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  make_tab(0);
  make_tab(1);
  __syncthreads();
  if (chunks > 0) {
    fetch(0);
    stage(0);
  }
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    const int buf = c & 1;
    if (c + 2 < chunks) make_tab(c + 2);
    if (c + 1 < chunks) fetch(c + 1);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
      f32x2 b[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&As[buf][kk][ty * TM + i]);
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(&Bs[buf][kk][j * (BN * 4 / TN) + tx * 4]);
        b[2 * j] = f2_pack(v.x, v.y);
        b[2 * j + 1] = f2_pack(v.z, v.w);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const f32x2 aa = f2_pack(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = f2_fma(aa, b[j], acc[i][j]);
      }
    }
    if (c + 1 < chunks) stage(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= g.M) continue;
    const float bv = (bias != nullptr) ? to_f<T>(bias[grp * g.M + m]) : 0.f;
    T* o = dst + (long long)m * g.dst_m;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const int p = (j >> 1) * (BN * 4 / TN) + tx * 4 + (j & 1) * 2;
      float lo, hi;
      f2_unpack(acc[i][j], lo, hi);
      if (out_off[p] >= 0) o[out_off[p]] = from_f<T>(lo + bv);
      if (out_off[p + 1] >= 0) o[out_off[p + 1]] = from_f<T>(hi + bv);
      nan |= (lo != lo) | (hi != hi);
    }
  }
  if (nan)
    skip_nan_results<T, TM, TN>(src, wt, bias, dst, out_off, g, p0, grp, m0 + ty * TM, tx, ca, cb);
}

// Weight gradient: dw[oc, k] = sum_p dy[oc, p] * x(k, p), both operands contiguous along p. A block owns a
// BM x 64 tile of dw and one slice of the positions; slices write fp32 slabs that slab_fold_kernel adds in slice
// order, so that results stay bitwise reproducible. A thread adds at most 64 products in a row before it folds
// them into a second sum, so that chains stay as short as in the direct kernel's 256-thread block sum (error against
// 64 bits at N32 C64 56x56 OC64 k3: 3.6e-7 before, 1.9e-7 now). The direct kernel re-read both images for each of its
// blocks of one filter tap: 18393 -> 206 us at that shape, the fold of the slabs included.
constexpr int kWgBN = 64, kWgBP = 32, kWgThreads = 128, kWgFold = 2;

template <typename T, int BM>
__global__ void __launch_bounds__(kWgThreads, 4)
    conv_wgrad_kernel(const T* __restrict__ x, const T* __restrict__ dy, float* __restrict__ slabs, ConvGeom g,
                      long long slice) {
  constexpr int BN = kWgBN, BP = kWgBP, TM = BM / 8, TN = 4;
  constexpr int ldA = BM + 4, ldB = BN + 4;
  constexpr int RA = BM / 4, RB = BN / 4;        // rows each warp fetches
  __shared__ __align__(16) float As[2][BP][ldA];
  __shared__ __align__(16) float Bs[2][BP][ldB];
  __shared__ int4 tab[BN];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, tx = t & 15, ty = t >> 4;
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  const int taps = g.kH * g.kW, K = cg * taps;
  const int m_tiles = (ocg + BM - 1) / BM;
  const int grp = (int)blockIdx.y / m_tiles, m0 = ((int)blockIdx.y % m_tiles) * BM;
  const int k0 = (int)blockIdx.x * BN;
  const int spatial = g.OH * g.OW;
  const long long P = (long long)g.N * spatial;
  const long long pb = (long long)blockIdx.z * slice;
  const long long pe = pb + slice < P ? pb + slice : P;
  if (t < BN) {
    const int k = k0 + t;
    int4 e = make_int4(0, -(1 << 29), 0, 0);
    if (k < K) {
      const int ch = k / taps, r = k - ch * taps;
      const int kh = r / g.kW, kw = r - kh * g.kW;
      e = make_int4(ch * g.H * g.W + kh * g.dh * g.W + kw * g.dw, kh * g.dh, kw * g.dw, 0);
    }
    tab[t] = e;
  }
  const T* xg = x + (long long)grp * cg * g.H * g.W;
  const T* yg = dy + ((long long)grp * ocg + m0) * spatial;
  T ra[RA], rb[RB];
  auto fetch = [&](long long p) {
    p += lane;
    int h0 = -(1 << 29), w0 = 0;
    const T *sp = xg, *yp = yg;
    const bool live = p < pe;
    if (live) {
      const int n = (int)((unsigned)p / (unsigned)spatial);
      const int s = (int)p - n * spatial;
      const int oh = s / g.OW, ow = s - oh * g.OW;
      h0 = oh * g.sh - g.ph;
      w0 = ow * g.sw - g.pw;
      sp = xg + (long long)n * g.C * g.H * g.W + (long long)h0 * g.W + w0;
      yp = yg + (long long)n * g.OC * spatial + s;
    }
#pragma unroll
    for (int i = 0; i < RA; ++i) {
      const int m = warp * RA + i;
      ra[i] = (live && m0 + m < ocg) ? yp[(long long)m * spatial] : from_f<T>(0.f);
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      const int4 e = tab[warp * RB + i];
      const bool ok = ((unsigned)(h0 + e.y) < (unsigned)g.H) & ((unsigned)(w0 + e.z) < (unsigned)g.W);
      rb[i] = ok ? sp[e.x] : from_f<T>(0.f);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < RA; i += 4)
      *reinterpret_cast<float4*>(&As[buf][lane][warp * RA + i]) =
          make_float4(to_f<T>(ra[i]), to_f<T>(ra[i + 1]), to_f<T>(ra[i + 2]), to_f<T>(ra[i + 3]));
#pragma unroll
    for (int i = 0; i < RB; i += 4)
      *reinterpret_cast<float4*>(&Bs[buf][lane][warp * RB + i]) =
          make_float4(to_f<T>(rb[i]), to_f<T>(rb[i + 1]), to_f<T>(rb[i + 2]), to_f<T>(rb[i + 3]));
  };
  f32x2 acc[TM][TN / 2];
  float sum[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      sum[i][j] = 0.f;
      if (j < TN / 2) acc[i][j] = 0ull;
    }
  __syncthreads();
  const int chunks = pb < pe ? (int)((pe - pb + BP - 1) / BP) : 0;
  if (chunks > 0) {
    fetch(pb);
    stage(0);
  }
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    const int buf = c & 1;
    if (c + 1 < chunks) fetch(pb + (long long)(c + 1) * BP);
#pragma unroll 8
    for (int p = 0; p < BP; ++p) {
      float a[TM];
      if constexpr (TM >= 4) {
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(&As[buf][p][ty * TM + i]);
          a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
        }
      } else {
        const float2 v = *reinterpret_cast<const float2*>(&As[buf][p][ty * TM]);
        a[0] = v.x; a[1] = v.y;
      }
      const float4 v = *reinterpret_cast<const float4*>(&Bs[buf][p][tx * 4]);
      const f32x2 b0 = f2_pack(v.x, v.y), b1 = f2_pack(v.z, v.w);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const f32x2 aa = f2_pack(a[i], a[i]);
        acc[i][0] = f2_fma(aa, b0, acc[i][0]);
        acc[i][1] = f2_fma(aa, b1, acc[i][1]);
      }
    }
    if (c + 1 < chunks) stage(buf ^ 1);
    if ((c + 1) % kWgFold == 0 || c + 1 == chunks) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          float lo, hi;
          f2_unpack(acc[i][j], lo, hi);
          sum[i][2 * j] += lo;
          sum[i][2 * j + 1] += hi;
          acc[i][j] = 0ull;
        }
    }
    __syncthreads();
  }
  float* out = slabs + (long long)blockIdx.z * g.OC * K + (long long)(grp * ocg) * K;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= ocg) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int k = k0 + tx * 4 + j;
      if (k < K) out[(long long)m * K + k] = sum[i][j];
    }
  }
}

// The tiles multiply pixels outside the image as zeros, which an infinite dy turns into NaN where the tap does not exist:
// a NaN sum again without such pixels, in chains of 64 and slices as well. i: (filter, channel, tap).
template <typename T>
__device__ __noinline__ void wgrad_skip_sum(const T* x, const T* dy, T* dst, const ConvGeom& g, long long i,
                                            long long slice) {
  const int cg = g.C / g.groups, taps = g.kH * g.kW, K = cg * taps, spatial = g.OH * g.OW;
  const int oc = (int)(i / K), k = (int)(i - (long long)oc * K), ch = k / taps, t = k - ch * taps;
  const int eh = t / g.kW * g.dh - g.ph, ew = t % g.kW * g.dw - g.pw;
  if (eh >= 0 && (g.OH - 1) * g.sh + eh < g.H && ew >= 0 && (g.OW - 1) * g.sw + ew < g.W) return;   // never outside
  const T* xc = x + (long long)(oc / (g.OC / g.groups) * cg + ch) * g.H * g.W;
  float all = 0.f, total = 0.f, part = 0.f;
  const long long P = (long long)g.N * spatial;
  for (long long p = 0; p < P; ++p) {
    const int n = (int)(p / spatial), s = (int)(p - (long long)n * spatial);
    const int h = s / g.OW * g.sh + eh, w = s % g.OW * g.sw + ew;
    if ((unsigned)h < (unsigned)g.H && (unsigned)w < (unsigned)g.W)
      part = fmaf(to_f<T>(dy[((long long)n * g.OC + oc) * spatial + s]),
                  to_f<T>(xc[(long long)n * g.C * g.H * g.W + (long long)h * g.W + w]), part);
    if ((p & 63) == 63) {
      total += part;
      part = 0.f;
    }
    if ((p + 1) % slice == 0) {
      all += total + part;
      total = part = 0.f;
    }
  }
  dst[i] = from_f<T>(all + total + part);
}

// dst[i] = sum over S slabs: 8 lanes of slabs per element group, folded in a fixed order. kConv: slabs of a weight
// gradient over slices of `slice` positions; its NaNs are looked at last, in 32 registers, so that they cost the fold
// neither registers nor blocks (a call among its loads took 1 x 4096 channels, 1000 filters from 150 to 359 us).
template <typename T, bool kConv>
__global__ void __launch_bounds__(256, 8) slab_fold_kernel(const float* __restrict__ slabs, T* __restrict__ dst,
                                                           long long n, int S, const T* __restrict__ x,
                                                           const T* __restrict__ dy, const __grid_constant__ ConvGeom g,
                                                           long long slice) {
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * 32 + lane;
  float a = 0.f;
  if (i < n)
    for (int s = row; s < S; s += 8) a += slabs[(long long)s * n + i];
  part[row][lane] = a;
  __syncthreads();
  if (row != 0 || i >= n) return;
#pragma unroll
  for (int r = 1; r < 8; ++r) a += part[r][lane];
  dst[i] = from_f<T>(a);
  if (kConv && a != a) wgrad_skip_sum<T>(x, dy, dst, g, i, slice);
}

// db[oc] = sum_{n, oh, ow} dy[n, oc, oh, ow]: `splits` blocks per channel over whole images (one block per channel
// left 84 of 148 SMs idle at 64 channels: 223 us for 25.7 MB), folded in order by slab_fold_kernel; a single block
// writes its sum itself. 2^log_row threads share an image's positions, the others take further images: with 256 on one
// position each, 256 images of 1 x 1 in 128 channels took 24 us, 2.0 now.
template <typename T>
__global__ void __launch_bounds__(256) channel_sum_kernel(const T* __restrict__ dy, float* __restrict__ part,
                                                          T* __restrict__ db, int N, int OC, long long spatial, int splits,
                                                          int log_row) {
  __shared__ float red[8];
  const int oc = blockIdx.x, z = blockIdx.y;
  float acc = 0.f;
  const T* p = dy + (long long)oc * spatial;
  const long long image = (long long)OC * spatial;
  if (spatial > 256) {
    for (int n = z; n < N; n += splits) {
      const T* q = p + n * image;
      float a0 = 0.f;
#pragma unroll 4
      for (long long i = threadIdx.x; i < spatial; i += 256) a0 += to_f<T>(q[i]);
      acc += a0;
    }
  } else {   // a position to a thread: loads of several images in flight
    const int col = (int)threadIdx.x & ((1 << log_row) - 1), step = splits * (256 >> log_row);
    if (col < spatial) {
      p += col;
#pragma unroll 8
      for (int n = z + splits * ((int)threadIdx.x >> log_row); n < N; n += step) acc += to_f<T>(p[n * image]);
    }
  }
  acc = block_sum_256(acc, red);
  if (threadIdx.x != 0) return;
  if (splits > 1) part[(long long)z * OC + oc] = acc;
  else db[oc] = from_f<T>(acc);
}

// ---- pooling ----------------------------------------------------------------------------------------------
struct PoolGeom {
  int NC, H, W, OH, OW, kH, kW, sh, sw, ph, pw;
  int count_include_pad;
};

// idx[i] = flat position (h * W + w) of the maximum inside the plane; the first maximum wins (NaN wins
// over numbers, as in the usual definition).
template <typename T>
__global__ void maxpool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int* __restrict__ idx, PoolGeom g) {
  const long long total = (long long)g.NC * g.OH * g.OW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ow = (int)(i % g.OW);
    const int oh = (int)((i / g.OW) % g.OH);
    const long long nc = i / ((long long)g.OW * g.OH);
    const T* xp = x + nc * g.H * g.W;
    float best = -INFINITY;
    int bi = -1;
    for (int kh = 0; kh < g.kH; ++kh) {
      const int h = oh * g.sh - g.ph + kh;
      if (h < 0 || h >= g.H) continue;
      for (int kw = 0; kw < g.kW; ++kw) {
        const int w = ow * g.sw - g.pw + kw;
        if (w < 0 || w >= g.W) continue;
        const float v = to_f<T>(xp[h * g.W + w]);
        if (bi < 0 || v > best || v != v) {
          if (!(best != best)) {  // keep an earlier NaN
            best = v;
            bi = h * g.W + w;
          }
        }
      }
    }
    y[i] = from_f<T>(best);
    if (idx != nullptr) idx[i] = bi;
  }
}

// dx[nc, h, w] = sum of dy over the windows whose arg-max is (h, w): every input element looks at the
// windows that contain it (gather), so overlapping windows need no atomics.
template <typename T>
__global__ void maxpool_bwd_kernel(const T* __restrict__ dy, const int* __restrict__ idx, T* __restrict__ dx,
                                   PoolGeom g) {
  const long long total = (long long)g.NC * g.H * g.W;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(i % g.W);
    const int h = (int)((i / g.W) % g.H);
    const long long nc = i / ((long long)g.W * g.H);
    const int me = h * g.W + w;
    // windows (oh, ow) with oh*sh - ph <= h < oh*sh - ph + kH
    const int oh_lo = max(0, (h + g.ph - g.kH + g.sh) / g.sh), oh_hi = min(g.OH - 1, (h + g.ph) / g.sh);
    const int ow_lo = max(0, (w + g.pw - g.kW + g.sw) / g.sw), ow_hi = min(g.OW - 1, (w + g.pw) / g.sw);
    float acc = 0.f;
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        const long long o = (nc * g.OH + oh) * g.OW + ow;
        if (idx[o] == me) acc += to_f<T>(dy[o]);
      }
    dx[i] = from_f<T>(acc);
  }
}

__device__ __forceinline__ int pool_count(const PoolGeom& g, int oh, int ow) {
  if (g.count_include_pad) return g.kH * g.kW;
  const int h0 = max(0, oh * g.sh - g.ph), h1 = min(g.H, oh * g.sh - g.ph + g.kH);
  const int w0 = max(0, ow * g.sw - g.pw), w1 = min(g.W, ow * g.sw - g.pw + g.kW);
  return max(1, (h1 - h0) * (w1 - w0));
}

template <typename T>
__global__ void avgpool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, PoolGeom g) {
  const long long total = (long long)g.NC * g.OH * g.OW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int ow = (int)(i % g.OW);
    const int oh = (int)((i / g.OW) % g.OH);
    const long long nc = i / ((long long)g.OW * g.OH);
    const T* xp = x + nc * g.H * g.W;
    float acc = 0.f;
    for (int kh = 0; kh < g.kH; ++kh) {
      const int h = oh * g.sh - g.ph + kh;
      if (h < 0 || h >= g.H) continue;
      for (int kw = 0; kw < g.kW; ++kw) {
        const int w = ow * g.sw - g.pw + kw;
        if (w < 0 || w >= g.W) continue;
        acc += to_f<T>(xp[h * g.W + w]);
      }
    }
    y[i] = from_f<T>(acc / (float)pool_count(g, oh, ow));
  }
}

template <typename T>
__global__ void avgpool_bwd_kernel(const T* __restrict__ dy, T* __restrict__ dx, PoolGeom g) {
  const long long total = (long long)g.NC * g.H * g.W;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(i % g.W);
    const int h = (int)((i / g.W) % g.H);
    const long long nc = i / ((long long)g.W * g.H);
    const int oh_lo = max(0, (h + g.ph - g.kH + g.sh) / g.sh), oh_hi = min(g.OH - 1, (h + g.ph) / g.sh);
    const int ow_lo = max(0, (w + g.pw - g.kW + g.sw) / g.sw), ow_hi = min(g.OW - 1, (w + g.pw) / g.sw);
    float acc = 0.f;
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow)
        acc += to_f<T>(dy[(nc * g.OH + oh) * g.OW + ow]) / (float)pool_count(g, oh, ow);
    dx[i] = from_f<T>(acc);
  }
}

static inline int grid_1d(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  return b < 1 ? 1 : (int)b;
}

static inline ConvGeom make_geom(const int* g) {
  ConvGeom c;
  c.N = g[0]; c.C = g[1]; c.H = g[2]; c.W = g[3]; c.OC = g[4]; c.kH = g[5]; c.kW = g[6]; c.OH = g[7]; c.OW = g[8];
  c.sh = g[9]; c.sw = g[10]; c.ph = g[11]; c.pw = g[12]; c.dh = g[13]; c.dw = g[14]; c.groups = g[15];
  return c;
}

static inline bool geom_ok(const ConvGeom& c) {
  return c.N > 0 && c.C > 0 && c.OC > 0 && c.groups > 0 && c.C % c.groups == 0 && c.OC % c.groups == 0 &&
         c.sh > 0 && c.sw > 0 && c.dh > 0 && c.dw > 0 && c.kH > 0 && c.kW > 0 && c.OH > 0 && c.OW > 0;
}

}  // namespace mmj

using namespace mmj;
#define STREAM ((cudaStream_t)stream)
#define DISPATCH(dtype, CALL_F32, CALL_BF16) \
  do {                                       \
    if ((dtype) == 1) { CALL_F32; }          \
    else if ((dtype) == 0) { CALL_BF16; }    \
    else return -1;                          \
  } while (0)

// geom: host int[16] = N, C, H, W, OC, kH, kW, OH, OW, sh, sw, ph, pw, dh, dw, groups. dtype: 0 bf16, 1 fp32.
MMJ_API int mmj_im2col(const void* x, void* cols, const int* geom, long long ldc, int dtype, void* stream) {
  const ConvGeom g = make_geom(geom);
  if (!geom_ok(g) || ldc < (long long)g.C * g.kH * g.kW || ldc > 0x7fffffc0LL) return -2;
  const long long total = (long long)g.N * g.OH * g.OW * ldc;
  if (total <= 131072) {
    const unsigned small_grid = (unsigned)((total + 255) / 256);
    DISPATCH(dtype, (im2col_small_kernel<float><<<small_grid, 256, 0, STREAM>>>((const float*)x, (float*)cols, g, (int)ldc)),
             (im2col_small_kernel<__nv_bfloat16><<<small_grid, 256, 0, STREAM>>>((const __nv_bfloat16*)x,
                                                                                 (__nv_bfloat16*)cols, g, (int)ldc)));
    return (int)cudaGetLastError();
  }
  const long long pos_tiles = ((long long)g.N * g.OH * g.OW + 31) / 32;
  // 16 columns to a warp while 64 would leave an SM fewer than eight warps (times above the kernel)
  const bool narrow = pos_tiles * ((ldc + 63) / 64) < 148 * 8;
  const long long blocks = (pos_tiles * (narrow ? (ldc + 15) / 16 : (ldc + 63) / 64) + 3) / 4;
  const unsigned grid = (unsigned)(blocks < 148 * 32 ? blocks : 148 * 32);
  // 16-byte stores need rows that are whole vectors
  const int vec = ldc % (dtype == 1 ? 4 : 8) == 0 && ((uintptr_t)cols & 15) == 0;
  const float* xf = (const float*)x;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  if (dtype == 1 && narrow) im2col_kernel<float, 16><<<grid, 128, 0, STREAM>>>(xf, (float*)cols, g, ldc, vec);
  else if (dtype == 1) im2col_kernel<float, 64><<<grid, 128, 0, STREAM>>>(xf, (float*)cols, g, ldc, vec);
  else if (dtype == 0 && narrow) im2col_kernel<__nv_bfloat16, 16><<<grid, 128, 0, STREAM>>>(xb, (__nv_bfloat16*)cols, g, ldc, vec);
  else if (dtype == 0) im2col_kernel<__nv_bfloat16, 64><<<grid, 128, 0, STREAM>>>(xb, (__nv_bfloat16*)cols, g, ldc, vec);
  else return -1;
  return (int)cudaGetLastError();
}
MMJ_API int mmj_col2im(const void* cols, void* dx, const int* geom, long long ldc, int dtype, void* stream) {
  const ConvGeom g = make_geom(geom);
  if (!geom_ok(g) || ldc < (long long)g.C * g.kH * g.kW) return -2;
  const long long total = (long long)g.N * g.C * g.H * g.W;
  DISPATCH(dtype, (col2im_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)cols, (float*)dx, g, ldc)),
           (col2im_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>((const __nv_bfloat16*)cols,
                                                                              (__nv_bfloat16*)dx, g, ldc)));
  return (int)cudaGetLastError();
}
// The tiled kernels address one image and one filter bank with 32-bit offsets. Their narrowest tile has 16 output
// channels, so a depthwise layer fills one row of it and stays with the one-thread-per-output kernels (N32 C64
// 56x56 k3, direct / tiled, us: forward 128 / 230, input gradient 223 / 343, weight gradient 361 / 853). From two
// channels per group the tiles win (32 groups of 2: 190 / 180, 386 / 235, 685 / 368), and without groups a single
// filter mostly does (N16 C64 56x56 OC1: forward 88 / 55, weight gradient 182 / 62; see lone_channel_direct).
static inline bool tiled_ok(const ConvGeom& g, int m_per_group) {
  const long long lim = 0x3fffffffLL;
  return (m_per_group >= 2 || g.groups == 1) && (long long)g.C * g.H * g.W < lim && (long long)g.OC * g.OH * g.OW < lim &&
         (long long)g.OC * (g.C / g.groups) * g.kH * g.kW < lim && (long long)g.kH * g.dh * g.W < lim &&
         (long long)g.H + g.ph + (long long)g.kH * g.dh < (1 << 28) &&
         (long long)g.W + g.pw + (long long)g.kW * g.dw < (1 << 28);
}
// One output channel without groups: the tiles win by their blocks in flight, until the positions alone give the direct
// kernel enough of them and long rows of taps read the image from cache. fp32, direct / tiled, us: forward of 200704
// positions, 3x3 taps of 1 / 3 / 8 / 32 channels 6.8 / 9.1, 12.1 / 13.6, 24.8 / 25.5, 85.7 / 79.3, 5x5 of 1 / 64 channels
// 8.7 / 13.3, 303 / 420; of 65536 positions 3x3 of 1 channel 3.4 / 4.1; of 50176 3x3 of 8 12.2 / 8.6, 5x5 of 1 / 64 4.4 / 4.9, 136 / 126, 11x11 of 64
// 483 / 593; of 12544 positions 11x11 of 64 453 / 332. The input gradient's direct kernel checks every tap against the
// stride: 200704 positions, 3x3 taps of 1 / 3 filters 10.5 / 12.1, 24.0 / 16.4.
static inline bool lone_channel_direct(const GatherGeom& t) {
  if (t.M != 1 || t.cls_h != 1 || t.cls_w != 1) return false;
  const long long P = (long long)t.N * t.PHf * t.PWf;
  const int taps = t.kH * t.kW;
  if (t.transposed) return P >= 768 * 148 && taps >= 9 && t.channels * taps <= 9;
  return (P >= 768 * 148 && (taps >= 25 || (taps >= 9 && t.channels <= 8))) ||
         (P >= 256 * 148 && (taps >= 81 || (taps >= 25 && t.channels <= 8) || (taps >= 9 && t.channels == 1)));
}
// 64-channel tiles unless they would leave a half-empty last one
static inline int tile_rows(int m) { return m <= 16 ? 16 : (m % 64 >= 1 && m % 64 <= 32) ? 32 : 64; }

template <typename T>
static int launch_gather(const void* src, const void* w, const void* bias, void* dst, const GatherGeom& g,
                         cudaStream_t st) {
  const long long P = (long long)g.N * ((g.PHf + g.cls_h - 1) / g.cls_h) * ((g.PWf + g.cls_w - 1) / g.cls_w);
  // smaller tiles while the blocks would not reach every SM
  int bm = tile_rows(g.M);
  while (bm > 16 && ((P + kGatherBN - 1) / kGatherBN) * ((g.M + bm - 1) / bm) * g.groups * g.cls_h * g.cls_w < 148)
    bm /= 2;
  const dim3 grid((unsigned)((P + kGatherBN - 1) / kGatherBN), (unsigned)(((g.M + bm - 1) / bm) * g.groups),
                  (unsigned)(g.cls_h * g.cls_w));
  const T *s = (const T*)src, *wt = (const T*)w, *b = (const T*)bias;
  if (bm == 64) conv_gather_kernel<T, 64, 8, 8><<<grid, kGatherThreads, 0, st>>>(s, wt, b, (T*)dst, g);
  else if (bm == 32) conv_gather_kernel<T, 32, 4, 8><<<grid, kGatherThreads, 0, st>>>(s, wt, b, (T*)dst, g);
  else conv_gather_kernel<T, 16, 4, 4><<<grid, kGatherThreads, 0, st>>>(s, wt, b, (T*)dst, g);
  return (int)cudaGetLastError();
}
static inline bool grid_fits(const GatherGeom& g) {
  const long long P = (long long)g.N * g.PHf * g.PWf;
  return P / kGatherBN < 0x7ffffff0LL && (long long)((g.M + 15) / 16) * g.groups <= 65535 &&
         (long long)g.cls_h * g.cls_w <= 65535;
}

MMJ_API int mmj_conv2d_fwd(const void* x, const void* w, const void* bias, void* y, const int* geom, int dtype,
                           void* stream) {
  const ConvGeom g = make_geom(geom);
  if (!geom_ok(g)) return -2;
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  GatherGeom t = {};
  t.SH = g.H; t.SW = g.W; t.cls_h = t.cls_w = 1; t.PHf = g.OH; t.PWf = g.OW;
  t.pos_s_h = g.sh; t.pos_s_w = g.sw; t.pos_o_h = -g.ph; t.pos_o_w = -g.pw;
  t.kH = g.kH; t.kW = g.kW; t.dh = g.dh; t.dw = g.dw; t.ph = g.ph; t.pw = g.pw;
  t.channels = cg; t.M = ocg; t.groups = g.groups; t.N = g.N;
  t.src_n = (long long)g.C * g.H * g.W; t.src_g = (long long)cg * g.H * g.W;
  t.w_ch = (long long)g.kH * g.kW; t.w_m = t.w_ch * cg; t.w_g = t.w_m * ocg;
  t.dst_m = (long long)g.OH * g.OW; t.dst_g = t.dst_m * ocg; t.dst_n = t.dst_m * g.OC;
  if (tiled_ok(g, ocg) && grid_fits(t) && !lone_channel_direct(t)) {
    DISPATCH(dtype, return launch_gather<float>(x, w, bias, y, t, STREAM),
             return launch_gather<__nv_bfloat16>(x, w, bias, y, t, STREAM));
  }
  const long long total = (long long)g.N * g.OC * g.OH * g.OW;
  DISPATCH(dtype, (conv2d_fwd_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)x, (const float*)w,
                                                                                 (const float*)bias, (float*)y, g)),
           (conv2d_fwd_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>(
               (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, (__nv_bfloat16*)y, g)));
  return (int)cudaGetLastError();
}
MMJ_API int mmj_conv2d_dx(const void* dy, const void* w, const void* bias, void* dx, const int* geom, int dtype,
                          void* stream) {
  const ConvGeom g = make_geom(geom);
  if (!geom_ok(g)) return -2;
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  GatherGeom t = {};
  t.SH = g.OH; t.SW = g.OW; t.cls_h = g.sh; t.cls_w = g.sw; t.PHf = g.H; t.PWf = g.W;
  t.pos_s_h = t.pos_s_w = 1;
  t.kH = g.kH; t.kW = g.kW; t.dh = g.dh; t.dw = g.dw; t.ph = g.ph; t.pw = g.pw;
  t.transposed = 1; t.channels = ocg; t.M = cg; t.groups = g.groups; t.N = g.N;
  t.src_n = (long long)g.OC * g.OH * g.OW; t.src_g = (long long)ocg * g.OH * g.OW;
  t.w_m = (long long)g.kH * g.kW; t.w_ch = t.w_m * cg; t.w_g = t.w_ch * ocg;
  t.dst_m = (long long)g.H * g.W; t.dst_g = t.dst_m * cg; t.dst_n = t.dst_m * g.C;
  // a stride larger than the image would leave classes without pixels
  if (tiled_ok(g, cg) && grid_fits(t) && g.sh <= g.H && g.sw <= g.W && !lone_channel_direct(t)) {
    DISPATCH(dtype, return launch_gather<float>(dy, w, bias, dx, t, STREAM),
             return launch_gather<__nv_bfloat16>(dy, w, bias, dx, t, STREAM));
  }
  const long long total = (long long)g.N * g.C * g.H * g.W;
  DISPATCH(dtype, (conv2d_dx_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)dy, (const float*)w,
                                                                                (const float*)bias, (float*)dx, g)),
           (conv2d_dx_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>(
               (const __nv_bfloat16*)dy, (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, (__nv_bfloat16*)dx, g)));
  return (int)cudaGetLastError();
}

// Slices of the positions in a tiled weight gradient (0: the direct kernel runs, no workspace). Enough blocks for
// two rounds of four per SM, at least 256 positions each, and at most 64 MB of slabs.
static int wgrad_slices(const ConvGeom& g, long long* slice) {
  const int cg = g.C / g.groups, ocg = g.OC / g.groups;
  const long long K = (long long)cg * g.kH * g.kW, P = (long long)g.N * g.OH * g.OW;
  const int bm = tile_rows(ocg);
  const long long tiles_m = (long long)((ocg + bm - 1) / bm) * g.groups, tiles_k = (K + kWgBN - 1) / kWgBN;
  // fewer than 8 filter taps in a 64-wide tile is mostly padding
  if (!tiled_ok(g, ocg) || K < 8 || tiles_m > 65535 || P > 0x7fffff00LL) return 0;
  // A small gradient stays with the direct kernel, one block to an element: the tiles' chain and the fold take 11 to 14 us
  // at least, the direct blocks about 2.4 us a thousand positions (of 1000 and more) and 500 elements. Direct / tiled, us:
  // one filter of 9 weights, 196 positions 2.4 / 11.2, 3136 8.9 / 14.1, 12544 29.3 / 13.3; 3 x 121 weights, 3136 positions
  // 12.0 / 14.1; 64 x 9 14.8 / 14.0; 64 x 25, 784 positions 14.7 / 13.8; 8 x 576, 12544 positions 315 / 19.
  const long long elems = g.OC * K, pos = P > 1000 ? P : 1000;
  if (pos * (elems > 500 ? elems : 500) < 3700 * 500) return 0;
  long long s = (2 * 4 * 148 + tiles_m * tiles_k - 1) / (tiles_m * tiles_k);
  const long long by_work = P / 256, by_mem = (64LL << 20) / (4 * g.OC * K);
  if (s > by_work) s = by_work;
  if (s > by_mem) s = by_mem;
  if (s > 1024) s = 1024;
  if (s < 1) s = 1;
  long long len = (P + s - 1) / s;
  len = (len + kWgBP - 1) / kWgBP * kWgBP;
  *slice = len;
  return (int)((P + len - 1) / len);
}
// fp32 values of workspace that mmj_conv2d_dw needs for this geometry
MMJ_API long long mmj_conv2d_dw_scratch(const int* geom) {
  const ConvGeom g = make_geom(geom);
  long long len = 0;
  if (!geom_ok(g)) return 0;
  return wgrad_slices(g, &len) * (long long)g.OC * (g.C / g.groups) * g.kH * g.kW;
}
template <typename T>
static int launch_wgrad(const void* x, const void* dy, void* dw, float* scratch, const ConvGeom& g, int S,
                        long long len, cudaStream_t st) {
  const int ocg = g.OC / g.groups;
  const long long K = (long long)(g.C / g.groups) * g.kH * g.kW, n = g.OC * K;
  const int bm = tile_rows(ocg);
  const dim3 grid((unsigned)((K + kWgBN - 1) / kWgBN), (unsigned)(((ocg + bm - 1) / bm) * g.groups), (unsigned)S);
  if (bm == 64) conv_wgrad_kernel<T, 64><<<grid, kWgThreads, 0, st>>>((const T*)x, (const T*)dy, scratch, g, len);
  else if (bm == 32) conv_wgrad_kernel<T, 32><<<grid, kWgThreads, 0, st>>>((const T*)x, (const T*)dy, scratch, g, len);
  else conv_wgrad_kernel<T, 16><<<grid, kWgThreads, 0, st>>>((const T*)x, (const T*)dy, scratch, g, len);
  slab_fold_kernel<T, true><<<(unsigned)((n + 31) / 32), 256, 0, st>>>(scratch, (T*)dw, n, S, (const T*)x, (const T*)dy, g,
                                                                     len);
  return (int)cudaGetLastError();
}
MMJ_API int mmj_conv2d_dw(const void* x, const void* dy, void* dw, float* scratch, const int* geom, int dtype,
                          void* stream) {
  const ConvGeom g = make_geom(geom);
  if (!geom_ok(g)) return -2;
  long long len = 0;
  const int S = scratch != nullptr ? wgrad_slices(g, &len) : 0;
  if (S > 0) {
    DISPATCH(dtype, return launch_wgrad<float>(x, dy, dw, scratch, g, S, len, STREAM),
             return launch_wgrad<__nv_bfloat16>(x, dy, dw, scratch, g, S, len, STREAM));
  }
  const long long elems = (long long)g.OC * (g.C / g.groups) * g.kH * g.kW;
  if (elems > 0x7fffffffLL) return -3;
  DISPATCH(dtype, (conv2d_dw_kernel<float><<<(unsigned)elems, 256, 0, STREAM>>>((const float*)x, (const float*)dy,
                                                                                 (float*)dw, g)),
           (conv2d_dw_kernel<__nv_bfloat16><<<(unsigned)elems, 256, 0, STREAM>>>(
               (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dw, g)));
  return (int)cudaGetLastError();
}
// Blocks per channel: two to an SM where each still has 1024 values, since a second one costs a fold.
MMJ_API int mmj_channel_sum_splits(int N, int OC, long long spatial) {
  long long s = (2 * 148 + OC - 1) / OC;
  const long long by_work = N * spatial / 1024;
  if (s > by_work) s = by_work;
  if (s > N) s = N;
  return s < 1 ? 1 : (int)s;
}
// scratch: mmj_channel_sum_splits(N, OC, spatial) * OC fp32 values where that is more than one row of them
MMJ_API int mmj_channel_sum(const void* dy, void* db, float* scratch, int N, int OC, long long spatial, int dtype,
                            void* stream) {
  if (N <= 0 || OC <= 0 || spatial <= 0) return -2;
  const int S = mmj_channel_sum_splits(N, OC, spatial);
  int log_row = 0;
  while (log_row < 8 && (1 << log_row) < spatial) ++log_row;
  const dim3 grid((unsigned)OC, (unsigned)S);
  DISPATCH(dtype, (channel_sum_kernel<float><<<grid, 256, 0, STREAM>>>((const float*)dy, scratch, (float*)db, N, OC, spatial,
                                                                       S, log_row)),
           (channel_sum_kernel<__nv_bfloat16><<<grid, 256, 0, STREAM>>>(
               (const __nv_bfloat16*)dy, scratch, (__nv_bfloat16*)db, N, OC, spatial, S, log_row)));
  if (S == 1) return (int)cudaGetLastError();
  const ConvGeom none = {};
  DISPATCH(dtype, (slab_fold_kernel<float, false><<<(OC + 31) / 32, 256, 0, STREAM>>>(scratch, (float*)db, OC, S, nullptr,
                                                                                      nullptr, none, 0)),
           (slab_fold_kernel<__nv_bfloat16, false><<<(OC + 31) / 32, 256, 0, STREAM>>>(scratch, (__nv_bfloat16*)db, OC, S,
                                                                                       nullptr, nullptr, none, 0)));
  return (int)cudaGetLastError();
}

// pool geom: host int[12] = NC, H, W, OH, OW, kH, kW, sh, sw, ph, pw, count_include_pad
static inline PoolGeom make_pool(const int* g) {
  PoolGeom p;
  p.NC = g[0]; p.H = g[1]; p.W = g[2]; p.OH = g[3]; p.OW = g[4]; p.kH = g[5]; p.kW = g[6]; p.sh = g[7]; p.sw = g[8];
  p.ph = g[9]; p.pw = g[10]; p.count_include_pad = g[11];
  return p;
}
static inline bool pool_ok(const PoolGeom& p) {
  return p.NC > 0 && p.H > 0 && p.W > 0 && p.OH > 0 && p.OW > 0 && p.kH > 0 && p.kW > 0 && p.sh > 0 && p.sw > 0 &&
         (long long)p.H * p.W < 0x7fffffffLL;
}
MMJ_API int mmj_maxpool2d_fwd(const void* x, void* y, int* idx, const int* geom, int dtype, void* stream) {
  const PoolGeom g = make_pool(geom);
  if (!pool_ok(g)) return -2;
  const long long total = (long long)g.NC * g.OH * g.OW;
  DISPATCH(dtype, (maxpool_fwd_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)x, (float*)y, idx, g)),
           (maxpool_fwd_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>((const __nv_bfloat16*)x,
                                                                                   (__nv_bfloat16*)y, idx, g)));
  return (int)cudaGetLastError();
}
MMJ_API int mmj_maxpool2d_bwd(const void* dy, const int* idx, void* dx, const int* geom, int dtype, void* stream) {
  const PoolGeom g = make_pool(geom);
  if (!pool_ok(g)) return -2;
  const long long total = (long long)g.NC * g.H * g.W;
  DISPATCH(dtype, (maxpool_bwd_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)dy, idx, (float*)dx, g)),
           (maxpool_bwd_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>((const __nv_bfloat16*)dy, idx,
                                                                                   (__nv_bfloat16*)dx, g)));
  return (int)cudaGetLastError();
}
MMJ_API int mmj_avgpool2d_fwd(const void* x, void* y, const int* geom, int dtype, void* stream) {
  const PoolGeom g = make_pool(geom);
  if (!pool_ok(g)) return -2;
  const long long total = (long long)g.NC * g.OH * g.OW;
  DISPATCH(dtype, (avgpool_fwd_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)x, (float*)y, g)),
           (avgpool_fwd_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>((const __nv_bfloat16*)x,
                                                                                   (__nv_bfloat16*)y, g)));
  return (int)cudaGetLastError();
}
MMJ_API int mmj_avgpool2d_bwd(const void* dy, void* dx, const int* geom, int dtype, void* stream) {
  const PoolGeom g = make_pool(geom);
  if (!pool_ok(g)) return -2;
  const long long total = (long long)g.NC * g.H * g.W;
  DISPATCH(dtype, (avgpool_bwd_kernel<float><<<grid_1d(total), 256, 0, STREAM>>>((const float*)dy, (float*)dx, g)),
           (avgpool_bwd_kernel<__nv_bfloat16><<<grid_1d(total), 256, 0, STREAM>>>((const __nv_bfloat16*)dy,
                                                                                   (__nv_bfloat16*)dx, g)));
  return (int)cudaGetLastError();
}
