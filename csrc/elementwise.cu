// Memory-bound kernels of the training step for sm_100a: RMSNorm, RoPE, SwiGLU, vocabulary
// cross-entropy, embedding, the sharded AdamW update fused with the bf16 all-gather-input refresh,
// gradient sum-of-squares, and flat casts.  All are 16-byte vectorised and sized to keep
// 148 SMs x several CTAs in flight; each is bandwidth-bound by design (one read and one write of
// every operand).
#include "common.cuh"
#include "yafsdp_b200.h"


namespace {

struct alignas(16) bf16x8 {
  uint32_t u[4];
};
YF_DEVINL void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
YF_DEVINL void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 v;
  v.x = pack_bf16x2(f[0], f[1]);
  v.y = pack_bf16x2(f[2], f[3]);
  v.z = pack_bf16x2(f[4], f[5]);
  v.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = v;
}

template <int THREADS>
YF_DEVINL float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < THREADS / 32) ? red[l] : 0.f;
  t = warp_sum(t);
  return t;
}
template <int THREADS>
YF_DEVINL float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < THREADS / 32) ? red[l] : -INFINITY;
  t = warp_max(t);
  return t;
}

// ------------------------------------------------------------------ RMSNorm
// y = x * rsqrt(mean(x^2) + eps) * w ; one CTA per row, the row stays in registers between passes.
constexpr int RN_THREADS = 256;
constexpr int RN_MAXV = 4;  // vectors of 8 per thread held in registers: D <= 256*8*4 = 8192

__global__ void __launch_bounds__(RN_THREADS) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                 const __nv_bfloat16* __restrict__ w,
                                                                 __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                                                 int T, int D, float eps) {
  __shared__ float red[32];
  const int nvec = D / 8;
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    const __nv_bfloat16* xr = x + (size_t)row * D;
    float xv[RN_MAXV][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < RN_MAXV; ++i) {
      const int v = threadIdx.x + i * RN_THREADS;
      if (v < nvec) {
        load8(xr + v * 8, xv[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += xv[i][j] * xv[i][j];
      }
    }
    for (int v = threadIdx.x + RN_MAXV * RN_THREADS; v < nvec; v += RN_THREADS) {  // rows wider than the register tile
      float t[8];
      load8(xr + v * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += t[j] * t[j];
    }
    ss = block_sum<RN_THREADS>(ss, red);
    const float r = rsqrtf(ss / (float)D + eps);
    if (threadIdx.x == 0 && rstd) rstd[row] = r;
    __nv_bfloat16* yr = y + (size_t)row * D;
#pragma unroll
    for (int i = 0; i < RN_MAXV; ++i) {
      const int v = threadIdx.x + i * RN_THREADS;
      if (v < nvec) {
        float wv[8], o[8];
        load8(w + v * 8, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = xv[i][j] * r * wv[j];
        store8(yr + v * 8, o);
      }
    }
    for (int v = threadIdx.x + RN_MAXV * RN_THREADS; v < nvec; v += RN_THREADS) {
      float t[8], wv[8], o[8];
      load8(xr + v * 8, t);
      load8(w + v * 8, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = t[j] * r * wv[j];
      store8(yr + v * 8, o);
    }
  }
}

// G warps per row (G = 1, 2 or 4; D <= 32 * G * 8 * RNW_NV), four warps per CTA: the row stays in registers as packed bf16,
// every operand of a row is requested before anything is reduced (one exposed memory latency per row, not one per pass),
// and the only synchronisation is a named barrier among the G warps of the row.  Thread t of a row's group holds the
// vectors t, t + 32 G, ... of the row (contiguous 512 G bytes per load instruction).
constexpr int RNW_WARPS = 4;
constexpr int RNW_NV = 8;  // vectors of a row per thread
YF_DEVINL void unpack8(const uint4& v, float (&f)[8]) {
  float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
template <int G>
YF_DEVINL float row_group_sum(float v, float* red, int row_in_cta) {
  v = warp_sum(v);
  if (G == 1) return v;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  if (row_in_cta == 0) named_bar_sync(1, 32 * G);  // literal barrier numbers: a computed one reserves all sixteen
  else named_bar_sync(2, 32 * G);
  float t = 0.f;
#pragma unroll
  for (int g = 0; g < G; ++g) t += red[row_in_cta * G + g];
  return t;
}

template <int G>
__global__ void __launch_bounds__(RNW_WARPS * 32) rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x,
                                                                          const __nv_bfloat16* __restrict__ w,
                                                                          __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                                                          int T, int D, float eps) {
  __shared__ float red[RNW_WARPS];
  constexpr int ROWS = RNW_WARPS / G, TPR = 32 * G;
  const int row_in_cta = threadIdx.x / TPR, tr = threadIdx.x % TPR;
  const int row = blockIdx.x * ROWS + row_in_cta;
  if (row >= T) return;
  const int nvec = D / 8;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * D);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4 xv[RNW_NV], wv[RNW_NV];
#pragma unroll
  for (int i = 0; i < RNW_NV; ++i) {
    const int v = tr + TPR * i;
    xv[i] = v < nvec ? xr[v] : make_uint4(0u, 0u, 0u, 0u);
    wv[i] = v < nvec ? __ldg(wr + v) : make_uint4(0u, 0u, 0u, 0u);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < RNW_NV; ++i) {
    float f[8];
    unpack8(xv[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = row_group_sum<G>(ss, red, row_in_cta);
  const float r = rsqrtf(ss / (float)D + eps);
  if (tr == 0 && rstd) rstd[row] = r;
  __nv_bfloat16* yr = y + (size_t)row * D;
#pragma unroll
  for (int i = 0; i < RNW_NV; ++i) {
    const int v = tr + TPR * i;
    if (v < nvec) {
      float f[8], wf[8], o[8];
      unpack8(xv[i], f);
      unpack8(wv[i], wf);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = f[j] * r * wf[j];
      store8(yr + v * 8, o);
    }
  }
}

// Backward: dx = r * (dy*w - xhat * mean(dy*w*xhat)) (+ dres, the gradient arriving through the residual branch) and
// dw = sum_rows dy * xhat.  TPR threads per row (D <= 32 TPR), 256 threads = 256 / TPR rows at a time, two CTAs per SM that walk
// over the rows: a thread holds the same columns of every row, so dw is summed in registers on the way and x and dy are read once
// (a column reduction of its own read both again).  The row groups of a CTA meet in shared memory at the end (unless all
// of them together are below 2 MB); the sums go to rows of `partials`, added up in a fixed order by rmsnorm_bwd_dw_kernel, or, without
// partials, atomically to dw.
// Bound by HBM: 8 bytes per element with dres.  With dres, both kernels: 2048 x 4096 23 us, 8192 x 4096 57 us,
// 2048 x 8192 34 us (the dx and column kernels before: 27, 90 and 56 us).
constexpr int RNB_NV = 4;  // vectors of 8 per thread
constexpr int RNB_THREADS = 256;
template <int TPR>
__global__ void __launch_bounds__(RNB_THREADS, 2) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                     const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd,
                                                                     const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                                                     float* __restrict__ partials, float* __restrict__ dw, int T, int D, int combine) {
  constexpr int ROWS = RNB_THREADS / TPR;
  __shared__ float red[2][RNB_THREADS / 32];
  __shared__ float sums[ROWS > 1 ? TPR * RNB_NV * 8 : 1];
  const int group = threadIdx.x / TPR, tr = threadIdx.x % TPR;
  const int nvec = D / 8;
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  float acc[RNB_NV][8];
#pragma unroll
  for (int i = 0; i < RNB_NV; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  int parity = 0;
  for (int row = blockIdx.x * ROWS + group; row < T; row += gridDim.x * ROWS, parity ^= 1) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * D);
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + (size_t)row * D);
    const uint4* er = reinterpret_cast<const uint4*>(dres ? dres + (size_t)row * D : x);
    uint4 xv[RNB_NV], dv[RNB_NV], ev[RNB_NV];
#pragma unroll
    for (int i = 0; i < RNB_NV; ++i) {
      const int v = tr + TPR * i;
      const bool in = v < nvec;
      xv[i] = in ? xr[v] : make_uint4(0u, 0u, 0u, 0u);
      dv[i] = in ? dyr[v] : make_uint4(0u, 0u, 0u, 0u);
      ev[i] = (in && dres) ? er[v] : make_uint4(0u, 0u, 0u, 0u);
    }
    const float r = rstd[row];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < RNB_NV; ++i) {
      const int v = tr + TPR * i;
      if (v < nvec) {  // w comes from the L1 both times: its registers would cost the second CTA
        float xf[8], df[8], wf[8];
        unpack8(xv[i], xf);
        unpack8(dv[i], df);
        unpack8(__ldg(wr + v), wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float p = df[j] * (xf[j] * r);
          dot += p * wf[j];
          acc[i][j] += p;
        }
      }
    }
    dot = warp_sum(dot);
    if (TPR > 32) {  // the row's warps; two sets of slots, so one barrier per row is enough
      if ((threadIdx.x & 31) == 0) red[parity][threadIdx.x >> 5] = dot;
      if (group == 0) named_bar_sync(1, TPR);  // literal barrier numbers: a computed one reserves all sixteen
      else if (group == 1) named_bar_sync(2, TPR);
      else if (group == 2) named_bar_sync(3, TPR);
      else named_bar_sync(4, TPR);
      dot = 0.f;
#pragma unroll
      for (int g = 0; g < TPR / 32; ++g) dot += red[parity][group * (TPR / 32) + g];
    }
    dot /= (float)D;
    __nv_bfloat16* dxr = dx + (size_t)row * D;
#pragma unroll
    for (int i = 0; i < RNB_NV; ++i) {
      const int v = tr + TPR * i;
      if (v < nvec) {
        float xf[8], df[8], wf[8], ef[8], o[8];
        unpack8(xv[i], xf);
        unpack8(dv[i], df);
        unpack8(ev[i], ef);
        unpack8(__ldg(wr + v), wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = r * (df[j] * wf[j] - xf[j] * r * dot) + ef[j];
        store8(dxr + v * 8, o);
      }
    }
  }
  if (dw == nullptr) return;
  int part_row = blockIdx.x * ROWS + group;
  if (ROWS > 1 && combine) {  // sum the row groups: the last one ends up with the total
#pragma unroll 1
    for (int g = 0; g < ROWS; ++g) {
      if (group == g) {
#pragma unroll
        for (int i = 0; i < RNB_NV; ++i) {
          float* at = sums + (tr + TPR * i) * 8;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (g > 0) acc[i][j] += at[j];
            at[j] = acc[i][j];
          }
        }
      }
      __syncthreads();
    }
    if (group != ROWS - 1) return;
    part_row = blockIdx.x;
  }
#pragma unroll
  for (int i = 0; i < RNB_NV; ++i) {
    const int v = tr + TPR * i;
    if (v < nvec) {
      if (partials != nullptr) {
        float4* at = reinterpret_cast<float4*>(partials + (size_t)part_row * D + v * 8);
        at[0] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        at[1] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) atomicAdd(dw + v * 8 + j, acc[i][j]);
      }
    }
  }
}
// dw (= or +=) column sums of partials [n, D]: 32 columns per CTA, 32 row lanes
// sumsq (optional): += the squares of what was written
__global__ void __launch_bounds__(1024) rmsnorm_bwd_dw_kernel(const float* __restrict__ partials, float* __restrict__ dw, int n, int D, int add,
                                                              float* __restrict__ sumsq) {
  __shared__ float part[32][33];
  const int c = threadIdx.x & 31, lane_row = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + c;
  float s = 0.f;
  if (col < D)
    for (int i = lane_row; i < n; i += 32) s += partials[(size_t)i * D + col];
  part[lane_row][c] = s;
  __syncthreads();
  s = warp_sum(part[c][lane_row]);  // warp lane_row sums column blockIdx.x * 32 + lane_row over the row lanes
  const int mine = blockIdx.x * 32 + lane_row;
  if (add && mine < D) s += dw[mine];
  __syncthreads();
  if (c == 0) {
    if (mine < D) dw[mine] = s;
    part[0][lane_row] = mine < D ? s * s : 0.f;
  }
  __syncthreads();
  if (sumsq != nullptr && lane_row == 0) {
    const float total = warp_sum(part[0][c]);
    if (c == 0) atomicAdd(sumsq, total);
  }
}

// ------------------------------------------------------------------ RoPE (rotate-half pairing, in place)
// qkv: [T, row_stride] bf16 with n_heads heads of head_dim starting at column col0; pos = row % seq_len.
// cos/sin table: [seq_len, head_dim/2] fp32.  sign = +1 forward, -1 backward (inverse rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cs, int T, int seq_len,
                            long long row_stride, int col0, int n_heads, int head_dim, float sign) {
  const int half = head_dim / 2;
  const int vec_per_head = half / 8;
  const long long total = (long long)T * n_heads * vec_per_head;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(i % vec_per_head);
    const long long th = i / vec_per_head;
    const int h = (int)(th % n_heads);
    const long long t = th / n_heads;
    const int pos = (int)(t % seq_len);
    __nv_bfloat16* p = qkv + t * row_stride + col0 + h * head_dim + v * 8;
    float a[8], b[8], oa[8], ob[8];
    load8(p, a);
    load8(p + half, b);
    const float* c = cs + ((size_t)pos * half + v * 8) * 2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float co = c[2 * j], si = c[2 * j + 1] * sign;
      oa[j] = a[j] * co - b[j] * si;
      ob[j] = b[j] * co + a[j] * si;
    }
    store8(p, oa);
    store8(p + half, ob);
  }
}

// ------------------------------------------------------------------ SwiGLU
// gu: [T, 2F] (gate columns [0,F), up columns [F,2F)); h = silu(gate) * up
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h, long long T, int F) {
  const int vpr = F / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    float g[8], u[8], o[8];
    load8(gu + t * 2 * F + v * 8, g);
    load8(gu + t * 2 * F + F + v * 8, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    store8(h + t * F + v * 8, o);
  }
}
// dgate = dh * up * (sig + g*sig*(1-sig)), dup = dh * silu(g); written into dgu [T, 2F]
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dh,
                                  __nv_bfloat16* __restrict__ dgu, long long T, int F) {
  const int vpr = F / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    float g[8], u[8], d[8], og[8], ou[8];
    load8(gu + t * 2 * F + v * 8, g);
    load8(gu + t * 2 * F + F + v * 8, u);
    load8(dh + t * F + v * 8, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      og[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
      ou[j] = d[j] * g[j] * s;
    }
    store8(dgu + t * 2 * F + v * 8, og);
    store8(dgu + t * 2 * F + F + v * 8, ou);
  }
}

// ------------------------------------------------------------------ cross-entropy (forward + backward in one pass pair)
// logits [T, V] bf16 (row pitch ldl) are replaced in place by dlogits = (softmax - onehot) * grad_scale, where grad_scale is
// the host value times *scale_ptr when that device pointer is given (e.g. 1 / number of valid labels, counted on the device);
// loss_rows[t] = logsumexp - logit[label] (0 for ignored rows, label < 0).  One CTA per row.
// A row is read twice, and the rows in flight together stay in the L2, where the second read finds them.  The exponentials and the
// instructions around them bound it as much as the memory: two ex2 per logit (one instruction each, differences scaled by log2 e),
// the maximum of a batch of four vectors on packed bf16 with one rescale for all of them, and the label's term set apart.
// 8192 x 128256: 875 us (with a rescale per vector, __expf's guarded sequence and a label test per logit: 1075 us); 2048 x 32000: 62 us
// (73 us); 999 x 32000: 29 us.  Batches of two vectors: 1040 and 69 us; 256 threads: 960 and 57 us; 1024 threads: 940 and 81 us.
constexpr int CE_THREADS = 512, CE_BATCH = 4;
constexpr float LOG2E = 1.4426950408889634f;
// probabilities are computed 2^16 times too large: fast_exp2 flushes results below 2^-126, bf16 goes down to 2^-133
constexpr float CE_SHIFT = 16.f, CE_UNSHIFT = 1.f / 65536.f;
constexpr uint32_t BF16X2_NEG_INF = 0xff80ff80u;
YF_DEVINL uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_kernel(__nv_bfloat16* __restrict__ logits,
                                                                   const long long* __restrict__ labels,
                                                                   float* __restrict__ loss_rows, int T, int V,
                                                                   long long ldl, float grad_scale,
                                                                   const float* __restrict__ scale_ptr, int write_grad) {
  __shared__ float red[32];
  const int nvec = V / 8;
  if (scale_ptr != nullptr) grad_scale *= *scale_ptr;
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    __nv_bfloat16* lr = logits + (size_t)row * ldl;
    const long long label = labels[row];
    if (label < 0 || label >= V) {
      if (threadIdx.x == 0) loss_rows[row] = 0.f;
      if (write_grad) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int v = threadIdx.x; v < nvec; v += CE_THREADS) *reinterpret_cast<uint4*>(lr + v * 8) = z;
        for (int j = nvec * 8 + threadIdx.x; j < V; j += CE_THREADS) lr[j] = __float2bfloat16_rn(0.f);
      }
      continue;
    }
    // online max / sum-exp, CE_BATCH vectors at a time: one rescale for all of them
    float m = -INFINITY, s = 0.f;
    for (int v0 = threadIdx.x; v0 < nvec; v0 += CE_BATCH * CE_THREADS) {
      uint4 x[CE_BATCH];
#pragma unroll
      for (int i = 0; i < CE_BATCH; ++i) {
        const int v = v0 + i * CE_THREADS;
        x[i] = v < nvec ? *reinterpret_cast<const uint4*>(lr + v * 8) : make_uint4(BF16X2_NEG_INF, BF16X2_NEG_INF, BF16X2_NEG_INF, BF16X2_NEG_INF);
      }
      uint32_t mx = max_bf16x2(max_bf16x2(x[0].x, x[0].y), max_bf16x2(x[0].z, x[0].w));
#pragma unroll
      for (int i = 1; i < CE_BATCH; ++i)
        mx = max_bf16x2(mx, max_bf16x2(max_bf16x2(x[i].x, x[i].y), max_bf16x2(x[i].z, x[i].w)));
      const float2 pair = unpack_bf16x2(mx);
      const float nm = fmaxf(m, fmaxf(pair.x, pair.y));
      const float ref = nm == -INFINITY ? 0.f : nm;  // nothing but -inf so far: every term is zero
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < CE_BATCH; ++i) {
        if (v0 + i * CE_THREADS >= nvec) break;
        const uint32_t u[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(u[j]);
          acc += fast_exp2((f.x - ref) * LOG2E);
          acc += fast_exp2((f.y - ref) * LOG2E);
        }
      }
      s = s * fast_exp2((m - ref) * LOG2E) + acc;
      m = nm;
    }
    for (int j = nvec * 8 + threadIdx.x; j < V; j += CE_THREADS) {
      const float f = __bfloat162float(lr[j]);
      const float nm = fmaxf(m, f);
      const float ref = nm == -INFINITY ? 0.f : nm;
      s = s * fast_exp2((m - ref) * LOG2E) + fast_exp2((f - ref) * LOG2E);
      m = nm;
    }
    const float gm = block_max<CE_THREADS>(m, red);
    const float contrib = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
    const float gs = block_sum<CE_THREADS>(contrib, red);
    // differences to the maximum first: they are exact, logsumexp itself would be rounded at its own size
    const float log_gs = __logf(gs);
    if (threadIdx.x == 0) loss_rows[row] = (gm - __bfloat162float(lr[label])) + log_gs;
    if (write_grad) {
      __syncthreads();  // the label logit was read above before anyone overwrites it
      const float shift = CE_SHIFT - __log2f(gs), unshift = grad_scale * CE_UNSHIFT;
      const int label_vec = (int)(label >> 3), label_elem = (int)(label & 7);
      for (int v0 = threadIdx.x; v0 < nvec; v0 += CE_BATCH * CE_THREADS) {
        uint4 x[CE_BATCH];
#pragma unroll
        for (int i = 0; i < CE_BATCH; ++i)
          if (v0 + i * CE_THREADS < nvec) x[i] = *reinterpret_cast<const uint4*>(lr + (v0 + i * CE_THREADS) * 8);
#pragma unroll
        for (int i = 0; i < CE_BATCH; ++i) {
          const int v = v0 + i * CE_THREADS;
          if (v >= nvec) break;
          const uint32_t u[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
          float o[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(u[j]);
            o[2 * j] = fast_exp2(fmaf(f.x - gm, LOG2E, shift)) * unshift;
            o[2 * j + 1] = fast_exp2(fmaf(f.y - gm, LOG2E, shift)) * unshift;
          }
          if (v == label_vec) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float2 f = unpack_bf16x2(u[j / 2]);
              if (j == label_elem) o[j] = (__expf(((j & 1 ? f.y : f.x) - gm) - log_gs) - 1.f) * grad_scale;
            }
          }
          store8(lr + v * 8, o);
        }
      }
      for (int j = nvec * 8 + threadIdx.x; j < V; j += CE_THREADS) {
        float p = __expf((__bfloat162float(lr[j]) - gm) - log_gs);
        if (j == label) p -= 1.f;
        lr[j] = __float2bfloat16_rn(p * grad_scale);
      }
    }
  }
}

// The loss's two scalars, one block each: bound by the latency of a launch up to some 10^5 values.  Device time, us, against PyTorch's
// comparison, sum, clamp, cast and reciprocal / sum and product: 8192 tokens 2.2 against 12 / 2.2 against 4.4; 131072 tokens 6.5 against
// 19 / 4.6 against 10; 524288 tokens 19 against 19 / 11 against 10; 1048576 tokens 36 against 20 / 20 against 11 (next to 0.2 s of head
// GEMMs).
constexpr int ONE_BLOCK = 1024;
__global__ void __launch_bounds__(ONE_BLOCK) inv_valid_labels_kernel(const long long* __restrict__ labels, long long n, float* __restrict__ out) {
  __shared__ int count;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  int c = 0;
  for (long long i = threadIdx.x; i < n; i += ONE_BLOCK) c += labels[i] >= 0 ? 1 : 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(&count, c);
  __syncthreads();
  if (threadIdx.x == 0) *out = 1.f / (float)max(count, 1);
}
// out[b, s] = labels[b, s + 1], -100 at the end of a row (row pitch ld)
__global__ void shift_labels_kernel(const long long* __restrict__ labels, long long* __restrict__ out, long long n, int seq, long long ld) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / seq;
    const int s = (int)(i - b * seq);
    out[i] = s + 1 < seq ? labels[b * ld + s + 1] : -100;
  }
}
__global__ void __launch_bounds__(ONE_BLOCK) scaled_sum_kernel(const float* __restrict__ x, long long n, const float* __restrict__ scale, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += ONE_BLOCK) s += x[i];
  s = block_sum<ONE_BLOCK>(s, red);
  if (threadIdx.x == 0) *out = s * *scale;
}

// ------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const __nv_bfloat16* __restrict__ table, const long long* __restrict__ ids,
                                     __nv_bfloat16* __restrict__ out, long long T, int D, int V) {
  const int vpr = D / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    long long id = ids[t];
    uint4 val = make_uint4(0, 0, 0, 0);
    if (id >= 0 && id < V) val = *reinterpret_cast<const uint4*>(table + id * D + v * 8);
    *reinterpret_cast<uint4*>(out + t * D + v * 8) = val;
  }
}
// dtable[ids[t], :] += dout[t, :]  (fp32 table gradient; token ids repeat: atomics, four floats each).  `owner` (optional, V ints
// that need no initial value): one of the tokens with id i is left in owner[i].
__global__ void embedding_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const long long* __restrict__ ids,
                                     float* __restrict__ dtable, int* __restrict__ owner, long long T, int D, int V, int aligned) {
  const int vpr = D / 8;
  const long long total = T * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int v = (int)(i % vpr);
    const long long id = ids[t];
    if (id < 0 || id >= V) continue;
    float f[8];
    load8(dout + t * D + v * 8, f);
    float* dst = dtable + id * D + v * 8;
    if (aligned) {
      asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
      asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7]) : "memory");
    } else {  // a table that starts anywhere in a flat buffer
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dst + j, f[j]);
    }
    if (v == 0 && owner != nullptr) atomicExch(owner + id, (int)t);  // any of them will do
  }
}
// *out += sum of squares of the rows that some token touched, each row once: the token that owner[] names reads it.  The other
// rows of a gradient that started from zeros are zero: 32000 x 4096 after 2048 tokens, 33 MB instead of 524 MB.
__global__ void __launch_bounds__(256) embedding_sumsq_kernel(const float* __restrict__ dtable, const long long* __restrict__ ids,
                                                              const int* __restrict__ owner, float* __restrict__ out, long long T, int D, int V) {
  __shared__ float red[32];
  float acc = 0.f;
  for (long long t = blockIdx.x; t < T; t += gridDim.x) {
    const long long id = ids[t];
    if (id < 0 || id >= V || owner[id] != (int)t) continue;
    const float* row = dtable + id * D;
    for (int v = threadIdx.x; v < D; v += 256) acc += row[v] * row[v];
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

// ------------------------------------------------------------------ AdamW on the flat fp32 master shard
// p, m, v updated in place from g (scaled by *grad_scale_ptr when given, e.g. the clip coefficient);
// the bf16 copy that the next all-gather reads is refreshed in the same pass.
struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay, bc1, bc2;  // bc = 1 - beta^step
};
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                                    float* __restrict__ v, __nv_bfloat16* __restrict__ p_bf16,
                                                    const float* __restrict__ grad_scale_ptr, long long n, AdamArgs a) {
  const float gs = grad_scale_ptr ? *grad_scale_ptr : 1.f;
  const float inv_bc1 = 1.f / a.bc1;
  const float inv_sqrt_bc2 = rsqrtf(a.bc2);
  const long long nvec = n / 4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float4 pv = reinterpret_cast<float4*>(p)[i];
    const float4 gv = reinterpret_cast<const float4*>(g)[i];
    float4 mv = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float pe[4] = {pv.x, pv.y, pv.z, pv.w}, ge[4] = {gv.x, gv.y, gv.z, gv.w}, me[4] = {mv.x, mv.y, mv.z, mv.w},
          ve[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float gr = ge[j] * gs;
      pe[j] *= (1.f - a.lr * a.weight_decay);
      me[j] = a.beta1 * me[j] + (1.f - a.beta1) * gr;
      ve[j] = a.beta2 * ve[j] + (1.f - a.beta2) * gr * gr;
      const float denom = sqrtf(ve[j]) * inv_sqrt_bc2 + a.eps;
      pe[j] -= a.lr * (me[j] * inv_bc1) / denom;
    }
    reinterpret_cast<float4*>(p)[i] = make_float4(pe[0], pe[1], pe[2], pe[3]);
    reinterpret_cast<float4*>(m)[i] = make_float4(me[0], me[1], me[2], me[3]);
    reinterpret_cast<float4*>(v)[i] = make_float4(ve[0], ve[1], ve[2], ve[3]);
    if (p_bf16) {
      uint2 o;
      o.x = pack_bf16x2(pe[0], pe[1]);
      o.y = pack_bf16x2(pe[2], pe[3]);
      reinterpret_cast<uint2*>(p_bf16)[i] = o;
    }
  }
  // tail (n not a multiple of 4)
  for (long long i = nvec * 4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gr = g[i] * gs;
    float pe = p[i] * (1.f - a.lr * a.weight_decay);
    const float me = a.beta1 * m[i] + (1.f - a.beta1) * gr;
    const float ve = a.beta2 * v[i] + (1.f - a.beta2) * gr * gr;
    pe -= a.lr * (me * inv_bc1) / (sqrtf(ve) * inv_sqrt_bc2 + a.eps);
    p[i] = pe; m[i] = me; v[i] = ve;
    if (p_bf16) p_bf16[i] = __float2bfloat16_rn(pe);
  }
}

// ------------------------------------------------------------------ sum of squares (gradient norm), fp32 -> *out += sum
__global__ void __launch_bounds__(256) sumsq_kernel(const float* __restrict__ g, long long n, float* __restrict__ out) {
  __shared__ float red[32];
  float acc = 0.f;
  const long long nvec = n / 4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const float4 v = reinterpret_cast<const float4*>(g)[i];
    acc += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  for (long long i = nvec * 4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    acc += g[i] * g[i];
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

// ------------------------------------------------------------------ clipping a flat run of fp32 gradients
// Bound by HBM: one read for the norm, one read and write for the scaling.  The run may start at any element (a
// parameter's place in a flat buffer): up to three elements in front of the first 16-byte boundary are taken singly.
// Every thread keeps four 16-byte loads in flight.  Measured on 90 M elements: sum of squares 61 us = 5.9 TB/s (as abs, pow
// and sum, three kernels with fp32 tensors in between: 303 us), scaling 124 us = 5.8 TB/s (a broadcast multiplication: 220 us).
YF_DEVINL long long run_head(const float* p, long long n) {
  const long long h = (long long)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / 4;
  return h < n ? h : n;
}
// partials[blockIdx.x] = this block's share of sum(g^2): no atomics, so the sum of the partials does not vary from run to run
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const float* __restrict__ g, long long n, float* __restrict__ partials) {
  __shared__ float red[32];
  const long long head = run_head(g, n), nvec = (n - head) / 4, tail = head + nvec * 4;
  const float4* v = reinterpret_cast<const float4*>(g + head);
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  long long i = tid;
  for (; i + 3 * step < nvec; i += 4 * step) {
    const float4 a[4] = {v[i], v[i + step], v[i + 2 * step], v[i + 3 * step]};
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] += (a[j].x * a[j].x + a[j].y * a[j].y) + (a[j].z * a[j].z + a[j].w * a[j].w);
  }
  for (; i < nvec; i += step) acc[0] += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  if (tid < head) acc[1] += g[tid] * g[tid];
  if (tid < n - tail) acc[2] += g[tail + tid] * g[tail + tid];
  const float sum = block_sum<256>((acc[0] + acc[1]) + (acc[2] + acc[3]), red);
  if (threadIdx.x == 0) partials[blockIdx.x] = sum;
}
// x *= *coef; a coefficient of one (nothing to clip) leaves x as it is without touching it
__global__ void __launch_bounds__(256) scale_kernel(float* __restrict__ x, long long n, const float* __restrict__ coef) {
  const float c = *coef;
  if (c == 1.f) return;
  const long long head = run_head(x, n), nvec = (n - head) / 4, tail = head + nvec * 4;
  float4* v = reinterpret_cast<float4*>(x + head);
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  long long i = tid;
  for (; i + 3 * step < nvec; i += 4 * step) {
    float4 a[4] = {v[i], v[i + step], v[i + 2 * step], v[i + 3 * step]};
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i + j * step] = make_float4(a[j].x * c, a[j].y * c, a[j].z * c, a[j].w * c);
  }
  for (; i < nvec; i += step) v[i] = make_float4(v[i].x * c, v[i].y * c, v[i].z * c, v[i].w * c);
  if (tid < head) x[tid] *= c;
  if (tid < n - tail) x[tail + tid] *= c;
}

// clip coefficient from the total squared norm: coef = min(1, max_norm / (sqrt(total) + 1e-6)); norm_out = sqrt(total)
__global__ void clip_coef_kernel(const float* __restrict__ total_sq, float max_norm, float* __restrict__ coef,
                                 float* __restrict__ norm_out) {
  const float nrm = sqrtf(*total_sq);
  if (norm_out) *norm_out = nrm;
  *coef = fminf(1.f, max_norm / (nrm + 1e-6f));
}

// ------------------------------------------------------------------ flat casts / scale
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
  const long long nvec = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const float4 a = reinterpret_cast<const float4*>(src)[2 * i], b = reinterpret_cast<const float4*>(src)[2 * i + 1];
    uint4 o;
    o.x = pack_bf16x2(a.x, a.y);
    o.y = pack_bf16x2(a.z, a.w);
    o.z = pack_bf16x2(b.x, b.y);
    o.w = pack_bf16x2(b.z, b.w);
    reinterpret_cast<uint4*>(dst)[i] = o;
  }
  for (long long i = nvec * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}
// dst(fp32) = or += scale * src(bf16)
__global__ void accum_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, long long n,
                                         float scale, int accumulate) {
  const long long nvec = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float f[8];
    load8(src + i * 8, f);
    float4 a = make_float4(f[0] * scale, f[1] * scale, f[2] * scale, f[3] * scale);
    float4 b = make_float4(f[4] * scale, f[5] * scale, f[6] * scale, f[7] * scale);
    if (accumulate) {
      const float4 oa = reinterpret_cast<float4*>(dst)[2 * i], ob = reinterpret_cast<float4*>(dst)[2 * i + 1];
      a.x += oa.x; a.y += oa.y; a.z += oa.z; a.w += oa.w;
      b.x += ob.x; b.y += ob.y; b.z += ob.z; b.w += ob.w;
    }
    reinterpret_cast<float4*>(dst)[2 * i] = a;
    reinterpret_cast<float4*>(dst)[2 * i + 1] = b;
  }
  for (long long i = nvec * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float f = __bfloat162float(src[i]) * scale;
    dst[i] = accumulate ? dst[i] + f : f;
  }
}
// The same for many tensors in one launch (the gradients of a group's parameters, which autograd left in bf16, into their places
// of the flat fp32 gradient): blocks are dealt by chunks of 16384 elements.  A place may start anywhere: without 16-byte
// alignment on both sides a tensor's elements are taken singly.  90 M elements in four matrices and two vectors: 95 us =
// 5.6 TB/s, added to what is there 142 us = 6.3 TB/s (foreach copy and add: 151 and 317 us).
constexpr int MULTI_MAX = 48, MULTI_CHUNK = 16384;
struct MultiAccum {
  const __nv_bfloat16* src[MULTI_MAX];
  float* dst[MULTI_MAX];
  long long n[MULTI_MAX];
  int first_block[MULTI_MAX + 1];  // prefix sums of the tensors' chunks
  int count;
};
__global__ void __launch_bounds__(256) accum_bf16_to_f32_multi_kernel(const __grid_constant__ MultiAccum a, int accumulate) {
  int t = 0;
  while (t + 1 < a.count && (int)blockIdx.x >= a.first_block[t + 1]) ++t;
  const long long lo = (long long)((int)blockIdx.x - a.first_block[t]) * MULTI_CHUNK, hi = min(a.n[t], lo + MULTI_CHUNK);
  const __nv_bfloat16* src = a.src[t];
  float* dst = a.dst[t];
  long long done = lo;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
    const long long v1 = hi / 8;
#pragma unroll 4
    for (long long i = lo / 8 + threadIdx.x; i < v1; i += 256) {
      float f[8];
      load8(src + i * 8, f);
      float4* d = reinterpret_cast<float4*>(dst + i * 8);
      if (accumulate) {
        const float4 o = d[0], p = d[1];
        f[0] += o.x; f[1] += o.y; f[2] += o.z; f[3] += o.w;
        f[4] += p.x; f[5] += p.y; f[6] += p.z; f[7] += p.w;
      }
      d[0] = make_float4(f[0], f[1], f[2], f[3]);
      d[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    done = v1 * 8;
  }
  for (long long i = done + threadIdx.x; i < hi; i += 256) {
    const float f = __bfloat162float(src[i]);
    dst[i] = accumulate ? dst[i] + f : f;
  }
}
// y = a + b (bf16), used for residual joins in backward
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ y, long long n) {
  const long long nvec = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float x[8], z[8], o[8];
    load8(a + i * 8, x);
    load8(b + i * 8, z);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = x[j] + z[j];
    store8(y + i * 8, o);
  }
  for (long long i = nvec * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16_rn(__bfloat162float(a[i]) + __bfloat162float(b[i]));
}

inline int grid_for(long long work_items, int threads, int ctas_per_sm) {
  long long need = (work_items + threads - 1) / threads;
  long long cap = (long long)yf_num_sms() * ctas_per_sm;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

#define YF_STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define YF_LAUNCH_RET() return -(int)cudaGetLastError()

extern "C" int yf_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int T, int D, float eps, void* stream) {
  if (T <= 0 || D <= 0 || (D % 8) || !aligned16(x) || !aligned16(w) || !aligned16(y)) return -1;
  if (D <= 32 * 4 * 8 * RNW_NV) {  // G warps per row
    const __nv_bfloat16 *xp = (const __nv_bfloat16*)x, *wp = (const __nv_bfloat16*)w;
    __nv_bfloat16* yp = (__nv_bfloat16*)y;
    const int g = D <= 32 * 8 * RNW_NV ? 1 : (D <= 64 * 8 * RNW_NV ? 2 : 4);
    const int rows = RNW_WARPS / g, ctas = (T + rows - 1) / rows;
    if (g == 1) rmsnorm_fwd_warp_kernel<1><<<ctas, RNW_WARPS * 32, 0, YF_STREAM(stream)>>>(xp, wp, yp, rstd, T, D, eps);
    else if (g == 2) rmsnorm_fwd_warp_kernel<2><<<ctas, RNW_WARPS * 32, 0, YF_STREAM(stream)>>>(xp, wp, yp, rstd, T, D, eps);
    else rmsnorm_fwd_warp_kernel<4><<<ctas, RNW_WARPS * 32, 0, YF_STREAM(stream)>>>(xp, wp, yp, rstd, T, D, eps);
    YF_LAUNCH_RET();
  }
  const int grid = T < yf_num_sms() * 8 ? T : yf_num_sms() * 8;
  rmsnorm_fwd_kernel<<<grid, RN_THREADS, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                                                                 (__nv_bfloat16*)y, rstd, T, D, eps);
  YF_LAUNCH_RET();
}
static int rmsnorm_bwd_tpr(int D) { return D <= 1024 ? 32 : (D <= 2048 ? 64 : (D <= 4096 ? 128 : 256)); }
static int rmsnorm_bwd_ctas(int T, int D) {
  const int rows = RNB_THREADS / rmsnorm_bwd_tpr(D), need = (T + rows - 1) / rows, cap = 2 * yf_num_sms();
  return need < cap ? need : cap;
}
static bool rmsnorm_bwd_combines(int T, int D) {
  return (long long)rmsnorm_bwd_ctas(T, D) * (RNB_THREADS / rmsnorm_bwd_tpr(D)) * D * 4 > (2ll << 20);
}
// rows of yf_rmsnorm_bwd_ws's partials
extern "C" int yf_rmsnorm_bwd_partials(int T, int D) {
  if (T <= 0 || D <= 0 || (D % 8) || D > RNB_THREADS * 8 * RNB_NV) return -1;
  return rmsnorm_bwd_ctas(T, D) * (rmsnorm_bwd_combines(T, D) ? 1 : RNB_THREADS / rmsnorm_bwd_tpr(D));
}
extern "C" int yf_rmsnorm_bwd_ws(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx, float* dw,
                                 int zero_dw, float* partials, float* sumsq, int T, int D, void* stream) {
  if (T <= 0 || D <= 0 || (D % 8) || D > RNB_THREADS * 8 * RNB_NV) return -1;
  if (!aligned16(x) || !aligned16(w) || !aligned16(dy) || !aligned16(dx) || (dres && !aligned16(dres)) || (partials && !aligned16(partials))) return -1;
  if ((zero_dw || partials) && !dw) return -1;
  if (sumsq && !partials) return -1;
  cudaStream_t st = YF_STREAM(stream);
  if (zero_dw && !partials && cudaMemsetAsync(dw, 0, (size_t)D * sizeof(float), st) != cudaSuccess) return -2;
  const __nv_bfloat16 *xp = (const __nv_bfloat16*)x, *wp = (const __nv_bfloat16*)w, *dyp = (const __nv_bfloat16*)dy, *ep = (const __nv_bfloat16*)dres;
  __nv_bfloat16* dxp = (__nv_bfloat16*)dx;
  const int ctas = rmsnorm_bwd_ctas(T, D), combine = !partials || rmsnorm_bwd_combines(T, D) ? 1 : 0;
  if (D <= 1024) rmsnorm_bwd_kernel<32><<<ctas, RNB_THREADS, 0, st>>>(xp, wp, dyp, rstd, ep, dxp, partials, dw, T, D, combine);
  else if (D <= 2048) rmsnorm_bwd_kernel<64><<<ctas, RNB_THREADS, 0, st>>>(xp, wp, dyp, rstd, ep, dxp, partials, dw, T, D, combine);
  else if (D <= 4096) rmsnorm_bwd_kernel<128><<<ctas, RNB_THREADS, 0, st>>>(xp, wp, dyp, rstd, ep, dxp, partials, dw, T, D, combine);
  else rmsnorm_bwd_kernel<256><<<ctas, RNB_THREADS, 0, st>>>(xp, wp, dyp, rstd, ep, dxp, partials, dw, T, D, combine);
  if (partials) rmsnorm_bwd_dw_kernel<<<(D + 31) / 32, 1024, 0, st>>>(partials, dw, yf_rmsnorm_bwd_partials(T, D), D,
                                                                        zero_dw ? 0 : 1, sumsq);
  YF_LAUNCH_RET();
}
extern "C" int yf_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx,
                              float* dw, int zero_dw, int T, int D, void* stream) {
  return yf_rmsnorm_bwd_ws(x, w, dy, rstd, dres, dx, dw, zero_dw, nullptr, nullptr, T, D, stream);
}
extern "C" int yf_rope(void* qkv, const float* cos_sin, int T, int seq_len, long long row_stride, int col0, int n_heads,
                       int head_dim, int backward, void* stream) {
  if (T <= 0 || n_heads <= 0 || (head_dim % 16) || (row_stride % 8) || (col0 % 8) || !aligned16(qkv)) return -1;
  const long long items = (long long)T * n_heads * (head_dim / 16);
  rope_kernel<<<grid_for(items, 256, 8), 256, 0, YF_STREAM(stream)>>>((__nv_bfloat16*)qkv, cos_sin, T, seq_len, row_stride, col0,
                                                                       n_heads, head_dim, backward ? -1.f : 1.f);
  YF_LAUNCH_RET();
}
extern "C" int yf_swiglu_fwd(const void* gu, void* h, long long T, int F, void* stream) {
  if (T <= 0 || F <= 0 || (F % 8) || !aligned16(gu) || !aligned16(h)) return -1;
  swiglu_fwd_kernel<<<grid_for(T * (F / 8), 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)h, T, F);
  YF_LAUNCH_RET();
}
extern "C" int yf_swiglu_bwd(const void* gu, const void* dh, void* dgu, long long T, int F, void* stream) {
  if (T <= 0 || F <= 0 || (F % 8) || !aligned16(gu) || !aligned16(dh) || !aligned16(dgu)) return -1;
  swiglu_bwd_kernel<<<grid_for(T * (F / 8), 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)gu, (const __nv_bfloat16*)dh,
                                                                                   (__nv_bfloat16*)dgu, T, F);
  YF_LAUNCH_RET();
}
extern "C" int yf_cross_entropy(void* logits, const long long* labels, float* loss_rows, int T, int V, long long ldl,
                                float grad_scale, const float* scale_ptr, int write_grad, void* stream) {
  if (T <= 0 || V <= 0 || (ldl % 8) || !aligned16(logits)) return -1;
  // Registers let two CTAs reside on an SM; twice as many are launched, so that an SM that is done early takes more rows (1024 x
  // 128256: 116 us, with two per SM 128 us).  One per SM where the rows in flight of two would exceed 80 MB of the L2.
  const int per_sm = (long long)V * 2 * yf_num_sms() * 2 <= (80ll << 20) ? 4 : 1;
  const int grid = T < yf_num_sms() * per_sm ? T : yf_num_sms() * per_sm;
  cross_entropy_kernel<<<grid, CE_THREADS, 0, YF_STREAM(stream)>>>((__nv_bfloat16*)logits, labels, loss_rows, T, V, ldl, grad_scale,
                                                                   scale_ptr, write_grad);
  YF_LAUNCH_RET();
}
extern "C" int yf_inv_valid_labels(const long long* labels, long long n, float* out, void* stream) {
  if (n < 0 || n > 0x7fffffffll) return -1;
  inv_valid_labels_kernel<<<1, ONE_BLOCK, 0, YF_STREAM(stream)>>>(labels, n, out);
  YF_LAUNCH_RET();
}
extern "C" int yf_shift_labels(const long long* labels, long long* out, long long batch, int seq, long long ld, void* stream) {
  if (batch < 0 || seq <= 0) return -1;
  if (batch == 0) return 0;
  shift_labels_kernel<<<grid_for(batch * seq, 256, 4), 256, 0, YF_STREAM(stream)>>>(labels, out, batch * seq, seq, ld);
  YF_LAUNCH_RET();
}
extern "C" int yf_scaled_sum(const float* x, long long n, const float* scale, float* out, void* stream) {
  if (n < 0) return -1;
  scaled_sum_kernel<<<1, ONE_BLOCK, 0, YF_STREAM(stream)>>>(x, n, scale, out);
  YF_LAUNCH_RET();
}
extern "C" int yf_embedding_fwd(const void* table, const long long* ids, void* out, long long T, int D, int V, void* stream) {
  if (T <= 0 || (D % 8) || !aligned16(table) || !aligned16(out)) return -1;
  embedding_fwd_kernel<<<grid_for(T * (D / 8), 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)table, ids,
                                                                                      (__nv_bfloat16*)out, T, D, V);
  YF_LAUNCH_RET();
}
extern "C" int yf_embedding_bwd_norm(const void* dout, const long long* ids, float* dtable, int* owner, float* sumsq, long long T, int D, int V,
                                     void* stream) {
  if (T <= 0 || T > 0x7fffffffll || (D % 8) || !aligned16(dout) || (sumsq != nullptr && owner == nullptr)) return -1;
  embedding_bwd_kernel<<<grid_for(T * (D / 8), 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)dout, ids, dtable, owner, T, D, V,
                                                                                      aligned16(dtable) ? 1 : 0);
  if (sumsq != nullptr)
    embedding_sumsq_kernel<<<(int)(T < yf_num_sms() * 8 ? T : yf_num_sms() * 8), 256, 0, YF_STREAM(stream)>>>(dtable, ids, owner, sumsq, T, D, V);
  YF_LAUNCH_RET();
}
extern "C" int yf_embedding_bwd(const void* dout, const long long* ids, float* dtable, long long T, int D, int V, void* stream) {
  return yf_embedding_bwd_norm(dout, ids, dtable, nullptr, nullptr, T, D, V, stream);
}
extern "C" int yf_adamw(float* p, const float* g, float* m, float* v, void* p_bf16, const float* grad_scale_ptr, long long n,
                        float lr, float beta1, float beta2, float eps, float weight_decay, int step, int max_ctas, void* stream) {
  if (n <= 0) return 0;
  if (!aligned16(p) || !aligned16(g) || !aligned16(m) || !aligned16(v) || (p_bf16 && (reinterpret_cast<uintptr_t>(p_bf16) & 7)))
    return -1;
  AdamArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weight_decay = weight_decay;
  a.bc1 = 1.f - powf(beta1, (float)step);
  a.bc2 = 1.f - powf(beta2, (float)step);
  // max_ctas > 0 caps the grid: when the update runs beside GEMMs on another stream, three CTAs per SM leave the
  // thread slots and registers that a persistent GEMM CTA needs and still keep HBM saturated
  int grid = grid_for(n / 4 + 1, 256, 8);
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  adamw_kernel<<<grid, 256, 0, YF_STREAM(stream)>>>(p, g, m, v, (__nv_bfloat16*)p_bf16, grad_scale_ptr, n, a);
  YF_LAUNCH_RET();
}
extern "C" int yf_sumsq(const float* g, long long n, float* out, void* stream) {
  if (n <= 0) return 0;
  if (!aligned16(g)) return -1;
  sumsq_kernel<<<grid_for(n / 4 + 1, 256, 4), 256, 0, YF_STREAM(stream)>>>(g, n, out);
  YF_LAUNCH_RET();
}
// partials: n_partials floats, one per block of the launch (at most yf_sm_count() * 8); g: 4-byte aligned
extern "C" int yf_sumsq_partials(const float* g, long long n, float* partials, int n_partials, void* stream) {
  if (n <= 0 || n_partials < 1 || (reinterpret_cast<uintptr_t>(g) & 3)) return -1;
  sumsq_partial_kernel<<<n_partials, 256, 0, YF_STREAM(stream)>>>(g, n, partials);
  YF_LAUNCH_RET();
}
extern "C" int yf_scale(float* x, long long n, const float* coef, void* stream) {
  if (n <= 0) return 0;
  if (reinterpret_cast<uintptr_t>(x) & 3) return -1;
  scale_kernel<<<grid_for(n / 16 + 1, 256, 8), 256, 0, YF_STREAM(stream)>>>(x, n, coef);
  YF_LAUNCH_RET();
}
extern "C" int yf_clip_coef(const float* total_sq, float max_norm, float* coef, float* norm_out, void* stream) {
  clip_coef_kernel<<<1, 1, 0, YF_STREAM(stream)>>>(total_sq, max_norm, coef, norm_out);
  YF_LAUNCH_RET();
}
extern "C" int yf_cast_f32_to_bf16(const float* src, void* dst, long long n, void* stream) {
  if (n <= 0) return 0;
  if (!aligned16(src) || !aligned16(dst)) return -1;
  cast_f32_to_bf16_kernel<<<grid_for(n / 8 + 1, 256, 8), 256, 0, YF_STREAM(stream)>>>(src, (__nv_bfloat16*)dst, n);
  YF_LAUNCH_RET();
}
extern "C" int yf_accum_bf16_to_f32(const void* src, float* dst, long long n, float scale, int accumulate, void* stream) {
  if (n <= 0) return 0;
  if (!aligned16(src) || !aligned16(dst)) return -1;
  accum_bf16_to_f32_kernel<<<grid_for(n / 8 + 1, 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)src, dst, n, scale, accumulate);
  YF_LAUNCH_RET();
}
extern "C" int yf_accum_bf16_to_f32_multi(int count, const void* const* src, float* const* dst, const long long* n, int accumulate, void* stream) {
  if (count < 0) return -1;
  for (int i = 0; i < count; ++i)
    if (n[i] < 0 || (reinterpret_cast<uintptr_t>(src[i]) & 1) || (reinterpret_cast<uintptr_t>(dst[i]) & 3)) return -1;
  MultiAccum a;
  for (int i = 0; i < count;) {
    a.count = 0;
    long long blocks = 0;
    for (; i < count && a.count < MULTI_MAX; ++i) {
      const long long mine = (n[i] + MULTI_CHUNK - 1) / MULTI_CHUNK;
      if (mine == 0) continue;
      if (mine > 0x7fffffffll) return -1;
      if (blocks + mine > 0x7fffffffll) break;  // the next launch takes it
      a.src[a.count] = (const __nv_bfloat16*)src[i];
      a.dst[a.count] = dst[i];
      a.n[a.count] = n[i];
      a.first_block[a.count++] = (int)blocks;
      blocks += mine;
    }
    a.first_block[a.count] = (int)blocks;
    if (blocks > 0) accum_bf16_to_f32_multi_kernel<<<(int)blocks, 256, 0, YF_STREAM(stream)>>>(a, accumulate);
  }
  YF_LAUNCH_RET();
}
extern "C" int yf_add_bf16(const void* a, const void* b, void* y, long long n, void* stream) {
  if (n <= 0) return 0;
  if (!aligned16(a) || !aligned16(b) || !aligned16(y)) return -1;
  add_bf16_kernel<<<grid_for(n / 8 + 1, 256, 8), 256, 0, YF_STREAM(stream)>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                                               (__nv_bfloat16*)y, n);
  YF_LAUNCH_RET();
}
