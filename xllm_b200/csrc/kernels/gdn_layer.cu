// Gated delta net layer between its projections, bf16 (Qwen3-Next / Qwen3.5): from the projection rows as the GEMMs left
// them to the rows of the output projection, decode rows and prompt portions of a batch alike.
//
//   q, k, v through a short causal convolution and silu; q, k unit vectors per head (q scaled); heads / key heads
//   neighbours share q and k;  g = -exp(A_log) softplus(a + dt_bias),  beta = sigmoid(b), one of each per head
//   S <- exp(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q            S [dk, dv] fp32, one per state slot
//   row <- w o / rms(o) silu(z)
//
//   gdn_conv_kernel   convolution -> bf16 rows, 1 / |q| and 1 / |k|, decays and betas
//   gdn_step_kernel   one token per sequence, from there to the finished row; the state crosses HBM once in each direction
//   gdn_scan_kernel   prompts: all sequences and heads at once, token by token in fp32 with the state in registers; the last
//                     inputs of a sequence -> its convolution tail
//   gdn_norm_kernel   prompts: norm, weight and gate
//
// Measured against the same layer as tensor operations around gdn.cu (one B200, 32 heads of 128 x 128, four prompts of up to
// 1024 tokens one after the other: 3.6 ms a layer; 64 decode rows: 0.55 ms), whose time went to some fifty launches of
// elementwise kernels, the prompts one by one, and two barriers per token in the recurrence.
//
// A sequence whose rows in the batch are its first tokens (kv_len == number of rows) starts from zeros whatever its slot
// holds; slot < 0 marks padding rows, which come out as zeros.  Built without fast-math: errors of a decay multiply up.
#include "recurrence.cuh"
#include "short_conv.cuh"

namespace xllm {

constexpr float kGdnUnitEps = 1e-6f;

struct GdnParams {
  float* state;               // [slots, H, dk, dv]
  bf16* tail;                 // [slots, C, taps - 1], C = 2 G dk + H dv channels: q | k | v, oldest input first
  const int32_t *slots, *cu_q, *kv_lens;
  const bf16 *q, *k, *v, *z;  // head 0's place in row 0 of the projection rows
  int64_t ld, z_ld;           // row strides of q, k, v and of z
  int qk_hs, v_gs, z_gs;      // strides of q and k heads, and of the v and z blocks of a key head's value heads
  const bf16 *b, *a;          // pre-sigmoid beta and pre-softplus decay of head 0
  int64_t ba_ld;
  int ba_gs;                  // stride of the blocks of a key head's value heads
  const bf16 *conv_w;         // [C, taps], the last tap is the current token's
  const bf16 *dt_bias, *a_log, *norm_w;
  bf16 *yq, *yk, *yv;         // [rows, G, dk], [rows, G, dk], [rows, H, dv]
  float *fq, *fk;             // [rows, G]: factors that make yq, yk unit vectors (yq: scaled)
  float2* gb;                 // [rows, H]: exp(g), beta
  float* o;                   // [rows, H, dv] (prompts)
  bf16* out;                  // [rows, H dv]
  int n_decode, n_seqs, rows, H, G, dk, dv, taps;
  float q_scale, eps;
  __host__ __device__ int64_t channels() const { return (int64_t)2 * G * dk + (int64_t)H * dv; }
};

// One warp per (run of rows, item): the heads of q | k | v, then one item for the decays and betas.  A lane owns four
// neighbouring channels (dk, dv <= 128) and keeps the last inputs in registers, so that every input is read once.
template <int RUN, int K1>
__global__ void __launch_bounds__(256) gdn_conv_kernel(GdnParams p) {
  const int lane = threadIdx.x & 31, items = 2 * p.G + p.H + 1;
  const unsigned it = blockIdx.x * 8 + (threadIdx.x >> 5), run = it / items;
  pdl_wait();
  pdl_launch_dependents();
  const int first = (int)run * RUN;
  if (first >= p.rows) return;
  int h = (int)(it - run * items);
  const int r = p.H / p.G;
  if (h == items - 1) {
    for (int row = first; row < min(first + RUN, p.rows); ++row)
      for (int n = lane; n < p.H; n += 32) {
        const int64_t at = row * p.ba_ld + (int64_t)(n / r) * p.ba_gs + n % r;
        const float x = __bfloat162float(p.a[at]) + __bfloat162float(p.dt_bias[n]);
        const float sp = x > 20.f ? x : log1pf(expf(x));
        p.gb[(int64_t)row * p.H + n] = make_float2(expf(-expf(__bfloat162float(p.a_log[n])) * sp), sigmoid_exact(__bfloat162float(p.b[at])));
      }
    return;
  }
  const int part = h < p.G ? 0 : (h < 2 * p.G ? 1 : 2);
  h -= part == 0 ? 0 : (part == 1 ? p.G : 2 * p.G);
  const int d = part == 2 ? p.dv : p.dk, c = lane * 4;
  const bool on = c < d;
  const int64_t ch = (part == 2 ? (int64_t)2 * p.G * p.dk : (int64_t)part * p.G * p.dk) + (int64_t)h * d + c, C = p.channels();
  const bf16* x = (part == 2 ? p.v + (int64_t)(h / r) * p.v_gs + (h % r) * d : (part == 0 ? p.q : p.k) + (int64_t)h * p.qk_hs) + c;
  bf16* y = (part == 0 ? p.yq : (part == 1 ? p.yk : p.yv)) + (int64_t)h * d + c;
  const int64_t y_ld = (int64_t)(part == 2 ? p.H : p.G) * d;
  float v[RUN + 3][4], w[4][4];                                     // w[taps back][channel]
#pragma unroll
  for (int i = 0; i < RUN + 3; ++i) {
    const int row = first + i - 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
    if (on && row >= 0 && row < p.rows) load_f32<4>(x + row * p.ld, v[i]);
  }
  // four channels of TAPS weights, or of K1 inputs in the tail, are neighbours: eight bytes at a time
  __align__(8) bf16 wr[4 * (K1 + 1)];
#pragma unroll
  for (int i = 0; i < K1 + 1; ++i)
    *reinterpret_cast<uint2*>(wr + 4 * i) = on ? reinterpret_cast<const uint2*>(p.conv_w + ch * (K1 + 1))[i] : make_uint2(0u, 0u);
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) w[t][j] = t <= K1 ? __bfloat162float(wr[j * (K1 + 1) + (t <= K1 ? K1 - t : 0)]) : 0.f;
  int b = -1, begin = 0, end = 0, slot = -1, len = 0;
#pragma unroll
  for (int i = 0; i < RUN; ++i) {
    const int row = first + i;
    if (row >= p.rows) break;
    if (row >= end) {                                               // the row starts another sequence, or is the first
      b = seq_of_row(p.cu_q, p.n_seqs, row);
      begin = b < 0 ? row : p.cu_q[b];
      end = b < 0 ? row + 1 : p.cu_q[b + 1];
      slot = b < 0 ? -1 : p.slots[b];
      len = b < 0 ? 0 : p.kv_lens[b];
    }
    if (slot < 0) continue;
    const int back = row - begin, n = end - begin;
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = v[i + 3][j] * w[0][j];
      if (back >= 1) s[j] += v[i + 2][j] * w[1][j];
      if (back >= 2) s[j] += v[i + 1][j] * w[2][j];
      if (back >= 3) s[j] += v[i][j] * w[3][j];
    }
    bf16* tail = p.tail + ((int64_t)slot * C + ch) * K1;            // [channel][input], oldest first
    if (back < K1 && on) {
      __align__(8) bf16 past[4 * K1];
      const bool old = len > n;                                     // the slot's tail belongs to this sequence
#pragma unroll
      for (int i = 0; i < K1; ++i)
        *reinterpret_cast<uint2*>(past + 4 * i) = old ? reinterpret_cast<const uint2*>(tail)[i] : make_uint2(0u, 0u);
#pragma unroll
      for (int u = 0; u < K1; ++u) {                                // u + 1 inputs before the sequence's rows
        const int t = u + 1 + back;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[j] += __bfloat162float(past[j * K1 + K1 - 1 - u]) * (t == 1 ? w[1][j] : (t == 2 ? w[2][j] : (t == 3 ? w[3][j] : 0.f)));
      }
      if (n == 1) {                                                 // this lane alone reads these inputs: move them up
        __align__(8) bf16 now[4 * K1];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int t = 0; t < K1; ++t) now[j * K1 + t] = t + 1 < K1 ? past[j * K1 + t + 1] : __float2bfloat16(v[i + 3][j]);
#pragma unroll
        for (int i2 = 0; i2 < K1; ++i2) reinterpret_cast<uint2*>(tail)[i2] = *reinterpret_cast<const uint2*>(now + 4 * i2);
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = on ? __bfloat162float(__float2bfloat16(s[j] * sigmoid_exact(s[j]))) : 0.f;
      ss += s[j] * s[j];
    }
    if (part < 2) {
      ss = warp_sum(ss);
      if (lane == 0) (part == 0 ? p.fq : p.fk)[(int64_t)row * p.G + h] = (part == 0 ? p.q_scale : 1.f) / sqrtf(ss + kGdnUnitEps);
    }
    if (on) store_f32<4>(y + row * y_ld, s);
  }
}

// silu(z) times the normed and weighted output, in the model's order of roundings
__device__ __forceinline__ bf16 gdn_finish(float o, float inv, bf16 w, float z) {
  const bf16 n = __float2bfloat16(o * inv);
  return __float2bfloat16(__bfloat162float(__float2bfloat16(__bfloat162float(w) * __bfloat162float(n))) * (z * sigmoid_exact(z)));
}

// ------------------------------------------------------------------------------------------------ decode
// grid (heads, sequences), 256 threads: dv / 4 column groups x row groups, NR rows of four columns per thread, all of whose
// loads are in flight together, in front of the wait for the convolution (a kernel that only starts when everything ahead of
// the convolution is done, and that writes no state).
template <int NR>
__global__ void __launch_bounds__(256, 2) gdn_step_kernel(GdnParams p) {
  __shared__ float qs[128], ks[128], vs[128], red32[32];
  __shared__ __align__(16) float red[256 * 4];                     // [row groups][dv]
  const int dk = p.dk, dv = p.dv, h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int CG = dv >> 2, RG = 256 / CG, cg = tid % CG, rg = tid / CG;
  const int slot = p.slots[b], len = p.kv_lens[b];
  const bool live = slot >= 0 && len > 0, active = rg < RG, fresh = len == 1;
  float* S = p.state + (((int64_t)max(slot, 0) * p.H + h) * dk) * dv + cg * 4;
  float4 s[NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) {
    const int i = rg + u * RG;
    s[u] = (live && active && !fresh && i < dk) ? *reinterpret_cast<const float4*>(S + i * dv) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  pdl_wait();
  pdl_launch_dependents();
  bf16* orow = p.out + ((int64_t)b * p.H + h) * dv;
  if (!live) {
    for (int i = tid; i < dv; i += 256) orow[i] = __float2bfloat16(0.f);
    return;
  }
  const int r = p.H / p.G;
  const int64_t qk = (int64_t)b * p.G + h / r, row = (int64_t)b * p.H + h;
  if (tid < dk) {
    qs[tid] = __bfloat162float(p.yq[qk * dk + tid]) * p.fq[qk];
    ks[tid] = __bfloat162float(p.yk[qk * dk + tid]) * p.fk[qk];
  }
  if (tid >= 128 && tid - 128 < dv) vs[tid - 128] = __bfloat162float(p.yv[row * dv + tid - 128]);
  const float2 gb = p.gb[row];
  const float z = tid < dv ? __bfloat162float(p.z[b * p.z_ld + (int64_t)(h / r) * p.z_gs + (h % r) * dv + tid]) : 0.f;
  const bf16 w_out = tid < dv ? p.norm_w[tid] : __float2bfloat16(0.f);
  __syncthreads();
  float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
  if (active) {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const int i = rg + u * RG;
      if (i >= dk) break;
      const float kk = ks[i];
      d.x += s[u].x * kk; d.y += s[u].y * kk; d.z += s[u].z * kk; d.w += s[u].w * kk;
    }
    *reinterpret_cast<float4*>(red + rg * dv + cg * 4) = d;
  }
  __syncthreads();
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (active) {
    d = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 0; i < RG; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(red + i * dv + cg * 4);
      d.x += x.x; d.y += x.y; d.z += x.z; d.w += x.w;
    }
    const float* v4 = vs + cg * 4;
    const float4 e = make_float4(gb.y * (v4[0] - gb.x * d.x), gb.y * (v4[1] - gb.x * d.y), gb.y * (v4[2] - gb.x * d.z),
                                 gb.y * (v4[3] - gb.x * d.w));
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const int i = rg + u * RG;
      if (i >= dk) break;
      const float kk = ks[i], qq = qs[i];
      float4 x = s[u];
      x.x = x.x * gb.x + kk * e.x; x.y = x.y * gb.x + kk * e.y; x.z = x.z * gb.x + kk * e.z; x.w = x.w * gb.x + kk * e.w;
      *reinterpret_cast<float4*>(S + i * dv) = x;
      o.x += qq * x.x; o.y += qq * x.y; o.z += qq * x.z; o.w += qq * x.w;
    }
  }
  __syncthreads();
  if (active) *reinterpret_cast<float4*>(red + rg * dv + cg * 4) = o;
  __syncthreads();
  float mine = 0.f;
  if (tid < dv)
    for (int i = 0; i < RG; ++i) mine += red[i * dv + tid];
  const float inv = 1.f / sqrtf(block_sum(mine * mine, red32) / (float)dv + p.eps);
  if (tid < dv) orow[tid] = gdn_finish(mine, inv, w_out, z);
}

// ------------------------------------------------------------------------------------------------ prompts: recurrence
// grid (slices of 32 columns, heads, sequences), four warps of eight columns (recurrence.cuh).  A token costs one pass over
// the state for S^T k, one that adds k u^T and takes S^T q, and no barrier.  The decay is no pass of its own: the registers
// hold S / c with c the product of the decays since it was last multiplied in, which happens before it falls below 2^-40.
// The next tile's vectors are on their way while one is worked on and meet their factors on the way into shared memory.
constexpr int kGdnWarps = 4, kGdnCols = kGdnWarps * kRecCols;

template <int J>
__global__ void __launch_bounds__(32 * kGdnWarps, 4) gdn_scan_kernel(GdnParams p) {
  constexpr int DK = 32 * J, TT = kRecTile, NT = 32 * kGdnWarps;
  __shared__ __align__(16) float ksm[2][TT][DK], qsm[2][TT][DK], vsm[2][TT][kGdnCols];
  __shared__ float2 gsm[2][TT];
  const int h = blockIdx.y, b = p.n_decode + blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rgrp = lane & 7, c0 = blockIdx.x * kGdnCols, lc = warp * kRecCols + (lane >> 3) * 2, col = c0 + lc;
  const int r = p.H / p.G, g = h / r, dk = p.dk, dv = p.dv;
  pdl_wait();
  pdl_launch_dependents();
  const int row0 = p.cu_q[b], n = p.cu_q[b + 1] - row0, slot = p.slots[b];
  if (n <= 0 || slot < 0) return;
  const bool fresh = p.kv_lens[b] == n, mine = col < dv;
  float* S = p.state + (((int64_t)slot * p.H + h) * dk) * dv + col;
  StateColumns<J> st;
  st.load(S, dk, dv, rgrp, mine && !fresh);
  if (blockIdx.x == 0 && n > 1) {                                   // the convolution has read the tails
    const int K1 = p.taps - 1;
    const int64_t C = p.channels();
    const bool qk = h % r == 0;
    for (int i = tid; i < dv + (qk ? 2 * dk : 0); i += NT) {
      const int part = i < dv ? 2 : (i < dv + dk ? 0 : 1), c = i - (part == 2 ? 0 : (part == 0 ? dv : dv + dk));
      const bf16* x = part == 2 ? p.v + (int64_t)g * p.v_gs + (h % r) * dv : (part == 0 ? p.q : p.k) + (int64_t)g * p.qk_hs;
      const int64_t ch = part == 2 ? (int64_t)2 * p.G * dk + (int64_t)h * dv + c : ((int64_t)part * p.G + g) * dk + c;
      bf16* tail = p.tail + ((int64_t)slot * C + ch) * K1;
      bf16 keep[3];
      for (int t = 0; t < K1; ++t) {                                // input t of the new tail, of tail | rows
        const int at = n - K1 + t;
        keep[t] = at >= 0 ? x[(row0 + at) * p.ld + c] : (fresh ? __float2bfloat16(0.f) : tail[n + t]);
      }
      for (int t = 0; t < K1; ++t) tail[t] = keep[t];
    }
  }
  for (int i = tid; i < 2 * TT * DK; i += NT) (&ksm[0][0][0])[i] = (&qsm[0][0][0])[i] = 0.f;      // zeros behind dk
  for (int i = tid; i < 2 * TT * kGdnCols; i += NT) (&vsm[0][0][0])[i] = 0.f;                     // and behind dv
  __syncthreads();
  // a thread's share of a tile: four values of q and k (FQ times), four of v, the decay and beta of one token
  constexpr int FQ = TT * DK / 4 / NT;
  uint2 qr[FQ], kr[FQ], vr;
  float qf[FQ], kf_[FQ];
  float2 gr = make_float2(1.f, 0.f);
  const int vt = tid / (kGdnCols / 4), vc = (tid % (kGdnCols / 4)) * 4;
  static_assert(TT * kGdnCols / 4 == NT, "one v load per thread");
  const auto fetch = [&](int t0) {
    const int m = min(TT, n - t0);
#pragma unroll
    for (int i = 0; i < FQ; ++i) {
      const int e = tid + i * NT, t = e / (DK / 4), c = (e % (DK / 4)) * 4;
      if (t < m && c < dk) {
        const int64_t at = (int64_t)(row0 + t0 + t) * p.G + g;
        qr[i] = *reinterpret_cast<const uint2*>(p.yq + at * dk + c);
        kr[i] = *reinterpret_cast<const uint2*>(p.yk + at * dk + c);
        qf[i] = p.fq[at];
        kf_[i] = p.fk[at];
      }
    }
    if (vt < m && c0 + vc < dv) vr = *reinterpret_cast<const uint2*>(p.yv + ((int64_t)(row0 + t0 + vt) * p.H + h) * dv + c0 + vc);
    if (tid < m) gr = p.gb[(int64_t)(row0 + t0 + tid) * p.H + h];
  };
  const auto widen = [](uint2 u, float f) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&u.y));
    return make_float4(a.x * f, a.y * f, b.x * f, b.y * f);
  };
  const auto put = [&](int t0, int buf) {
    const int m = min(TT, n - t0);
#pragma unroll
    for (int i = 0; i < FQ; ++i) {
      const int e = tid + i * NT, t = e / (DK / 4), c = (e % (DK / 4)) * 4;
      if (t < m && c < dk) {
        *reinterpret_cast<float4*>(&qsm[buf][t][c]) = widen(qr[i], qf[i]);
        *reinterpret_cast<float4*>(&ksm[buf][t][c]) = widen(kr[i], kf_[i]);
      }
    }
    if (vt < m && c0 + vc < dv) *reinterpret_cast<float4*>(&vsm[buf][vt][vc]) = widen(vr, 1.f);
    if (tid < m) gsm[buf][tid] = gr;
  };
  fetch(0);
  put(0, 0);
  __syncthreads();
  int buf = 0;
  float c = 1.f;
  for (int t0 = 0; t0 < n; t0 += TT, buf ^= 1) {
    const bool more = t0 + TT < n;
    if (more) fetch(t0 + TT);
    const int m = min(TT, n - t0);
    float* orow = p.o + ((int64_t)(row0 + t0) * p.H + h) * dv + col + (lane & 1);
    const bool writes = rgrp < 2 && col + (lane & 1) < dv;
#pragma unroll 2
    for (int t = 0; t < m; ++t) {
      const float2 gb = gsm[buf][t];
      c *= gb.x;
      if (c < 0x1p-40f) {                                           // uniform over the block
        const f2 cc = pack_f2(c, c);
#pragma unroll
        for (int j = 0; j < 2 * J; ++j) {
          st.s[0][j] = mul_f2(st.s[0][j], cc);
          st.s[1][j] = mul_f2(st.s[1][j], cc);
        }
        c = 1.f;
      }
      const float bc = gb.y / c;
      f2 kf[2 * J], qv[2 * J];
      load_rows<J>(&ksm[buf][t][0], rgrp, kf);
      f2 d0 = 0, d1 = 0, e0 = 0, e1 = 0;                            // packed zeros
#pragma unroll
      for (int j = 0; j < 2 * J; j += 2) {
        d0 = fma_f2(st.s[0][j], kf[j], d0);
        d1 = fma_f2(st.s[1][j], kf[j], d1);
        e0 = fma_f2(st.s[0][j + 1], kf[j + 1], e0);
        e1 = fma_f2(st.s[1][j + 1], kf[j + 1], e1);
      }
      const float2 a0 = unpack_f2(add_f2(d0, e0)), a1 = unpack_f2(add_f2(d1, e1));
      const float k0 = sum_row_groups(a0.x + a0.y), k1 = sum_row_groups(a1.x + a1.y);
      const float2 v = *reinterpret_cast<const float2*>(&vsm[buf][t][lc]);
      const float u0 = bc * (v.x - c * k0), u1 = bc * (v.y - c * k1);
      const f2 w0 = pack_f2(u0, u0), w1 = pack_f2(u1, u1);
      load_rows<J>(&qsm[buf][t][0], rgrp, qv);
      d0 = d1 = e0 = e1 = 0;
#pragma unroll
      for (int j = 0; j < 2 * J; j += 2) {
        st.s[0][j] = fma_f2(kf[j], w0, st.s[0][j]);
        st.s[1][j] = fma_f2(kf[j], w1, st.s[1][j]);
        st.s[0][j + 1] = fma_f2(kf[j + 1], w0, st.s[0][j + 1]);
        st.s[1][j + 1] = fma_f2(kf[j + 1], w1, st.s[1][j + 1]);
        d0 = fma_f2(st.s[0][j], qv[j], d0);
        d1 = fma_f2(st.s[1][j], qv[j], d1);
        e0 = fma_f2(st.s[0][j + 1], qv[j + 1], e0);
        e1 = fma_f2(st.s[1][j + 1], qv[j + 1], e1);
      }
      const float2 y0 = unpack_f2(add_f2(d0, e0)), y1 = unpack_f2(add_f2(d1, e1));
      const float y = c * sum_row_groups_2(y0.x + y0.y, y1.x + y1.y);
      if (writes) orow[(int64_t)t * p.H * dv] = y;
    }
    if (more) put(t0 + TT, buf ^ 1);             // that buffer was last read before the barrier at the end of the last tile
    __syncthreads();
  }
  const f2 cc = pack_f2(c, c);
#pragma unroll
  for (int j = 0; j < 2 * J; ++j) {
    st.s[0][j] = mul_f2(st.s[0][j], cc);
    st.s[1][j] = mul_f2(st.s[1][j], cc);
  }
  if (mine) st.store(S, dk, dv, rgrp);
}

// one warp per (row, head); a lane owns four neighbouring channels
__global__ void __launch_bounds__(256) gdn_norm_kernel(GdnParams p) {
  const int lane = threadIdx.x & 31, c = lane * 4;
  const int64_t it = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  pdl_wait();
  pdl_launch_dependents();
  const int row = p.n_decode + (int)(it / p.H), h = (int)(it % p.H), r = p.H / p.G;
  if (row >= p.rows) return;
  const int b = seq_of_row(p.cu_q, p.n_seqs, row);
  const bool live = b >= 0 && p.slots[b] >= 0, on = c < p.dv;
  float o[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
  if (live && on) {
    load_f32<4>(p.o + ((int64_t)row * p.H + h) * p.dv + c, o);
    load_f32<4>(p.z + row * p.z_ld + (int64_t)(h / r) * p.z_gs + (h % r) * p.dv + c, z);
  }
  const float ss = warp_sum(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]);
  const float inv = 1.f / sqrtf(ss / (float)p.dv + p.eps);
  if (!on) return;
  __align__(8) bf16 y[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) y[j] = live ? gdn_finish(o[j], inv, p.norm_w[c + j], z[j]) : __float2bfloat16(0.f);
  *reinterpret_cast<uint2*>(p.out + ((int64_t)row * p.H + h) * p.dv + c) = *reinterpret_cast<const uint2*>(y);
}

// out[t, h, i] *= sigmoid(gate[t * ld + h * hs + i]) in bf16, the gate of gated attention beside its query in the
// projection rows; eight elements a thread.
__global__ void __launch_bounds__(256) sigmoid_gate_kernel(bf16* __restrict__ out, const bf16* __restrict__ gate, int64_t ld,
                                                           int hs, int64_t n8, int heads, int d8) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n8) return;
  const int64_t th = i / d8, t = th / heads;
  const int e = (int)(i - th * d8), h = (int)(th - t * heads);
  float x[8], g[8];
  load_f32<8>(out + i * 8, x);
  load_f32<8>(gate + t * ld + (int64_t)h * hs + e * 8, g);
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] *= __bfloat162float(__float2bfloat16(sigmoid_as<bf16>(g[j])));
  store_f32<8>(out + i * 8, x);
}

}  // namespace xllm

XLLM_API int xllm_sigmoid_gate(void* out, const void* gate, int64_t ld, int hs, int64_t rows, int heads, int d, void* stream) {
  using namespace xllm;
  if (rows <= 0) return 0;
  if (heads <= 0 || d <= 0 || d % 8 != 0 || ld % 8 != 0 || hs % 8 != 0 || (((uintptr_t)out | (uintptr_t)gate) & 15) != 0)
    return (int)cudaErrorInvalidValue;
  const int64_t n8 = rows * heads * (d / 8);
  launch_pdl(sigmoid_gate_kernel, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, (bf16*)out,
             (const bf16*)gate, ld, hs, n8, heads, d / 8);
  return XLLM_LAUNCH_CHECK();
}

// Sequences 0 .. n_decode - 1 have one row each (rows 0 .. n_decode - 1), the others any number of rows behind them.
// dk, dv <= 128 and multiples of 4, taps 2 .. 4, all rows and heads 8-byte aligned.  Scratch: yq, yk [rows, G, dk],
// yv [rows, H, dv] bf16; fq, fk [rows, G], gb [rows, H, 2] fp32; o [rows, H, dv] fp32 where there are prompts.
XLLM_API int xllm_gdn_layer(void* state, void* tail, const void* slots, const void* cu_q, const void* kv_lens, const void* q,
                            const void* k, const void* v, const void* z, int64_t ld, int64_t z_ld, int qk_hs, int v_gs, int z_gs,
                            const void* b, const void* a, int64_t ba_ld, int ba_gs, const void* conv_w, const void* dt_bias,
                            const void* a_log, const void* norm_w, void* yq, void* yk, void* yv, void* fq, void* fk, void* gb,
                            void* o, void* out, int n_decode, int n_seqs, int rows, int H, int G, int dk, int dv, int taps,
                            float q_scale, float eps, void* stream) {
  using namespace xllm;
  if (rows <= 0 || n_seqs <= 0) return 0;
  const auto al8 = [](const void* x) { return (((uintptr_t)x) & 7) == 0; };
  if (H <= 0 || G <= 0 || H % G != 0 || dk <= 0 || dk > 128 || dk % 4 != 0 || dv <= 0 || dv > 128 || dv % 4 != 0 || taps < 2 ||
      taps > 4 || n_decode > rows || n_decode > n_seqs || ld % 4 != 0 || z_ld % 4 != 0 || qk_hs % 4 != 0 || v_gs % 4 != 0 ||
      z_gs % 4 != 0 || !al8(q) || !al8(k) || !al8(v) || !al8(z) || !al8(out) || !al8(yq) || !al8(yk) || !al8(yv) || !al8(tail) || !al8(conv_w) ||
      (((uintptr_t)state) & 15) != 0)
    return (int)cudaErrorInvalidValue;
  GdnParams p;
  p.state = (float*)state; p.tail = (bf16*)tail; p.slots = (const int32_t*)slots; p.cu_q = (const int32_t*)cu_q;
  p.kv_lens = (const int32_t*)kv_lens; p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.z = (const bf16*)z;
  p.ld = ld; p.z_ld = z_ld; p.qk_hs = qk_hs; p.v_gs = v_gs; p.z_gs = z_gs; p.b = (const bf16*)b; p.a = (const bf16*)a;
  p.ba_ld = ba_ld; p.ba_gs = ba_gs; p.conv_w = (const bf16*)conv_w; p.dt_bias = (const bf16*)dt_bias;
  p.a_log = (const bf16*)a_log; p.norm_w = (const bf16*)norm_w; p.yq = (bf16*)yq; p.yk = (bf16*)yk; p.yv = (bf16*)yv;
  p.fq = (float*)fq; p.fk = (float*)fk; p.gb = (float2*)gb; p.o = (float*)o; p.out = (bf16*)out;
  p.n_decode = n_decode; p.n_seqs = n_seqs; p.rows = rows; p.H = H; p.G = G; p.dk = dk; p.dv = dv; p.taps = taps;
  p.q_scale = q_scale; p.eps = eps;
  cudaStream_t s = (cudaStream_t)stream;
  // runs of four rows read an input once instead of four times; few rows need the warps more than the reuse
  const int items = 2 * G + H + 1, run = rows > 128 ? 4 : 1;
  const dim3 grid((unsigned)((((int64_t)rows + run - 1) / run * items + 7) / 8));
  const auto conv = [&](auto kernel) { launch_pdl(kernel, grid, dim3(256), 0, s, p); };
  if (taps == 4) conv(run == 4 ? gdn_conv_kernel<4, 3> : gdn_conv_kernel<1, 3>);
  else if (taps == 3) conv(run == 4 ? gdn_conv_kernel<4, 2> : gdn_conv_kernel<1, 2>);
  else conv(run == 4 ? gdn_conv_kernel<4, 1> : gdn_conv_kernel<1, 1>);
  int rc = XLLM_LAUNCH_CHECK();
  if (rc != 0) return rc;
  if (n_seqs > n_decode) {
    const dim3 sg((dv + kGdnCols - 1) / kGdnCols, H, n_seqs - n_decode), sb(32 * kGdnWarps);
    if (dk <= 32) launch_pdl(gdn_scan_kernel<1>, sg, sb, 0, s, p);
    else if (dk <= 64) launch_pdl(gdn_scan_kernel<2>, sg, sb, 0, s, p);
    else launch_pdl(gdn_scan_kernel<4>, sg, sb, 0, s, p);
    if ((rc = XLLM_LAUNCH_CHECK()) != 0) return rc;
  }
  if (n_decode > 0) {
    const int RG = 256 / (dv >> 2), nr = (dk + RG - 1) / RG;
    const dim3 grid(H, n_decode), block(256);
    if (nr <= 4) launch_pdl(gdn_step_kernel<4>, grid, block, 0, s, p);
    else if (nr <= 8) launch_pdl(gdn_step_kernel<8>, grid, block, 0, s, p);
    else launch_pdl(gdn_step_kernel<16>, grid, block, 0, s, p);
    if ((rc = XLLM_LAUNCH_CHECK()) != 0) return rc;
  }
  if (rows > n_decode && n_seqs > n_decode) {
    launch_pdl(gdn_norm_kernel, dim3((unsigned)(((int64_t)(rows - n_decode) * H + 7) / 8)), dim3(256), 0, s, p);
    rc = XLLM_LAUNCH_CHECK();
  }
  return rc;
}
