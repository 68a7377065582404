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
//   gdn_prep_kernel,  prompts: all sequences and heads at once, sixteen tokens at a time on the tensor cores (below); the last
//   gdn_chunk_kernel  inputs of a sequence -> its convolution tail
//   gdn_norm_kernel   prompts: norm, weight and gate
//
// Measured against the same layer as tensor operations around gdn.cu (one B200, 32 heads of 128 x 128, four prompts of up to
// 1024 tokens one after the other: 3.6 ms a layer; 64 decode rows: 0.55 ms), whose time went to some fifty launches of
// elementwise kernels, the prompts one by one, and two barriers per token in the recurrence.  Now 0.31 ms (convolution 60 us,
// chunks 20 and 198 us, norm 34 us) and 0.06 ms, of which the step takes 48 us (states: 268 MB, 41 us at the copy rate).
//
// A sequence whose rows in the batch are its first tokens (kv_len == number of rows) starts from zeros whatever its slot
// holds; slot < 0 marks padding rows, which come out as zeros.  Built without fast-math: errors of a decay multiply up.
#include "attn_common.cuh"
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
  bf16 *yq, *yk, *yv;         // [rows, G, dkp], [rows, G, dkp], [rows, H, dvp]; dkp: 64 or 128, zeros behind dk; dvp: dv in eights
  float *fq, *fk;             // [rows, G]: factors that make yq, yk unit vectors (yq: scaled)
  float2* gb;                 // [rows, H]: exp(g) (decode rows) or g, and beta
  uint8_t* blobs;             // prompts: see GdnBlob
  float* o;                   // [rows, H, dv] (prompts)
  bf16* out;                  // [rows, H dv]
  int n_decode, n_seqs, rows, H, G, dk, dv, dkp, dvp, taps;
  float q_scale, eps;
  __host__ __device__ int64_t channels() const { return (int64_t)2 * G * dk + (int64_t)H * dv; }
};

// One warp per (run of rows, item): the heads of q | k | v, then one item for the decays and betas.  A lane owns four
// neighbouring channels (dk, dv <= 128) and keeps the last inputs in registers, so that every input is read once.
template <int RUN, int K1>
__global__ void __launch_bounds__(256, RUN > 1 ? 3 : 2) gdn_conv_kernel(GdnParams p) {
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
        const float g = -expf(__bfloat162float(p.a_log[n])) * sp;
        p.gb[(int64_t)row * p.H + n] = make_float2(row < p.n_decode ? expf(g) : g, sigmoid_exact(__bfloat162float(p.b[at])));
      }
    return;
  }
  const int part = h < p.G ? 0 : (h < 2 * p.G ? 1 : 2);
  h -= part == 0 ? 0 : (part == 1 ? p.G : 2 * p.G);
  const int d = part == 2 ? p.dv : p.dk, c = lane * 4;
  const bool on = c < d;
  const int64_t ch = (part == 2 ? (int64_t)2 * p.G * p.dk : (int64_t)part * p.G * p.dk) + (int64_t)h * d + c, C = p.channels();
  const bf16* x = (part == 2 ? p.v + (int64_t)(h / r) * p.v_gs + (h % r) * d : (part == 0 ? p.q : p.k) + (int64_t)h * p.qk_hs) + c;
  const int dp = part == 2 ? p.dvp : p.dkp;
  bf16* y = (part == 0 ? p.yq : (part == 1 ? p.yk : p.yv)) + (int64_t)h * dp + c;
  const int64_t y_ld = (int64_t)(part == 2 ? p.H : p.G) * dp;
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
  const auto finish = [&](int row, float* s) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = on ? __bfloat162float(__float2bfloat16(silu_as<bf16>(s[j]))) : 0.f;
      ss += s[j] * s[j];
    }
    if (part < 2) {
      ss = warp_sum(ss);
      if (lane == 0) (part == 0 ? p.fq : p.fk)[(int64_t)row * p.G + h] = (part == 0 ? p.q_scale : 1.f) * rsqrtf(ss + kGdnUnitEps);
    }
    if (c < dp) store_f32<4>(y + row * y_ld, s);                     // zeros behind d
  };
  int b = seq_of_row(p.cu_q, p.n_seqs, first), begin = first, end = first + 1, slot = -1, len = 0;
  if (b >= 0) {
    begin = p.cu_q[b];
    end = p.cu_q[b + 1];
    slot = p.slots[b];
    len = p.kv_lens[b];
  }
  if (RUN > 1 && slot >= 0 && first - begin >= K1 && first + RUN <= end) {      // most runs: no edge of a sequence nearby
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      float s[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[j] = v[i + 3][j] * w[0][j];
#pragma unroll
        for (int t = 1; t <= K1; ++t) s[j] += v[i + 3 - t][j] * w[t][j];
      }
      finish(first + i, s);
    }
    return;
  }
#pragma unroll 1
  for (int i = 0; i < RUN; ++i) {
    const int row = first + i;
    if (row >= p.rows) break;
    float x0[4][4];                                                 // x0[t]: t rows back
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x0[t][j] = 0.f;
#pragma unroll
        for (int u = 0; u < RUN; ++u)
          if (u == i) x0[t][j] = v[u + 3 - t][j];
      }
    if (row >= end) {                                               // the row starts another sequence
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
      s[j] = x0[0][j] * w[0][j];
#pragma unroll
      for (int t = 1; t <= K1; ++t)
        if (back >= t) s[j] += x0[t][j] * w[t][j];
    }
    bf16* tail = p.tail + ((int64_t)slot * C + ch) * K1;            // [channel][input], oldest first
    if (back < K1 && on) {
      __align__(8) bf16 past[4 * K1];
      const bool old = len > n;                                     // the slot's tail belongs to this sequence
#pragma unroll
      for (int q = 0; q < K1; ++q)
        *reinterpret_cast<uint2*>(past + 4 * q) = old ? reinterpret_cast<const uint2*>(tail)[q] : make_uint2(0u, 0u);
#pragma unroll
      for (int u = 0; u < K1; ++u) {                                // u + 1 inputs before the sequence's rows
        const int t = u + 1 + back;
        if (t > K1) break;                                          // (zero times what is not finite would not be zero)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[j] += __bfloat162float(past[j * K1 + K1 - 1 - u]) * (t == 1 ? w[1][j] : (t == 2 ? w[2][j] : w[3][j]));
      }
      if (n == 1) {                                                 // this lane alone reads these inputs: move them up
        __align__(8) bf16 now[4 * K1];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int t = 0; t < K1; ++t) now[j * K1 + t] = t + 1 < K1 ? past[j * K1 + t + 1] : __float2bfloat16(x0[0][j]);
#pragma unroll
        for (int q = 0; q < K1; ++q) reinterpret_cast<uint2*>(tail)[q] = *reinterpret_cast<const uint2*>(now + 4 * q);
      }
    }
    finish(row, s);
  }
}

// silu(z) times the normed and weighted output, in the model's order of roundings
__device__ __forceinline__ bf16 gdn_finish(float o, float inv, bf16 w, float z) {
  const bf16 n = __float2bfloat16(o * inv);
  return __float2bfloat16(__bfloat162float(__float2bfloat16(__bfloat162float(w) * __bfloat162float(n))) * silu_as<bf16>(z));
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
    qs[tid] = __bfloat162float(p.yq[qk * p.dkp + tid]) * p.fq[qk];
    ks[tid] = __bfloat162float(p.yk[qk * p.dkp + tid]) * p.fk[qk];
  }
  if (tid >= 128 && tid - 128 < dv) vs[tid - 128] = __bfloat162float(p.yv[row * p.dvp + tid - 128]);
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

// ------------------------------------------------------------------------------------------------ prompts, chunks of 16
// With G_t the sum of a chunk's g through token t, S_0 the state before the chunk, y the convolution's q and k rows and f their
// factors,
//
//   A_ts = e^(G_t - G_s) f_t f_s y_t . y_s  (s < t),   P_ts = e^(G_t - G_s) fq_t f_s yq_t . y_s  (s <= t),
//   M = (I + diag(beta) A)^-1 diag(beta),    U = M (V - diag(f e^G) Y S_0),    O = diag(fq e^G) Yq S_0 + P U,
//   S <- e^(G_end) S_0 + Y^T diag(f e^(G_end - G)) U.
//
// Every decay is at most 1.  y and v are bf16 as the convolution leaves them, so that their products on the tensor cores are
// exact and accumulate in fp32; S, U, M and P are fp32 values as three bf16 terms (24 bits), of which products below 2^-24 of
// the largest are left out.  (A chunk with anything that is not finite goes token by token.)  gdn_prep_kernel makes M, P and the
// factors, all chunks side by side; gdn_chunk_kernel walks the chunks of a sequence: a warp owns 16 state columns for all of dk as
// accumulators of S^T, which are the A operand of S^T Y^T without leaving the registers, as U^T is of the products behind it.
//
// Token by token in fp32 (states in registers, no barriers) the walk took 600 us for four prompts of 1024, 549, 842 and 366
// tokens, 32 heads of 128 x 128 (one B200), some 1100 cycles a token in a chain of product, exchange, product; in chunks it
// takes 198 us, the preparation 20 us.
constexpr int kGC = 16, kGWarps = 4, kGCols = 16 * kGWarps, kGStages = 3, kGVld = kGCols + 8;

struct GdnBlob {                             // bytes of one (chunk, head)
  static constexpr int mat = kGC * kGC * 2;  // [16][16] bf16
  static constexpr int m = 0, p = 3 * mat;   // three terms behind one another
  static constexpr int f = 6 * mat;          // [16] float4: f e^G, fq e^G, f e^(G_end - G), e^(G_end)
  static constexpr int bytes = f + kGC * 16;
};
// chunk i of prompt b: unique because a sequence of n rows has at most n / 16 + 1 chunks
__host__ __device__ __forceinline__ int64_t gdn_chunk_slot(int64_t row0, int b, int i) { return row0 / kGC + b + i; }

__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const auto pack = [](bf162 v) { return *reinterpret_cast<const uint32_t*>(&v); };
  const bf162 h = __floats2bfloat162_rn(x, y);
  const float2 hf = __bfloat1622float2(h);
  const bf162 m = __floats2bfloat162_rn(x - hf.x, y - hf.y);
  const float2 mf = __bfloat1622float2(m);
  hi = pack(h);
  mid = pack(m);
  lo = pack(__floats2bfloat162_rn(x - hf.x - mf.x, y - hf.y - mf.y));
}
__device__ __forceinline__ void put3(bf16* at, int stride, float x) {
  const bf16 h = __float2bfloat16(x), m = __float2bfloat16(x - __bfloat162float(h));
  at[0] = h;
  at[stride] = m;
  at[2 * stride] = __float2bfloat16(x - __bfloat162float(h) - __bfloat162float(m));
}

// grid (chunks of a sequence, key heads, prompts), 128 threads: warps 0 and 1 take Y Y^T and Yq Y^T, then a warp a value head
template <int DK>
__global__ void __launch_bounds__(128) gdn_prep_kernel(GdnParams p) {
  constexpr int LD = DK + 8, PC = DK / 8;
  __shared__ __align__(16) bf16 rows[2][kGC][LD];                    // k, q
  __shared__ float dots[2][kGC][kGC + 1], am[4][kGC][kGC + 1], bs[4][kGC], ff[2][kGC];
  __shared__ double gs[4][kGC];                                      // sums of g: differences of large ones must not lose the small
  const int g = blockIdx.y, b = p.n_decode + blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  pdl_launch_dependents();
  const int first = p.cu_q[b], n_seq = p.cu_q[b + 1] - first, i0 = blockIdx.x * kGC;
  if (i0 >= n_seq || p.slots[b] < 0) return;
  const int n = min(kGC, n_seq - i0), row0 = first + i0, r = p.H / p.G;
  for (int i = tid; i < 2 * kGC * PC; i += 128) {
    const int which = i / (kGC * PC), t = i / PC % kGC, c = (i % PC) * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (t < n) v = *reinterpret_cast<const uint4*>((which ? p.yq : p.yk) + ((int64_t)(row0 + t) * p.G + g) * DK + c);
    *reinterpret_cast<uint4*>(&rows[which][t][c]) = v;
  }
  if (tid < 2 * kGC) {
    const int t = tid % kGC;
    ff[tid / kGC][t] = t < n ? (tid < kGC ? p.fk : p.fq)[(int64_t)(row0 + t) * p.G + g] : 0.f;
  }
  __syncthreads();
  const int ta = lane >> 2, kc = (lane & 3) * 2;
  if (warp < 2) {
    float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < DK; k += 16) {
      const auto at = [&](int which, int t, int c) { return *reinterpret_cast<const uint32_t*>(&rows[which][t][k + c]); };
      const uint32_t a[4] = {at(warp, ta, kc), at(warp, ta + 8, kc), at(warp, ta, kc + 8), at(warp, ta + 8, kc + 8)};
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_bf16_16816(d[j], a, at(0, 8 * j + ta, kc), at(0, 8 * j + ta, kc + 8));
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) dots[warp][ta + (e >> 1) * 8][8 * j + kc + (e & 1)] = d[j][e];
  }
  __syncthreads();
  for (int i = warp; i < r; i += 4) {
    const int h = g * r + i;
    uint8_t* blob = p.blobs + (gdn_chunk_slot(first, blockIdx.z, blockIdx.x) * p.H + h) * GdnBlob::bytes;
    double G = 0.;
    if (lane < kGC) {
      const float2 gb = lane < n ? p.gb[(int64_t)(row0 + lane) * p.H + h] : make_float2(0.f, 0.f);
      G = gb.x;                                                      // g: rows behind the last one add nothing
      bs[warp][lane] = gb.y;                                         // and have beta 0
    }
#pragma unroll
    for (int o = 1; o < kGC; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, G, o);
      if (lane >= o) G += x;
    }
    // a decay to zero within one token, or NaN: differences of its sums say nothing, and no token is a NaN end
    const bool finite = __all_sync(0xffffffffu, fabs(G) < (double)INFINITY);
    const double end = finite ? __shfl_sync(0xffffffffu, G, kGC - 1) : (double)NAN;
    if (lane < kGC) {
      gs[warp][lane] = G;
      const float e = expf((float)G);
      reinterpret_cast<float4*>(blob + GdnBlob::f)[lane] =
          make_float4(ff[0][lane] * e, ff[1][lane] * e, ff[0][lane] * expf((float)(end - G)), expf((float)end));
    }
    __syncwarp();
    for (int x = lane; x < kGC * kGC; x += 32) {
      const int t = x >> 4, s = x & 15;
      const float e = s <= t ? expf((float)(gs[warp][t] - gs[warp][s])) * ff[0][s] : 0.f;
      am[warp][t][s] = s < t ? bs[warp][t] * ff[0][t] * e * dots[0][t][s] : 0.f;
      put3(reinterpret_cast<bf16*>(blob + GdnBlob::p) + x, kGC * kGC, ff[1][t] * e * dots[1][t][s]);
    }
    __syncwarp();
    if (lane < kGC) {                                                // column `lane` of the inverse by forward substitution
      float x[kGC];
      const float bt = bs[warp][lane];
#pragma unroll
      for (int t = 0; t < kGC; ++t) {
        float y = t == lane ? 1.f : 0.f;
#pragma unroll
        for (int s = 0; s < t; ++s) y -= am[warp][t][s] * x[s];
        x[t] = y;
        put3(reinterpret_cast<bf16*>(blob + GdnBlob::m) + t * kGC + lane, kGC * kGC, y * bt);
      }
    }
    __syncwarp();
  }
}

// n tokens from row0 on one after the other, for 16 columns of a state that lies in memory as the accumulators of the walk below
// (what a lane reads of it is what the lane wrote).  For chunks with anything that is not finite: by the chunk, zeros of M and P
// would carry it to tokens in front of it, and an infinite state has no three terms.
template <int DK>
__device__ __noinline__ void gdn_walk_tokens(const GdnParams& p, float* S, int row0, int n, int h, int g, int vrow, int kc) {
  const int dk = p.dk, dv = p.dv;
  for (int64_t row = row0; row < row0 + n; ++row) {
    const float2 gb = p.gb[row * p.H + h];
    const float decay = expf(gb.x), fk = p.fk[row * p.G + g], fq = p.fq[row * p.G + g];
    const bf16 *yk = p.yk + (row * p.G + g) * DK, *yq = p.yq + (row * p.G + g) * DK, *yv = p.yv + (row * p.H + h) * p.dvp;
    float d[2] = {0.f, 0.f}, o[2] = {0.f, 0.f};
    for (int i = 0; i < DK / 4; ++i) {
      const int c = (i >> 1) * 8 + kc + (i & 1);
      for (int u = 0; u < 2; ++u)
        if (c < dk && vrow + 8 * u < dv) d[u] += S[(int64_t)c * dv + vrow + 8 * u] * decay * (__bfloat162float(yk[c]) * fk);
    }
    for (int u = 0; u < 2; ++u) {
      d[u] += __shfl_xor_sync(0xffffffffu, d[u], 1);
      d[u] += __shfl_xor_sync(0xffffffffu, d[u], 2);
      if (vrow + 8 * u < dv) d[u] = gb.y * (__bfloat162float(yv[vrow + 8 * u]) - d[u]);
    }
    for (int i = 0; i < DK / 4; ++i) {
      const int c = (i >> 1) * 8 + kc + (i & 1);
      for (int u = 0; u < 2; ++u)
        if (c < dk && vrow + 8 * u < dv) {
          float* at = S + (int64_t)c * dv + vrow + 8 * u;
          const float x = *at * decay + __bfloat162float(yk[c]) * fk * d[u];
          *at = x;
          o[u] += x * (__bfloat162float(yq[c]) * fq);
        }
    }
    for (int u = 0; u < 2; ++u) {
      o[u] += __shfl_xor_sync(0xffffffffu, o[u], 1);
      o[u] += __shfl_xor_sync(0xffffffffu, o[u], 2);
      if (kc == 0 && vrow + 8 * u < dv) p.o[(row * p.H + h) * dv + vrow + 8 * u] = o[u];
    }
  }
}

// grid (slices of 64 columns, heads, prompts)
template <int DK>
__global__ void __launch_bounds__(32 * kGWarps, 2) gdn_chunk_kernel(const __grid_constant__ GdnParams p) {
  constexpr int CH = DK / 8, NT = 32 * kGWarps, TILE = kGC * DK * 2;
  constexpr int V_OFF = 2 * TILE, B_OFF = V_OFF + kGC * kGVld * 2, STAGE = (B_OFF + GdnBlob::bytes + 127) / 128 * 128;
  static_assert(kGStages * STAGE <= 48 * 1024, "static limit of dynamic shared memory");
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sb = smem_u32(smem);
  const int h = blockIdx.y, b = p.n_decode + blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = p.H / p.G, g = h / r, dk = p.dk, dv = p.dv, dvp = p.dvp, c0 = blockIdx.x * kGCols;
  pdl_wait();
  pdl_launch_dependents();
  const int row0 = p.cu_q[b], n_all = p.cu_q[b + 1] - row0, slot = p.slots[b];
  if (n_all <= 0 || slot < 0) return;
  const bool fresh = p.kv_lens[b] == n_all, works = c0 + warp * 16 < dv;
  float* S = p.state + (((int64_t)slot * p.H + h) * dk) * dv;
  const int vloc = warp * 16 + (lane >> 2), vrow = c0 + vloc, kc = (lane & 3) * 2;
  float acc[DK / 8][4];                      // S^T: rows (value columns) lane / 4, + 8; key channels 8 nt + kc, + 1
#pragma unroll
  for (int nt = 0; nt < DK / 8; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = nt * 8 + kc + (e & 1), v = vrow + (e >> 1) * 8;
      acc[nt][e] = (!fresh && c < dk && v < dv) ? S[(int64_t)c * dv + v] : 0.f;
    }
  if (blockIdx.x == 0 && n_all > 1) {                               // the convolution has read the tails
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
        const int at = n_all - K1 + t;
        keep[t] = at >= 0 ? x[(row0 + at) * p.ld + c] : (fresh ? __float2bfloat16(0.f) : tail[n_all + t]);
      }
      for (int t = 0; t < K1; ++t) tail[t] = keep[t];
    }
  }
  const int chunks = (n_all + kGC - 1) / kGC;
  const uint8_t* blobs = p.blobs + (gdn_chunk_slot(row0, blockIdx.z, 0) * p.H + h) * GdnBlob::bytes;
  const auto load = [&](int j) {
    if (j < chunks) {
      const uint32_t st = sb + (j % kGStages) * STAGE;
      for (int i = tid; i < 2 * kGC * CH; i += NT) {
        const int which = i / (kGC * CH), t = i / CH % kGC, c = i % CH;
        const bool ok = j * kGC + t < n_all;
        const int64_t row = row0 + (ok ? j * kGC + t : 0);
        cp_async16(st + which * TILE + swz<CH>(t, c), (which ? p.yq : p.yk) + (row * p.G + g) * DK + c * 8, ok);
      }
      for (int i = tid; i < kGC * (kGCols / 8); i += NT) {
        const int t = i / (kGCols / 8), c = (i % (kGCols / 8)) * 8;
        const bool ok = j * kGC + t < n_all && c0 + c < dvp;
        const int64_t row = row0 + (ok ? j * kGC + t : 0);
        cp_async16(st + V_OFF + (t * kGVld + c) * 2, p.yv + (row * p.H + h) * dvp + (ok ? c0 + c : 0), ok);
      }
      const uint8_t* src = blobs + (int64_t)j * p.H * GdnBlob::bytes;
      for (int i = tid; i < GdnBlob::bytes / 16; i += NT) cp_async16(st + B_OFF + i * 16, src + i * 16, true);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < kGStages - 1; ++s) load(s);
  const int arow = (lane & 7) + (((lane >> 3) & 1) << 3), acb = lane >> 4;
  const int brow = (lane & 7) + ((lane >> 4) << 3), bcb = (lane >> 3) & 1;
  for (int j = 0; j < chunks; ++j) {
    const int n = min(kGC, n_all - j * kGC);
    cp_async_wait<kGStages - 2>();
    __syncthreads();                         // chunk j is here, and everybody is done with the stage that is filled next
    load(j + kGStages - 1);
    if (!works) continue;
    const uint32_t st = sb + (j % kGStages) * STAGE;
    const uint8_t* stp = smem + (j % kGStages) * STAGE;
    float w[2][4], wl[2][4], o[2][4], ol[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) w[i][e] = wl[i][e] = o[i][e] = ol[i][e] = 0.f;
    // ---- S^T Y^T, S^T Yq^T
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk) {
      uint32_t kf[4], qf[4], hi[4], mid[4], lo[4];
      const uint32_t at = st + swz<CH>(brow, kk * 2 + bcb);
      ldmatrix_x4(kf[0], kf[1], kf[2], kf[3], at);
      ldmatrix_x4(qf[0], qf[1], qf[2], qf[3], at + TILE);
      split3(acc[2 * kk][0], acc[2 * kk][1], hi[0], mid[0], lo[0]);
      split3(acc[2 * kk][2], acc[2 * kk][3], hi[1], mid[1], lo[1]);
      split3(acc[2 * kk + 1][0], acc[2 * kk + 1][1], hi[2], mid[2], lo[2]);
      split3(acc[2 * kk + 1][2], acc[2 * kk + 1][3], hi[3], mid[3], lo[3]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mma_bf16_16816(w[i], hi, kf[2 * i], kf[2 * i + 1]);
        mma_bf16_16816(o[i], hi, qf[2 * i], qf[2 * i + 1]);
        mma_bf16_16816(wl[i], mid, kf[2 * i], kf[2 * i + 1]);
        mma_bf16_16816(ol[i], mid, qf[2 * i], qf[2 * i + 1]);
        mma_bf16_16816(wl[i], lo, kf[2 * i], kf[2 * i + 1]);
        mma_bf16_16816(ol[i], lo, qf[2 * i], qf[2 * i + 1]);
      }
    }
    // ---- U^T = (V - W)^T M^T
    const float4* fs = reinterpret_cast<const float4*>(stp + B_OFF + GdnBlob::f);
    const bf16* vs = reinterpret_cast<const bf16*>(stp + V_OFF);
    float4 f[2][2];                          // of tokens 8 i + kc, + 1
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) f[i][e] = fs[8 * i + kc + e];
    uint32_t xh[4], xm[4], xl[4];
    // every term of bf16: an infinite state, or input, is seen in the products with it, whatever they are multiplied with
    bool tame = fabsf(f[0][0].w) <= 1.f;
    const auto is_tame = [](float x) { return fabsf(x) < 3.38e38f; };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const bf16* v = vs + (8 * i + kc) * kGVld + vloc + 8 * u;
        const float x = __bfloat162float(v[0]) - f[i][0].x * (w[i][2 * u] + wl[i][2 * u]);
        const float y = __bfloat162float(v[kGVld]) - f[i][1].x * (w[i][2 * u + 1] + wl[i][2 * u + 1]);
        tame = tame && is_tame(x) && is_tame(y);
        split3(x, y, xh[2 * i + u], xm[2 * i + u], xl[2 * i + u]);
      }
    const uint32_t small = st + B_OFF + (uint32_t)(brow * kGC * 2 + bcb * 16);
    float uu[2][4], pu[2][4];
    // X^T times a matrix of three terms, the smallest products first
    const auto product = [&](float (&d)[2][4], int at) {
      uint32_t t0[4], t1[4], t2[4];
      ldmatrix_x4(t0[0], t0[1], t0[2], t0[3], small + at);
      ldmatrix_x4(t1[0], t1[1], t1[2], t1[3], small + at + GdnBlob::mat);
      ldmatrix_x4(t2[0], t2[1], t2[2], t2[3], small + at + 2 * GdnBlob::mat);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int e = 0; e < 4; ++e) d[i][e] = 0.f;
        mma_bf16_16816(d[i], xl, t0[2 * i], t0[2 * i + 1]);
        mma_bf16_16816(d[i], xm, t1[2 * i], t1[2 * i + 1]);
        mma_bf16_16816(d[i], xh, t2[2 * i], t2[2 * i + 1]);
        mma_bf16_16816(d[i], xm, t0[2 * i], t0[2 * i + 1]);
        mma_bf16_16816(d[i], xh, t1[2 * i], t1[2 * i + 1]);
        mma_bf16_16816(d[i], xh, t0[2 * i], t0[2 * i + 1]);
      }
    };
    product(uu, GdnBlob::m);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) tame = tame && is_tame(uu[i][e]);
    if (!__all_sync(0xffffffffu, tame)) {
      const auto elements = [&](auto&& f) {
#pragma unroll
        for (int nt = 0; nt < DK / 8; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = nt * 8 + kc + (e & 1), v = vrow + (e >> 1) * 8;
            if (c < dk && v < dv) f(acc[nt][e], S[(int64_t)c * dv + v]);
          }
      };
      elements([](float a, float& m) { m = a; });
      gdn_walk_tokens<DK>(p, S, row0 + j * kGC, n, h, g, vrow, kc);
      elements([](float& a, float m) { a = m; });
      continue;
    }
    // ---- O^T
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int u = 0; u < 2; ++u) split3(uu[i][2 * u], uu[i][2 * u + 1], xh[2 * i + u], xm[2 * i + u], xl[2 * i + u]);
    product(pu, GdnBlob::p);
    // ---- S^T <- e^(G_end) S^T + U^T diag(f e^(G_end - G)) Y
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int u = 0; u < 2; ++u)
        split3(uu[i][2 * u] * f[i][0].z, uu[i][2 * u + 1] * f[i][1].z, xh[2 * i + u], xm[2 * i + u], xl[2 * i + u]);
    const float end = f[0][0].w;
#pragma unroll
    for (int nt = 0; nt < DK / 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[nt][e] *= end;
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk) {
      uint32_t kf[4];
      ldmatrix_x4_trans(kf[0], kf[1], kf[2], kf[3], st + swz<CH>(arow, kk * 2 + acb));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mma_bf16_16816(acc[2 * kk + i], xl, kf[2 * i], kf[2 * i + 1]);
        mma_bf16_16816(acc[2 * kk + i], xm, kf[2 * i], kf[2 * i + 1]);
        mma_bf16_16816(acc[2 * kk + i], xh, kf[2 * i], kf[2 * i + 1]);
      }
    }
    const int64_t row = row0 + j * kGC;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * i + kc + (e & 1), v = vrow + (e >> 1) * 8;
        if (t < n && v < dv) p.o[((row + t) * p.H + h) * dv + v] = f[i][e & 1].y * (o[i][e] + ol[i][e]) + pu[i][e];
      }
  }
  cp_async_wait<0>();
  if (!works) return;
#pragma unroll
  for (int nt = 0; nt < DK / 8; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = nt * 8 + kc + (e & 1), v = vrow + (e >> 1) * 8;
      if (c < dk && v < dv) S[(int64_t)c * dv + v] = acc[nt][e];
    }
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
// dk, dv <= 128 and multiples of 4, taps 2 .. 4, all rows and heads 8-byte aligned; no prompt has more than max_q_len rows.
// Scratch: yq, yk [rows, G, 64 or 128], yv [rows, H, dv in eights] bf16; fq, fk [rows, G], gb [rows, H, 2] fp32; where there
// are prompts o [rows, H, dv] fp32 and xllm_gdn_blob_bytes() bytes.
XLLM_API int64_t xllm_gdn_blob_bytes(int rows, int prompts, int H) {
  return (xllm::gdn_chunk_slot(rows, prompts, 1) + 1) * H * xllm::GdnBlob::bytes;
}
XLLM_API int xllm_gdn_layer(void* state, void* tail, const void* slots, const void* cu_q, const void* kv_lens, const void* q,
                            const void* k, const void* v, const void* z, int64_t ld, int64_t z_ld, int qk_hs, int v_gs, int z_gs,
                            const void* b, const void* a, int64_t ba_ld, int ba_gs, const void* conv_w, const void* dt_bias,
                            const void* a_log, const void* norm_w, void* yq, void* yk, void* yv, void* fq, void* fk, void* gb,
                            void* o, void* blobs, void* out, int n_decode, int n_seqs, int rows, int max_q_len, int H, int G,
                            int dk, int dv, int taps, float q_scale, float eps, void* stream) {
  using namespace xllm;
  if (rows <= 0 || n_seqs <= 0) return 0;
  const auto al8 = [](const void* x) { return (((uintptr_t)x) & 7) == 0; };
  if (H <= 0 || G <= 0 || H % G != 0 || dk <= 0 || dk > 128 || dk % 4 != 0 || dv <= 0 || dv > 128 || dv % 4 != 0 || taps < 2 ||
      taps > 4 || n_decode > rows || n_decode > n_seqs || ld % 4 != 0 || z_ld % 4 != 0 || qk_hs % 4 != 0 || v_gs % 4 != 0 ||
      z_gs % 4 != 0 || !al8(q) || !al8(k) || !al8(v) || !al8(z) || !al8(out) || !al8(yq) || !al8(yk) || !al8(yv) || !al8(tail) || !al8(conv_w) ||
      ((((uintptr_t)state | (uintptr_t)yq | (uintptr_t)yk | (uintptr_t)yv | (uintptr_t)blobs) & 15) != 0) ||
      (n_seqs > n_decode && (o == nullptr || blobs == nullptr || max_q_len <= 0)))
    return (int)cudaErrorInvalidValue;
  GdnParams p;
  p.state = (float*)state; p.tail = (bf16*)tail; p.slots = (const int32_t*)slots; p.cu_q = (const int32_t*)cu_q;
  p.kv_lens = (const int32_t*)kv_lens; p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.z = (const bf16*)z;
  p.ld = ld; p.z_ld = z_ld; p.qk_hs = qk_hs; p.v_gs = v_gs; p.z_gs = z_gs; p.b = (const bf16*)b; p.a = (const bf16*)a;
  p.ba_ld = ba_ld; p.ba_gs = ba_gs; p.conv_w = (const bf16*)conv_w; p.dt_bias = (const bf16*)dt_bias;
  p.a_log = (const bf16*)a_log; p.norm_w = (const bf16*)norm_w; p.yq = (bf16*)yq; p.yk = (bf16*)yk; p.yv = (bf16*)yv;
  p.fq = (float*)fq; p.fk = (float*)fk; p.gb = (float2*)gb; p.o = (float*)o; p.blobs = (uint8_t*)blobs;
  p.out = (bf16*)out; p.dkp = dk <= 64 ? 64 : 128; p.dvp = (dv + 7) & ~7;
  p.n_decode = n_decode; p.n_seqs = n_seqs; p.rows = rows; p.H = H; p.G = G; p.dk = dk; p.dv = dv; p.taps = taps;
  p.q_scale = q_scale; p.eps = eps;
  cudaStream_t s = (cudaStream_t)stream;
  // Runs of four rows read seven inputs of a channel where four single rows read sixteen; few rows need the warps more than
  // the reuse.  Bound by latency and instructions: the registers of longer runs cost more in warps than their reuse gives.
  const int items = 2 * G + H + 1, run = rows > 128 ? 4 : 1;
  const dim3 grid((unsigned)((((int64_t)rows + run - 1) / run * items + 7) / 8));
  const auto conv = [&](auto kernel) { launch_pdl(kernel, grid, dim3(256), 0, s, p); };
  if (taps == 4) conv(run > 1 ? gdn_conv_kernel<4, 3> : gdn_conv_kernel<1, 3>);
  else if (taps == 3) conv(run > 1 ? gdn_conv_kernel<4, 2> : gdn_conv_kernel<1, 2>);
  else conv(run > 1 ? gdn_conv_kernel<4, 1> : gdn_conv_kernel<1, 1>);
  int rc = XLLM_LAUNCH_CHECK();
  if (rc != 0) return rc;
  if (n_seqs > n_decode) {
    const int np = n_seqs - n_decode;
    const dim3 pg((max_q_len + kGC - 1) / kGC, G, np), wg((dv + kGCols - 1) / kGCols, H, np);
    const auto walk = [&](auto prep, auto chunk, int DK) {
      const size_t smem = (size_t)kGStages * ((2 * kGC * DK * 2 + kGC * kGVld * 2 + GdnBlob::bytes + 127) / 128 * 128);
      launch_pdl(prep, pg, dim3(128), 0, s, p);
      launch_pdl(chunk, wg, dim3(32 * kGWarps), smem, s, p);
    };
    if (p.dkp == 64) walk(gdn_prep_kernel<64>, gdn_chunk_kernel<64>, 64);
    else walk(gdn_prep_kernel<128>, gdn_chunk_kernel<128>, 128);
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
