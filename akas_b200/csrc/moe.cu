// A routed feed-forward (mixture of experts): the router, and the experts for steps of few tokens and for float32.
//
// Router, per token, all in float32: logits z = W_r h over the R router outputs (one chain of sums per (token,
// output) whose order depends on the width only), s = softmax(z); the choice score is s + correction; the outputs
// form `groups` equal groups of neighbours, a group's score is its largest choice score, only outputs of the `keep`
// best groups can be chosen; the `top` largest choice scores among those are chosen (ties: the lower index); the
// weights are the chosen outputs' s over their sum (+ 1e-20). Router outputs from `experts` on are identity experts:
// they have no matrices and return their input. Options: `sigmoid`, s = 1 / (1 + exp(-z)) per output instead of the
// softmax; no correction (a null pointer); `renorm` 0, the weights are the chosen s as they are; `extra` more rows of
// W_r behind the R that compete, whose sigmoids are returned beside the choice (gates that read the router's input).
// Without a correction the choice goes by the logits themselves, which order as the scores do. `group_best` B > 1: a
// group's score is the sum of its B largest choice scores (and the choice then goes by the scores in any case);
// `wscale`: every weight times this constant.
//
// Experts, token by token (moe_gate_up, moe_down): act[pair] = silu(W_gate h) * (W_up h) for every (token, chosen
// real expert) pair, then out[n] = sum over the token's chosen outputs of weight * (W_down act, or h for an identity
// expert), added in the order of the choice. Every output is one warp's sum over the inner size in a fixed order, so
// a token's result does not depend on what else the step holds. (bfloat16 steps of few pairs take an expert's rows once for
// all of its pairs where a model's sizes suit that: "experts, few pairs".) Weights of all experts are stacked: gate and up as
// [experts, 2 F, C] (gate rows first), down as [experts, C, F]. Where the weight multiplies the expert's INPUT
// (out[n] = sum expert(w h)), moe_gate_up gets the weights and scales both of its float32 sums (W (w h) = w (W h))
// before the activation, and moe_down gets none. Ungated experts (`plain`, an AKAS_PLAIN_* activation): the stack is
// [experts, F, C] and act[pair] = act(W_up h). moe_down can also add a dense result of every token (a shared
// expert's), times a gate per token.
#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

using namespace akas;
using tc::mbar_arrive;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::smem_u32;

namespace {

constexpr int kRouteTokens = 8;   // tokens of a router block = its warps
constexpr int kRouteChunk = 2048; // channels of h staged at a time (64 KB of float32 rows for the block's tokens)
constexpr int kRouteOutputs = 4;  // router outputs whose rows a warp reads at the same time

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
// An activation without a gate in full float32 (AKAS_PLAIN_*).
__device__ __forceinline__ float plain_activation(float x, int act) {
  if (act == AKAS_PLAIN_RELU2) { const float r = fmaxf(x, 0.f); return r * r; }
  if (act == AKAS_PLAIN_GELU_TANH) return 0.5f * x * (1.f + tanhf(0.7978845608028654f * fmaf(0.044715f * x * x, x, x)));
  return act == AKAS_PLAIN_SILU ? silu_f(x) : x;
}

// One warp chooses for token n from its logits zt [RC + extra] (see above); zt and pt become scores, gt holds the groups'.
__device__ __forceinline__ void choose_outputs(float* zt, float* pt, float* gt, const float* __restrict__ correction,
                                               int* __restrict__ chosen, float* __restrict__ weights, int n, int lane, int RC,
                                               int groups, int keep, int top, int sigmoid, int renorm, int extra,
                                               float* __restrict__ extras, int group_best, float wscale) {
  for (int j = lane; j < extra; j += 32) extras[(size_t)n * extra + j] = 1.f / (1.f + expf(-zt[RC + j]));
  const int R = RC;  // from here on: the outputs that compete
  if (sigmoid) {
    // Without a correction the choice goes by the logits themselves: the same order as their sigmoids', and two large
    // logits whose sigmoids both round to one still compare.
    for (int e = lane; e < R; e += 32) {
      const float logit = zt[e];
      zt[e] = 1.f / (1.f + expf(-logit));
      pt[e] = correction != nullptr ? zt[e] + correction[e] : group_best > 1 ? zt[e] : logit;
    }
  } else {
    float top_z = -INFINITY;
    for (int e = lane; e < R; e += 32) top_z = fmaxf(top_z, zt[e]);
    top_z = warp_max(top_z);
    float sum = 0.f;
    for (int e = lane; e < R; e += 32) {
      pt[e] = zt[e];  // without a correction: the choice goes by the logits
      const float p = expf(zt[e] - top_z);
      zt[e] = p;
      sum += p;
    }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
    for (int e = lane; e < R; e += 32) {
      zt[e] *= inv;
      if (correction != nullptr) pt[e] = zt[e] + correction[e];
      else if (group_best > 1) pt[e] = zt[e];
    }
  }
  __syncwarp();
  const int size = R / groups;
  if (groups > 1 && keep < groups) {
    for (int g = lane; g < groups; g += 32) {
      float sum = 0.f, taken = INFINITY;
      int at = -1;  // the last that was added, and its value: the next one is the largest behind it (ties: by index)
      for (int b = 0; b < min(group_best, size); ++b) {
        float best = -INFINITY;
        int next = -1;
        for (int e = g * size; e < (g + 1) * size; ++e) {
          const float v = pt[e];
          if ((v < taken || (v == taken && e > at)) && (next < 0 || v > best)) { best = v; next = e; }
        }
        if (next < 0) break;
        sum += best;
        taken = best;
        at = next;
      }
      gt[g] = sum;
    }
    __syncwarp();
    // a group stays iff fewer than `keep` groups beat it (a tie goes to the lower index)
    for (int g = lane; g < groups; g += 32) {
      int ahead = 0;
      for (int o = 0; o < groups; ++o) ahead += gt[o] > gt[g] || (gt[o] == gt[g] && o < g);
      if (ahead >= keep)
        for (int e = g * size; e < (g + 1) * size; ++e) pt[e] = -INFINITY;
    }
    __syncwarp();
  }
  float total = 0.f, mine = 0.f;  // mine: the score of the lane-th choice
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < R; e += 32)
      if (pt[e] > best) { best = pt[e]; at = e; }  // ascending e: the first of equal scores stays
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (at == 0x7fffffff) at = 0;  // fewer choosable outputs than `top`: cannot happen for a valid configuration
    if (lane == 0) {
      chosen[(size_t)n * top + k] = at;
      if (!renorm || k >= 32) weights[(size_t)n * top + k] = renorm ? zt[at] : zt[at] * wscale;
      pt[at] = -INFINITY;
    }
    if (lane == k) mine = zt[at];
    total += zt[at];
    __syncwarp();
  }
  if (renorm) {
    const float norm = wscale / (total + 1e-20f);
    if (lane < top) weights[(size_t)n * top + lane] = mine * norm;
    for (int k = 32; lane == 0 && k < top; ++k) weights[(size_t)n * top + k] *= norm;
  }
}

template <typename T>
__global__ void __launch_bounds__(kRouteTokens * 32)
moe_route_kernel(const T* __restrict__ h, long long ldh, const float* __restrict__ w, const float* __restrict__ correction,
                 int* __restrict__ chosen, float* __restrict__ weights, int N, int C, int RC, int groups, int keep, int top,
                 int sigmoid, int renorm, int extra, float* __restrict__ extras, int group_best, float wscale) {
  extern __shared__ __align__(16) float smem[];
  const int R = RC + extra;                        // rows of the matrix: the RC outputs that compete, then the extra ones
  float* rows = smem;                              // [kRouteTokens][kRouteChunk]
  float* z = rows + kRouteTokens * kRouteChunk;    // [kRouteTokens][R] logits, then scores
  float* pick = z + kRouteTokens * R;              // [kRouteTokens][R] choice scores
  float* gbest = pick + kRouteTokens * R;          // [kRouteTokens][groups]
  float* part = gbest + kRouteTokens * groups;     // [warps][kRouteOutputs][kRouteTokens] the warps' partial sums
  const int n0 = blockIdx.x * kRouteTokens;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kRouteTokens * R; i += blockDim.x) z[i] = 0.f;
  if (gridDim.x <= 16) {
    // a step of few tokens is a few blocks that wait for memory: the whole matrix is asked into the L2 at once, so that
    // the reads below, one group of outputs after another, do not each wait for DRAM
    const char* bytes = reinterpret_cast<const char*>(w);
    const size_t total = (size_t)R * C * sizeof(float);
    for (size_t off = (size_t)threadIdx.x * 128; off < total; off += (size_t)blockDim.x * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(bytes + off));
  }
  for (int c0 = 0; c0 < C; c0 += kRouteChunk) {
    const int width = min(kRouteChunk, C - c0);
    __syncthreads();
    if (C % 8 == 0 && ldh % 8 == 0 && ((uintptr_t)h % 16) == 0) {  // eight channels a load
      const int per_row = width / 8;
      for (int i = threadIdx.x; i < kRouteTokens * per_row; i += blockDim.x) {
        const int t = i / per_row, c = (i % per_row) * 8;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (n0 + t < N) load8(h + (size_t)(n0 + t) * ldh + c0 + c, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) rows[t * kRouteChunk + c + j] = v[j];
      }
    } else {
      for (int i = threadIdx.x; i < kRouteTokens * width; i += blockDim.x) {
        const int t = i / width, c = i % width;
        rows[t * kRouteChunk + c] = n0 + t < N ? to_f32(h[(size_t)(n0 + t) * ldh + c0 + c]) : 0.f;
      }
    }
    __syncthreads();
    // Warp w takes the w-th eighth of the staged channels for EVERY router output, so that all of a lane's loads of
    // the matrix are in flight at once (one trip to memory instead of one per output); the warps' partial sums meet
    // in shared memory and are added in the order of the warps: the order of a (token, output) sum depends on the
    // width only.
    const bool vec = C % 4 == 0 && ((uintptr_t)w % 16) == 0;
    const int slice = ((width + kRouteTokens - 1) / kRouteTokens + 3) / 4 * 4;
    const int s0 = min(width, warp * slice), s1 = min(width, s0 + slice);
    for (int e0 = 0; e0 < R; e0 += kRouteOutputs) {
      float acc[kRouteOutputs][kRouteTokens];
#pragma unroll
      for (int o = 0; o < kRouteOutputs; ++o)
#pragma unroll
        for (int t = 0; t < kRouteTokens; ++t) acc[o][t] = 0.f;
      if (vec) {
        for (int c = s0 + lane * 4; c < s1; c += 128) {
          float4 wv[kRouteOutputs];
#pragma unroll
          for (int o = 0; o < kRouteOutputs; ++o)
            wv[o] = *reinterpret_cast<const float4*>(w + (size_t)min(e0 + o, R - 1) * C + c0 + c);  // (no load hangs on a condition)
#pragma unroll
          for (int t = 0; t < kRouteTokens; ++t) {
            const float4 hv = *reinterpret_cast<const float4*>(rows + t * kRouteChunk + c);
#pragma unroll
            for (int o = 0; o < kRouteOutputs; ++o) {
              acc[o][t] = fmaf(hv.x, wv[o].x, acc[o][t]); acc[o][t] = fmaf(hv.y, wv[o].y, acc[o][t]);
              acc[o][t] = fmaf(hv.z, wv[o].z, acc[o][t]); acc[o][t] = fmaf(hv.w, wv[o].w, acc[o][t]);
            }
          }
        }
      } else {
        for (int c = s0 + lane; c < s1; c += 32) {
#pragma unroll
          for (int o = 0; o < kRouteOutputs; ++o) {
            const float wv = e0 + o < R ? w[(size_t)(e0 + o) * C + c0 + c] : 0.f;
#pragma unroll
            for (int t = 0; t < kRouteTokens; ++t) acc[o][t] = fmaf(rows[t * kRouteChunk + c], wv, acc[o][t]);
          }
        }
      }
      // the lanes' 32 sums each (4 outputs x 8 tokens) are added across the warp so that lane l ends with the total of
      // sum number l: every round a lane hands one half of what it still holds to its partner and keeps the other
      // (31 shuffles instead of 32 x 5); the order of the additions is the same for every token and batch
      static_assert(kRouteOutputs * kRouteTokens == 32, "one sum per lane");
      float* v = &acc[0][0];
#pragma unroll
      for (int off = 16, n = 32; off >= 1; off >>= 1, n >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
          const float send = upper ? v[i] : v[i + n / 2];
          const float keep = upper ? v[i + n / 2] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
      part[warp * 32 + lane] = v[0];  // [warp][output][token]
      __syncthreads();
      for (int i = threadIdx.x; i < kRouteOutputs * kRouteTokens; i += blockDim.x) {
        const int o = i / kRouteTokens, t = i % kRouteTokens;
        if (e0 + o < R) {
          float sum = z[t * R + e0 + o];
          for (int ww = 0; ww < kRouteTokens; ++ww) sum += part[(ww * kRouteOutputs + o) * kRouteTokens + t];
          z[t * R + e0 + o] = sum;
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  // warp t chooses for token n0 + t
  const int n = n0 + warp;
  if (n >= N) return;
  choose_outputs(z + warp * R, pick + warp * R, gbest + warp * groups, correction, chosen, weights, n, lane, RC, groups, keep, top,
                 sigmoid, renorm, extra, extras, group_best, wscale);
}

// Four neighbouring elements as floats (16 bytes of float32, 8 of bfloat16).
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 a = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(a.x << 16); v[1] = __uint_as_float(a.x & 0xffff0000u);
  v[2] = __uint_as_float(a.y << 16); v[3] = __uint_as_float(a.y & 0xffff0000u);
}

// The router for steps of few tokens: a block per token instead of one per eight, because what such a step waits for is the
// trip of the matrix's rows to one SM, again for every four outputs. Here a warp asks for its slice of sixteen outputs'
// rows at once. Slices, chains and the order in which lanes and warps meet are those of the kernel above, so both give the
// same bits. Rows of whole 16-byte words only. Up to two blocks an SM come at once; more of them wait for a second turn, and then
// the rows' trips per token weigh as much. bfloat16 rows, us, the kernel above / this one: 16 outputs of 1,536 at 1, 8 and 296 tokens
// 11.3 / 5.9, 12.3 / 6.1 and 12.3 / 6.7; 256 of 2,048 110 / 36, 111 / 37 and 104 / 42; at 512 tokens 12.3 / 11.6 and 104 / 82, but
// 8 outputs of 512 7.3 / 10.0 (at 296 7.3 / 5.8).
constexpr int kRouteFewOutputs = 16;

template <typename T>
__global__ void __launch_bounds__(kRouteTokens * 32)
moe_route_few_kernel(const T* __restrict__ h, long long ldh, const float* __restrict__ w, const float* __restrict__ correction,
                     int* __restrict__ chosen, float* __restrict__ weights, int C, int RC, int groups, int keep, int top,
                     int sigmoid, int renorm, int extra, float* __restrict__ extras, int group_best, float wscale) {
  extern __shared__ __align__(16) float smem[];
  const int R = RC + extra, n = blockIdx.x;
  float* z = smem;            // [R] logits, then scores
  float* pick = z + R;        // [R] choice scores
  float* gbest = pick + R;    // [groups]
  float* part = gbest + groups;  // [warps][kRouteFewOutputs]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* row = h + (size_t)n * ldh;
  for (int e0 = 0; e0 < R; e0 += kRouteFewOutputs) {
    float sum = 0.f;  // thread o < kRouteFewOutputs: the logit of output e0 + o
    for (int c0 = 0; c0 < C; c0 += kRouteChunk) {
      const int width = min(kRouteChunk, C - c0);
      const int slice = ((width + kRouteTokens - 1) / kRouteTokens + 3) / 4 * 4;
      const int s0 = min(width, warp * slice), s1 = min(width, s0 + slice);
      float v[kRouteFewOutputs];
#pragma unroll
      for (int o = 0; o < kRouteFewOutputs; ++o) v[o] = 0.f;
      constexpr int kTrips = kRouteChunk / kRouteTokens / 128;
#pragma unroll
      for (int u = 0; u < kTrips; ++u) {
        const int c = s0 + lane * 4 + u * 128;
        if (c >= s1) break;
        // all of the outputs' words in one trip to memory: no load hangs on a condition (outputs past the last take its row)
        float4 wv[kRouteFewOutputs];
#pragma unroll
        for (int o = 0; o < kRouteFewOutputs; ++o)
          wv[o] = *reinterpret_cast<const float4*>(w + (size_t)min(e0 + o, R - 1) * C + c0 + c);
        float x[4];
        load4(row + c0 + c, x);
#pragma unroll
        for (int o = 0; o < kRouteFewOutputs; ++o) {
          v[o] = fmaf(x[0], wv[o].x, v[o]); v[o] = fmaf(x[1], wv[o].y, v[o]);
          v[o] = fmaf(x[2], wv[o].z, v[o]); v[o] = fmaf(x[3], wv[o].w, v[o]);
        }
      }
#pragma unroll
      for (int off = 16, left = kRouteFewOutputs; off >= 2; off >>= 1, left >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < left / 2; ++i) {
          const float send = upper ? v[i] : v[i + left / 2];
          const float mine = upper ? v[i + left / 2] : v[i];
          v[i] = mine + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
      const float whole = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
      if ((lane & 1) == 0) part[warp * kRouteFewOutputs + (lane >> 1)] = whole;
      __syncthreads();
      if (threadIdx.x < kRouteFewOutputs)
        for (int ww = 0; ww < kRouteTokens; ++ww) sum += part[ww * kRouteFewOutputs + threadIdx.x];
      __syncthreads();
    }
    if (threadIdx.x < kRouteFewOutputs && e0 + (int)threadIdx.x < R) z[e0 + threadIdx.x] = sum;
  }
  __syncthreads();
  if (warp == 0)
    choose_outputs(z, pick, gbest, correction, chosen, weights, n, lane, RC, groups, keep, top, sigmoid, renorm, extra, extras,
                   group_best, wscale);
}

// One warp per (pair, hidden channel f): both dots over C, act = silu(gate) * up. Pairs of identity experts do nothing.
// in_weights (or null): the pair's weight multiplies both sums before the activation. plain (AKAS_PLAIN_*): no gate, one
// dot per hidden channel over rows of a stack [experts, F, C], act = that activation of it.
template <typename T>
__global__ void __launch_bounds__(256)
moe_gate_up_kernel(const T* __restrict__ h, long long ldh, const T* __restrict__ w_gate_up, const int* __restrict__ chosen,
                   T* __restrict__ act, int pairs, int top, int C, int F, int experts, const float* __restrict__ in_weights,
                   int plain) {
  const int pair = blockIdx.x;
  const int e = chosen[pair];
  if (e >= experts || e < 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const T* x = h + (size_t)(pair / top) * ldh;
  const T* wg = w_gate_up + (size_t)e * (plain ? 1 : 2) * F * C;
  const float scale = in_weights != nullptr ? in_weights[pair] : 1.f;
  constexpr int N = Vec<T>::N;
  const bool vec = C % N == 0 && ldh % N == 0 && ((uintptr_t)h % 16) == 0 && ((uintptr_t)w_gate_up % 16) == 0;
  for (int f = blockIdx.y * warps + warp; f < F; f += gridDim.y * warps) {
    const T* g_row = wg + (size_t)f * C;
    if (plain) {
      float sum = 0.f;
      if (vec) {
        for (int c = lane * N; c < C; c += 32 * N) {
          float xv[N], gv[N];
          load_vec(x + c, xv);
          load_vec(g_row + c, gv);
#pragma unroll
          for (int i = 0; i < N; ++i) sum = fmaf(xv[i], gv[i], sum);
        }
      } else {
        for (int c = lane; c < C; c += 32) sum = fmaf(to_f32(x[c]), to_f32(g_row[c]), sum);
      }
      sum = warp_sum(sum) * scale;
      if (lane == 0) act[(size_t)pair * F + f] = from_f32<T>(plain_activation(sum, plain));
      continue;
    }
    const T* u_row = wg + (size_t)(F + f) * C;
    float ag = 0.f, au = 0.f;
    if (vec) {
      for (int c = lane * N; c < C; c += 32 * N) {
        float xv[N], gv[N], uv[N];
        load_vec(x + c, xv);
        load_vec(g_row + c, gv);
        load_vec(u_row + c, uv);
#pragma unroll
        for (int i = 0; i < N; ++i) { ag = fmaf(xv[i], gv[i], ag); au = fmaf(xv[i], uv[i], au); }
      }
    } else {
      for (int c = lane; c < C; c += 32) {
        const float xv = to_f32(x[c]);
        ag = fmaf(xv, to_f32(g_row[c]), ag);
        au = fmaf(xv, to_f32(u_row[c]), au);
      }
    }
    ag = warp_sum(ag) * scale;
    au = warp_sum(au) * scale;
    if (lane == 0) act[(size_t)pair * F + f] = from_f32<T>(silu_f(ag) * au);
  }
}

// One warp per (token, output channel c): the weighted sum over the token's chosen outputs. With `x` the sum does not
// go to `out` but into the residual stream: x += mult * (ls_a * a + ls_b * sum), the update of a block whose mixer's
// result a and feed-forward meet the stream together (a null scale is all ones; a null a: none). Null weights: every weight is one.
// shared (or null): float32 [N, C] added to the sum, times shared_gate[n * ldsg] where that is given.
template <typename T>
__global__ void __launch_bounds__(256)
moe_down_kernel(const T* __restrict__ h, long long ldh, const T* __restrict__ w_down, const int* __restrict__ chosen,
                const float* __restrict__ weights, const T* __restrict__ act, float* __restrict__ out, int top, int C, int F,
                int experts, float* __restrict__ x, const float* __restrict__ a_res, const float* __restrict__ ls_a,
                const float* __restrict__ ls_b, float mult, const float* __restrict__ shared,
                const float* __restrict__ shared_gate, long long ldsg) {
  const int n = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  constexpr int N = Vec<T>::N;
  const bool vec = F % N == 0 && ((uintptr_t)act % 16) == 0 && ((uintptr_t)w_down % 16) == 0;
  for (int c = blockIdx.y * warps + warp; c < C; c += gridDim.y * warps) {
    float total = 0.f;
    for (int k = 0; k < top; ++k) {
      const int e = chosen[(size_t)n * top + k];
      const float g = weights != nullptr ? weights[(size_t)n * top + k] : 1.f;
      if (e >= experts) {
        total = fmaf(g, to_f32(h[(size_t)n * ldh + c]), total);
        continue;
      }
      const T* row = w_down + ((size_t)e * C + c) * F;
      const T* a = act + ((size_t)n * top + k) * F;
      float acc = 0.f;
      if (vec) {
        for (int f = lane * N; f < F; f += 32 * N) {
          float av[N], wv[N];
          load_vec(a + f, av);
          load_vec(row + f, wv);
#pragma unroll
          for (int i = 0; i < N; ++i) acc = fmaf(av[i], wv[i], acc);
        }
      } else {
        for (int f = lane; f < F; f += 32) acc = fmaf(to_f32(a[f]), to_f32(row[f]), acc);
      }
      total = fmaf(g, warp_sum(acc), total);
    }
    if (lane == 0) {
      if (shared != nullptr) total = fmaf(shared_gate != nullptr ? shared_gate[(size_t)n * ldsg] : 1.f, shared[(size_t)n * C + c], total);
      if (x != nullptr) {
        const size_t at = (size_t)n * C + c;
        x[at] = fmaf(mult, fmaf(ls_b ? ls_b[c] : 1.f, total, a_res ? (ls_a ? ls_a[c] : 1.f) * a_res[at] : 0.f), x[at]);
      } else {
        out[(size_t)n * C + c] = total;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ experts, few pairs
//
// bfloat16 steps of at most kFewPairs (token, expert) pairs: what bounds them is reading the chosen experts' matrices, once
// each. The kernels above walk pair by pair: an expert that two tokens chose is read twice (the second time from the L2), a
// warp has the loads of one row in flight, and widening and multiplying every weight for every pair keeps the issue slots
// busier than the memory (scalar warps behind the ring below still were: 31.9 and 23.0 us where these take 25.9 and 17.4).
// Here a block per SM walks tiles of 16 rows of an EXPERT: a producer warp keeps a ring of row copies full (cp.async.bulk, a
// lane a row, rows 16 bytes further apart than they are long, so that ldmatrix meets no bank twice; 150 to 200 KB on their
// way per SM; whole rows, because halves of them take twice the copies: 25.8 us for the down projection), and a consumer
// warp takes a whole tile against up to eight of the expert's pairs at a time by mma.sync m16n8k16, the rows as A, the
// pairs' vectors as B. (tcgen05 wants 64 rows a tile at least, four times what a stage holds.) Sixteen products at a time
// are summed by the tensor core and then added, rounded to nearest, by fours to one of four float32 sums: the core's own
// running sum cuts off what it cannot hold, step after step. So the error against 64 bits is the older kernels' (the down
// projection alone: 0.88e-7 to 0.92e-7 of the results' size at 1,536 x 1,728, 0.96e-7 to 0.98e-7 there). A (pair, row) sum is
// the same chain whatever else the step holds. Waits are bounded (akas_moe_status).
// 14 experts of 1,536 x 1,728, four a token, back to back (us: pair by pair / here / the bytes at 6.65 TB/s): gate and up at 1,
// 8 and 16 tokens 12.0 / 10.0 / 6.4, 42.3 / 25.9 / 20.8 and 72.4 / 34.4 / 22.4; down 13.4 / 8.4 / 3.2, 25.4 / 17.4 / 10.4 and
// 39.5 / 20.5 / 11.2. The rest is a launch's start: the choice sorted out, the first rows' way, the last tiles.
constexpr int kFewPairs = 64, kTileRows = 16, kPad = 8;  // kPad: elements between a row's end and the next row in shared memory
constexpr int kMostStages = 8, kStreamSmem = 225 * 1024;

__device__ int g_moe_status = 0;

__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// What every block of a step derives from the choice: the real experts that were chosen, in the order of their first pair,
// and every expert's pairs, one bit each.
struct Chosen {
  int picks[kFewPairs], experts[kFewPairs], used;
  unsigned long long pairs[kFewPairs];
  unsigned first[2];
};

__device__ __forceinline__ void sort_out(Chosen& c, const int* __restrict__ chosen, int pairs, int experts) {
  const int tid = threadIdx.x;
  if (tid < kFewPairs) c.picks[tid] = tid < pairs ? chosen[tid] : -1;
  __syncthreads();
  if (tid < kFewPairs) {
    const int e = c.picks[tid];
    unsigned long long mine = 0;
    for (int p = 0; p < pairs; ++p) mine |= (unsigned long long)(c.picks[p] == e) << p;
    const bool first = e >= 0 && e < experts && __ffsll((long long)mine) - 1 == tid;
    const unsigned votes = __ballot_sync(0xffffffffu, first);
    if ((tid & 31) == 0) c.first[tid >> 5] = votes;
    asm volatile("bar.sync 1, 64;" ::: "memory");
    if (first) {
      const int at = __popc(c.first[tid >> 5] & ((1u << (tid & 31)) - 1)) + (tid >= 32 ? __popc(c.first[0]) : 0);
      c.experts[at] = e;
      c.pairs[at] = mine;
    }
    if (tid == 0) c.used = __popc(c.first[0]) + __popc(c.first[1]);
  }
  __syncthreads();
}

// The ring of stages, one consumer warp a stage: a warp takes every consumers-th tile, and the ring's depth is the number of
// consumers, so that a stage is always the same warp's (a warp that came to another's stage for a later filling before the
// one in front of it had landed would find the barrier's parity as it wants it).
struct Ring {
  uint64_t full[kMostStages], empty[kMostStages];
  int abort;
};
__device__ __forceinline__ void ring_init(Ring& ring, int stages) {
  if (threadIdx.x == 0) {
    ring.abort = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ring.full[s], 1);
      mbar_init(&ring.empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
}
__device__ __forceinline__ bool ring_wait(Ring& ring, uint64_t* bar, unsigned parity, int code) {
  if (*(volatile int*)&ring.abort) return false;
  if (mbar_wait(bar, parity)) return true;
  *(volatile int*)&ring.abort = 1;
  atomicExch(&g_moe_status, code);
  return false;
}
__device__ __forceinline__ void ring_lost(Ring& ring) {
  if (*(volatile int*)&ring.abort)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // a lost launch: let copies in flight finish
}

// The fragments of 64 k, and their products: the tensor core's sums of 16 products, added in pairs.
struct Fragments {
  uint32_t a[4][4], b[2][4];
  __device__ __forceinline__ void load(const bf16* rows, const bf16* vectors) {
#pragma unroll
    for (int i = 0; i < 4; ++i) ldmatrix_x4(a[i], rows + i * 16);
#pragma unroll
    for (int i = 0; i < 2; ++i) ldmatrix_x4(b[i], vectors + i * 32);
  }
  __device__ __forceinline__ void add_product(float (&sum)[4]) const {
    float d[4][4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) mma_bf16(d[i], a[i], b[i >> 1][(i & 1) * 2], b[i >> 1][(i & 1) * 2 + 1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += (d[0][i] + d[1][i]) + (d[2][i] + d[3][i]);
  }
};

// acc = 16 rows (`tile`, `pitch` elements apart) times the eight vectors whose rows lie at the lanes' pointers (lane l: vector
// l % 8), over K elements, a multiple of 32. The next 64 k are read while these are multiplied. Fragment layouts: see mma.cuh.
__device__ __forceinline__ void tile_product(const bf16* tile, int pitch, const bf16* vector, int K, int lane, float (&acc)[4]) {
  const bf16* a = tile + (lane & 15) * pitch + (lane >> 4) * 8;
  const bf16* b = vector + (lane >> 3) * 8;  // the four 8-wide pieces of 32 k
  float sum[4][4] = {};
  const int blocks = K / 64;
  int i = 0;
  if (blocks >= 4) {
    Fragments even, odd;
    even.load(a, b);
    const int last = blocks - 1;
    for (; i + 4 <= blocks; i += 4) {
      odd.load(a + (i + 1) * 64, b + (i + 1) * 64);
      even.add_product(sum[0]);
      even.load(a + (i + 2) * 64, b + (i + 2) * 64);
      odd.add_product(sum[1]);
      odd.load(a + (i + 3) * 64, b + (i + 3) * 64);
      even.add_product(sum[2]);
      even.load(a + min(i + 4, last) * 64, b + min(i + 4, last) * 64);
      odd.add_product(sum[3]);
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (i + j >= blocks) break;
    Fragments f;
    f.load(a + (i + j) * 64, b + (i + j) * 64);
    f.add_product(sum[j]);
  }
  if (K % 64) {
    uint32_t a0[4], a1[4], bv[4];
    ldmatrix_x4(a0, a + blocks * 64);
    ldmatrix_x4(a1, a + blocks * 64 + 16);
    ldmatrix_x4(bv, b + blocks * 64);
    float d[2][4] = {};
    mma_bf16(d[0], a0, bv[0], bv[1]);
    mma_bf16(d[1], a1, bv[2], bv[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[3][j] += d[0][j] + d[1][j];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j] = (sum[0][j] + sum[1][j]) + (sum[2][j] + sum[3][j]);
}

// The next (up to) eight pairs out of the bits of `left`, packed a byte each.
__device__ __forceinline__ unsigned long long take_eight(unsigned long long& left, int& count) {
  unsigned long long list = 0;
  for (count = 0; count < 8 && left != 0; ++count) {
    list |= (unsigned long long)(__ffsll((long long)left) - 1) << (8 * count);
    left &= left - 1;
  }
  return list;
}
__device__ __forceinline__ int pair_at(unsigned long long list, int i) { return (int)(list >> (8 * i)) & 63; }

// act[pair] of every pair: tiles of eight hidden channels (the gate's rows, then the up projection's under them), or (PLAIN) of
// sixteen, of a chosen expert.
template <bool PLAIN>
__global__ void __launch_bounds__((kMostStages + 1) * 32)
moe_gate_up_stream_kernel(const bf16* __restrict__ h, long long ldh, const bf16* __restrict__ w_gate_up, const int* __restrict__ chosen,
                          bf16* __restrict__ act, int pairs, int top, int C, int F, int experts, const float* __restrict__ in_weights,
                          int plain, int stages) {
  constexpr int WIDE = PLAIN ? kTileRows : kTileRows / 2;  // hidden channels of a tile
  extern __shared__ __align__(128) unsigned char smem_bytes[];
  __shared__ Chosen picked;
  __shared__ Ring ring;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pitch = C + kPad, stage_elems = kTileRows * pitch, tokens = pairs / top;
  bf16* stage0 = reinterpret_cast<bf16*>(smem_bytes);
  bf16* x_s = stage0 + (size_t)stages * stage_elems;  // [tokens][pitch]
  ring_init(ring, stages);
  sort_out(picked, chosen, pairs, experts);
  const int tiles_of = (F + WIDE - 1) / WIDE, total = picked.used * tiles_of;
  if (warp == stages) {
    int s = 0, turn = 0;
    for (int id = blockIdx.x; id < total; id += gridDim.x) {
      if (turn && !ring_wait(ring, &ring.empty[s], (turn & 1) ^ 1, 1)) break;
      const int at = id / tiles_of, f0 = (id - at * tiles_of) * WIDE, live = min(WIDE, F - f0);
      const bf16* src = w_gate_up + ((size_t)picked.experts[at] * (PLAIN ? F : 2 * F) + f0) * C;
      if (lane == 0) mbar_expect_tx(&ring.full[s], (PLAIN ? 1 : 2) * live * C * (unsigned)sizeof(bf16));
      __syncwarp();
      const int row = lane % WIDE;
      if (lane < kTileRows && row < live)
        bulk_load(stage0 + (size_t)s * stage_elems + lane * pitch, src + ((size_t)row + (lane < WIDE ? 0 : F)) * C,
                  C * (unsigned)sizeof(bf16), &ring.full[s]);
      if (++s == stages) { s = 0; ++turn; }
    }
  } else {
    const int per_row = C / 8;
    for (int i = tid; i < tokens * per_row; i += stages * 32)
      *reinterpret_cast<uint4*>(x_s + (size_t)(i / per_row) * pitch + (i % per_row) * 8) =
          *reinterpret_cast<const uint4*>(h + (size_t)(i / per_row) * ldh + (i % per_row) * 8);
    asm volatile("bar.sync 2, %0;" ::"r"(stages * 32) : "memory");
    const int g = lane >> 2, t = lane & 3;
    int turn = 0;
    for (int id = blockIdx.x + warp * gridDim.x; id < total; id += stages * gridDim.x, ++turn) {
      const int at = id / tiles_of, f0 = (id - at * tiles_of) * WIDE;
      unsigned long long left = picked.pairs[at];
      if (!ring_wait(ring, &ring.full[warp], turn & 1, 2)) break;
      while (left != 0) {
        int count;
        const unsigned long long list = take_eight(left, count);
        float acc[4];
        tile_product(stage0 + (size_t)warp * stage_elems, pitch, x_s + (size_t)(pair_at(list, min(lane & 7, count - 1)) / top) * pitch, C,
                     lane, acc);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int p = 2 * t + j, pair = pair_at(list, min(p, count - 1));
          const float scale = in_weights != nullptr ? in_weights[pair] : 1.f;
          const float upper = acc[j] * scale, lower = acc[2 + j] * scale;
          bf16* dst = act + (size_t)pair * F + f0 + g;
          if (p < count && f0 + g < F) dst[0] = from_f32<bf16>(PLAIN ? plain_activation(upper, plain) : silu_f(upper) * lower);
          if (PLAIN && p < count && f0 + 8 + g < F) dst[8] = from_f32<bf16>(plain_activation(lower, plain));
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ring.empty[warp]);
    }
  }
  ring_lost(ring);
}

// The weighted sums of every token for the block's `channels` (at most 16) output channels: per chosen expert (and eight of its
// pairs) a stage holds the channels' rows of its matrix and the pairs' activations; the pairs' sums stay in shared memory
// until all experts have passed, and then a thread per (token, channel) adds them in the order of the choice.
__global__ void __launch_bounds__((kMostStages + 1) * 32)
moe_down_stream_kernel(const bf16* __restrict__ h, long long ldh, const bf16* __restrict__ w_down, const int* __restrict__ chosen,
                       const float* __restrict__ weights, const bf16* __restrict__ act, float* __restrict__ out, int pairs, int top, int C,
                       int F, int experts, float* __restrict__ x, const float* __restrict__ a_res, const float* __restrict__ ls_a,
                       const float* __restrict__ ls_b, float mult, const float* __restrict__ shared,
                       const float* __restrict__ shared_gate, long long ldsg, int channels, int stages) {
  extern __shared__ __align__(128) unsigned char smem_bytes[];
  __shared__ Chosen picked;
  __shared__ Ring ring;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = blockIdx.x * channels, live = min(channels, C - c0);
  // a stage: `channels` rows of the matrix, then eight rows for the pairs (the product's tile of 16 rows runs on into those
  // where the channels are fewer: what it makes of them is not looked at)
  const int pitch = F + kPad, stage_elems = max(channels + 8, kTileRows) * pitch;
  bf16* stage0 = reinterpret_cast<bf16*>(smem_bytes);
  float* dots = reinterpret_cast<float*>(stage0 + (size_t)stages * stage_elems);  // [pairs][channels]
  ring_init(ring, stages);
  sort_out(picked, chosen, pairs, experts);
  if (warp == stages) {
    int s = 0, turn = 0;
    bool lost = false;
    for (int at = 0; at < picked.used && !lost; ++at) {
      unsigned long long left = picked.pairs[at];
      while (left != 0) {
        if (turn && !ring_wait(ring, &ring.empty[s], (turn & 1) ^ 1, 3)) { lost = true; break; }
        int count;
        const unsigned long long list = take_eight(left, count);
        bf16* dst = stage0 + (size_t)s * stage_elems;
        const unsigned row = F * (unsigned)sizeof(bf16);
        if (lane == 0) mbar_expect_tx(&ring.full[s], (live + count) * row);
        __syncwarp();
        if (lane < live)
          bulk_load(dst + (size_t)lane * pitch, w_down + ((size_t)picked.experts[at] * C + c0 + lane) * F, row, &ring.full[s]);
        else if (lane >= 16 && lane - 16 < count)
          bulk_load(dst + (size_t)(channels + lane - 16) * pitch, act + (size_t)pair_at(list, lane - 16) * F, row, &ring.full[s]);
        if (++s == stages) { s = 0; ++turn; }
      }
    }
  } else {
    const int g = lane >> 2, t = lane & 3;
    int next = 0, turn = 0;  // the stage that the next tile lies in
    bool lost = false;
    for (int at = 0; at < picked.used && !lost; ++at) {
      unsigned long long left = picked.pairs[at];
      while (left != 0) {
        int count;
        const unsigned long long list = take_eight(left, count);
        const bool mine = next == warp;
        if (++next == stages) next = 0;
        if (!mine) continue;
        if (!ring_wait(ring, &ring.full[warp], turn & 1, 4)) { lost = true; break; }
        ++turn;
        const bf16* tile = stage0 + (size_t)warp * stage_elems;
        float acc[4];
        tile_product(tile, pitch, tile + (size_t)(channels + min(lane & 7, count - 1)) * pitch, F, lane, acc);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int p = 2 * t + (j & 1), r = g + (j >> 1) * 8;
          if (p < count && r < live) dots[pair_at(list, p) * channels + r] = acc[j];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ring.empty[warp]);
      }
    }
  }
  __syncthreads();
  if (*(volatile int*)&ring.abort) {
    ring_lost(ring);
    return;
  }
  for (int i = tid; i < pairs / top * live; i += blockDim.x) {
    const int n = i / live, j = i % live, c = c0 + j;
    float total = 0.f;
    for (int k = 0; k < top; ++k) {
      const int pair = n * top + k;
      const float g = weights != nullptr ? weights[pair] : 1.f;
      total = fmaf(g, picked.picks[pair] >= experts ? to_f32(h[(size_t)n * ldh + c]) : dots[pair * channels + j], total);
    }
    if (shared != nullptr) total = fmaf(shared_gate != nullptr ? shared_gate[(size_t)n * ldsg] : 1.f, shared[(size_t)n * C + c], total);
    const size_t place = (size_t)n * C + c;
    if (x != nullptr) x[place] = fmaf(mult, fmaf(ls_b ? ls_b[c] : 1.f, total, a_res ? (ls_a ? ls_a[c] : 1.f) * a_res[place] : 0.f), x[place]);
    else out[place] = total;
  }
}

// The shared-memory limit of a kernel, raised once per device.
template <typename K>
int allow_smem(K kernel, bool (&done)[64]) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return (int)cudaErrorInvalidDevice;
  if (!done[device]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
    if (e != cudaSuccess) return (int)e;
    done[device] = true;
  }
  return 0;
}

// Which models' experts the two below take. The lines go by a model's sizes alone, never by how many pairs a step holds, so that
// a token's result has the same bits whatever its company, up to kFewPairs. Measured at 1 to 64 pairs of 16 experts, caches cold
// (us, pair by pair / here):
//   gate and up: two stages must fit beside the rows of the most tokens (rows stay whole in shared memory: C up to 1,192 where a
//   token chooses one expert, 1,792 for two, 2,392 for four, 2,872 for eight). A launch of theirs starts 1 to 2 us later (the choice
//   sorted out, the first rows' way), which one token's experts make up for from C = 1,280 on: four of 1,280 x 1,152 7.2 / 7.8 at
//   one token, 18 / 14 at four, 29 / 17 at eight; 1,536 x 1,536 12.2 / 9.9, 26 / 20 and 41 / 26; of 1,024 x 1,152 6.6 / 7.3, 16 / 13
//   and 24 / 16, of 768 x 1,152 5.4 / 7.2, 13 / 13 and 21 / 16, of 1,024 x 128 3 / 4, 5 / 5 and 6 / 6.
//   down: a copy being 65 ns at least, rows want length and a token more than one expert: four of 1,024 x 960 13.1 / 7.1, 14 / 12
//   and 22 / 15, of 1,536 x 1,152 11 / 7.8, 14 / 14 and 22 / 18; but of 1,536 x 768 8.4 / 7.3, 11 / 13 and 16 / 17; two of
//   2,048 x 1,152 6.9 / 6.4, 12 / 11 and 17 / 14, of 1,536 x 1,152 6.6 / 6.1, 8.4 / 9.7 and 13 / 14; one of 2,048 x 1,536 4.8 / 6.0,
//   8.6 / 8.5 and 12 / 11.
constexpr int kFewStages = 2;
inline size_t gate_up_row(int C) { return (size_t)(C + kPad) * sizeof(bf16); }
inline bool streams_gate_up(int top, int C, int F, bool plain) {
  return C >= 1024 && C % 32 == 0 && (long long)top * F * (plain ? 1 : 2) >= 2048 &&
         (kFewStages * kTileRows + kFewPairs / top) * gate_up_row(C) <= kStreamSmem;
}
// The channels of a block of the down projection (as many as give every SM one, 16 at most), and a stage of its ring.
inline int down_channels(int C, int sms) { return min(16, (C + sms - 1) / sms); }
inline size_t down_stage(int channels, int F) { return (size_t)max(channels + 8, kTileRows) * (F + kPad) * sizeof(bf16); }
inline bool streams_down(int top, int C, int F, int sms) {
  const int channels = down_channels(C, sms);
  return F % 32 == 0 && ((top >= 4 && C >= 1024 && F >= 960) || (top >= 2 && C >= 1792 && F >= 1152)) &&
         kFewPairs * channels * sizeof(float) + kFewStages * down_stage(channels, F) <= kStreamSmem;
}

static_assert(kStreamSmem + sizeof(Chosen) + sizeof(Ring) + 256 <= 227 * 1024, "with the static arrays, what a block may have");

template <bool PLAIN>
int launch_gate_up_stream(const bf16* h, long long ldh, const bf16* w, const int* chosen, bf16* act, int pairs, int top, int C, int F,
                          int experts, const float* in_weights, int plain, cudaStream_t stream) {
  const size_t stage = kTileRows * gate_up_row(C), xs = (size_t)(pairs / top) * gate_up_row(C);
  const int sms = sm_count();
  if (sms <= 0) return (int)cudaErrorInvalidDevice;
  const int stages = (int)min((size_t)kMostStages, (kStreamSmem - xs) / stage);
  static bool done[64] = {};
  const int err = allow_smem(moe_gate_up_stream_kernel<PLAIN>, done);
  if (err) return err;
  const int wide = PLAIN ? kTileRows : kTileRows / 2;
  const long long tiles = (long long)min(pairs, experts) * ((F + wide - 1) / wide);
  return launch_ordinary(moe_gate_up_stream_kernel<PLAIN>, dim3((unsigned)min((long long)sms, tiles)), dim3((stages + 1) * 32),
                         stages * stage + xs, stream, h, ldh, w, chosen, act, pairs, top, C, F, experts, in_weights, plain, stages);
}

int launch_down_stream(const bf16* h, long long ldh, const bf16* w, const int* chosen, const float* weights, const bf16* act, float* out,
                       int pairs, int top, int C, int F, int experts, float* x, const float* a_res, const float* ls_a,
                       const float* ls_b, float mult, const float* shared, const float* shared_gate, long long ldsg,
                       int sms, cudaStream_t stream) {
  const int channels = down_channels(C, sms);
  const size_t stage = down_stage(channels, F), dots = (size_t)pairs * channels * sizeof(float);
  const int stages = (int)min((size_t)kMostStages, (kStreamSmem - dots) / stage);
  static bool done[64] = {};
  const int err = allow_smem(moe_down_stream_kernel, done);
  if (err) return err;
  return launch_ordinary(moe_down_stream_kernel, dim3((C + channels - 1) / channels), dim3((stages + 1) * 32), stages * stage + dots,
                         stream, h, ldh, w, chosen, weights, act, out, pairs, top, C, F, experts, x, a_res, ls_a, ls_b, mult, shared, shared_gate,
                         ldsg, channels, stages);
}

}  // namespace

// R: the outputs that compete; the matrix has R + extra rows.
AKAS_API int akas_moe_route(const void* h, long long ldh, const float* w, const float* correction, int* chosen, float* weights,
                            int N, int C, int R, int groups, int keep, int top, int dtype, int sigmoid, int renorm, int extra,
                            float* extras, int group_best, float wscale, cudaStream_t stream) {
  if (N <= 0) return 0;
  if (R <= 0 || groups <= 0 || R % groups || keep <= 0 || keep > groups || top <= 0 || top > keep * (R / groups) || extra < 0 || group_best < 1 ||
      (extra > 0 && extras == nullptr))
    return (int)cudaErrorInvalidValue;
  const size_t elem = dtype == AKAS_F32 ? 4 : 2;
  const size_t few_smem = sizeof(float) * (2 * (size_t)(R + extra) + groups + kRouteTokens * kRouteFewOutputs);
  if (N <= 2 * sm_count() && C % 4 == 0 && ldh % 4 == 0 && (uintptr_t)h % (4 * elem) == 0 && (uintptr_t)w % 16 == 0 &&
      few_smem <= 48 * 1024) {
    if (dtype == AKAS_F32)
      return launch_ordinary(moe_route_few_kernel<float>, dim3(N), dim3(kRouteTokens * 32), few_smem, stream, (const float*)h, ldh, w,
                             correction, chosen, weights, C, R, groups, keep, top, sigmoid, renorm, extra, extras, group_best, wscale);
    return launch_ordinary(moe_route_few_kernel<bf16>, dim3(N), dim3(kRouteTokens * 32), few_smem, stream, (const bf16*)h, ldh, w,
                           correction, chosen, weights, C, R, groups, keep, top, sigmoid, renorm, extra, extras, group_best, wscale);
  }
  const size_t smem = sizeof(float) * ((size_t)kRouteTokens * kRouteChunk + 2 * (size_t)kRouteTokens * (R + extra) + (size_t)kRouteTokens * groups +
                                       (size_t)kRouteTokens * kRouteOutputs * kRouteTokens);
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  const dim3 grid((N + kRouteTokens - 1) / kRouteTokens);
  static size_t allowed[64][2] = {};
  int device = 0;
  cudaGetDevice(&device);
  const int which = dtype == AKAS_F32 ? 0 : 1;
  if (smem > 48 * 1024 && device < 64 && allowed[device][which] < smem) {
    const cudaError_t e = which == 0
        ? cudaFuncSetAttribute(moe_route_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
        : cudaFuncSetAttribute(moe_route_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    allowed[device][which] = smem;
  }
  if (dtype == AKAS_F32)
    return launch_ordinary(moe_route_kernel<float>, grid, dim3(kRouteTokens * 32), smem, stream, (const float*)h, ldh, w,
                           correction, chosen, weights, N, C, R, groups, keep, top, sigmoid, renorm, extra, extras, group_best, wscale);
  return launch_ordinary(moe_route_kernel<bf16>, grid, dim3(kRouteTokens * 32), smem, stream, (const bf16*)h, ldh, w, correction,
                         chosen, weights, N, C, R, groups, keep, top, sigmoid, renorm, extra, extras, group_best, wscale);
}

// few: 0 keeps a step of few pairs on the kernels that walk pair by pair (both entries).
AKAS_API int akas_moe_gate_up(const void* h, long long ldh, const void* w_gate_up, const int* chosen, void* act, int N,
                              int top, int C, int F, int experts, int dtype, const float* in_weights, int plain, int few, cudaStream_t stream) {
  if (N <= 0 || top <= 0 || experts <= 0) return 0;
  if (plain < AKAS_PLAIN_NONE || plain > AKAS_PLAIN_SILU) return (int)cudaErrorInvalidValue;
  const int pairs = N * top;
  // few pairs: every chosen expert's rows once through the tensor cores' older path (both sums of a pair, gate and up, end in
  // one thread), where rows start on 16 bytes
  if (few && dtype == AKAS_BF16 && (long long)N * top <= kFewPairs && streams_gate_up(top, C, F, plain != 0) && ldh % 8 == 0 &&
      (uintptr_t)h % 16 == 0 && (uintptr_t)w_gate_up % 16 == 0)
    return plain ? launch_gate_up_stream<true>((const bf16*)h, ldh, (const bf16*)w_gate_up, chosen, (bf16*)act, pairs, top, C, F,
                                               experts, in_weights, plain, stream)
                 : launch_gate_up_stream<false>((const bf16*)h, ldh, (const bf16*)w_gate_up, chosen, (bf16*)act, pairs, top, C, F,
                                                experts, in_weights, plain, stream);
  // warps enough to fill the GPU when the pairs are few (a row of F per warp), fewer and longer-lived when they are many
  const dim3 grid(pairs, max(1, min((F + 7) / 8, pairs >= 4096 ? 2 : pairs >= 256 ? 16 : 256)));
  if (dtype == AKAS_F32)
    return launch_ordinary(moe_gate_up_kernel<float>, grid, dim3(256), 0, stream, (const float*)h, ldh, (const float*)w_gate_up,
                           chosen, (float*)act, pairs, top, C, F, experts, in_weights, plain);
  return launch_ordinary(moe_gate_up_kernel<bf16>, grid, dim3(256), 0, stream, (const bf16*)h, ldh, (const bf16*)w_gate_up,
                         chosen, (bf16*)act, pairs, top, C, F, experts, in_weights, plain);
}

AKAS_API int akas_moe_down(const void* h, long long ldh, const void* w_down, const int* chosen, const float* weights,
                           const void* act, float* out, int N, int top, int C, int F, int experts, int dtype, float* x,
                           const float* a_res, const float* ls_a, const float* ls_b, float mult, const float* shared,
                           const float* shared_gate, long long ldsg, int few, cudaStream_t stream) {
  if (N <= 0) return 0;
  const int sms = sm_count();
  if (few && dtype == AKAS_BF16 && top > 0 && (long long)N * top <= kFewPairs && sms > 0 && streams_down(top, C, F, sms) &&
      (uintptr_t)act % 16 == 0 && (uintptr_t)w_down % 16 == 0)
    return launch_down_stream((const bf16*)h, ldh, (const bf16*)w_down, chosen, weights, (const bf16*)act, out, N * top, top, C, F,
                              experts, x, a_res, ls_a, ls_b, mult, shared, shared_gate, ldsg, sms, stream);
  const dim3 grid(N, max(1, min((C + 7) / 8, N >= 2048 ? 2 : N >= 64 ? 32 : 256)));
  if (dtype == AKAS_F32)
    return launch_ordinary(moe_down_kernel<float>, grid, dim3(256), 0, stream, (const float*)h, ldh, (const float*)w_down, chosen,
                           weights, (const float*)act, out, top, C, F, experts, x, a_res, ls_a, ls_b, mult, shared, shared_gate, ldsg);
  return launch_ordinary(moe_down_kernel<bf16>, grid, dim3(256), 0, stream, (const bf16*)h, ldh, (const bf16*)w_down, chosen,
                         weights, (const bf16*)act, out, top, C, F, experts, x, a_res, ls_a, ls_b, mult, shared, shared_gate, ldsg);
}

// Whether the kernels for few pairs take these sizes (bfloat16): 1 for gate and up, 2 for the down projection, or both.
AKAS_API int akas_moe_few_takes(int top, int C, int F, int plain) {
  if (top <= 0 || top > kFewPairs || C <= 0 || F <= 0) return 0;
  const int sms = sm_count();
  return (streams_gate_up(top, C, F, plain != 0) ? 1 : 0) + (sms > 0 && streams_down(top, C, F, sms) ? 2 : 0);
}

// 0 unless a bounded wait of the kernels for few pairs has run out on the current device. Synchronises with the device.
AKAS_API int akas_moe_status() {
  int status = -1;
  const cudaError_t e = cudaMemcpyFromSymbol(&status, g_moe_status, sizeof(int));
  return e == cudaSuccess ? status : -(int)e;
}
