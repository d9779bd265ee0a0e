// Mixture-of-experts block on one device: router, grouping of the rows by expert, grouped GEMMs and
// the weighted combination, without a host synchronisation and with one launch per step for all
// experts. mm_moe_fwd / mm_moe_bwd queue the whole pass; the caller supplies one workspace.
//
//   plan       : [start | count | first tile] per expert, see gemm_grouped.cuh
//   pos[t*k+j] : row of the grouped buffers that holds choice j of token t
//   row_of[r]  : its inverse, -1 for the zero rows that fill a group up to a multiple of 64
//
// What bounded the loop over the experts that this replaces: on small blocks its ~200 launches and 16 host
// reads, on large ones fp32 weight gradients (zeroed, added and converted: 6 ms of 20) and six GEMMs per
// expert with their tails. Forward + backward, one B200: 4096 tokens, D 4096, F 14336, 8 experts, 2
// choices 20.9 -> 11.6 ms, 9.7 now (8.1 ms of it in the five grouped GEMMs and the forward's two); 300 tokens, D 512,
// F 1024, 4 experts 2.97 -> 0.27 ms.
//
// Rows of a group are in token order whatever the timing, so the results are reproducible.
//
// The backward pass needs neither the experts' outputs nor scaled output gradients: with
// u = dy W_down the gate's gradient is <u, h>, the activation's is gate * u, and the weight gradient
// of W_down is dy^T (gate * h). That is five grouped GEMMs instead of six and one rounding less.
#include "gemm_grouped.cuh"

namespace mm {

constexpr int ML_MAX_K = 4;
constexpr int ML_DWR_SPLIT = 16;

__device__ __forceinline__ float ml_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// a before b in descending order with NaN first, as torch.topk orders them
__device__ __forceinline__ bool ml_before(float a, float b) { return isnan(a) ? !isnan(b) : a > b; }

// Router: fp32 logits, the k largest (ties: lowest index) and the softmax over them. A block takes
// ML_TOK tokens and its four warps a quarter of the row each, so that the router weights - E * D * 2 bytes
// from L2 per block, which bound the kernel - serve eight tokens (4096 tokens, D 4096, 8 experts: a
// block's forward + backward, which routes twice, 10.16 -> 10.08 ms against two tokens per warp).
constexpr int ML_TOK = 8;
__global__ void __launch_bounds__(128)
    ml_route_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wr, int T, int D, int E, int k,
                    int* __restrict__ idx, float* __restrict__ gates) {
  __shared__ float part[4][ML_TOK][GG_MAX_E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * ML_TOK;
  const int nvec = D / 8;
  const uint4* rows[ML_TOK];
#pragma unroll
  for (int t = 0; t < ML_TOK; ++t) rows[t] = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(min(t0 + t, T - 1)) * D);
  for (int e0 = 0; e0 < E; e0 += 8) {
    float acc[ML_TOK][8];
#pragma unroll
    for (int t = 0; t < ML_TOK; ++t)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[t][j] = 0.f;
    for (int v = warp * 32 + lane; v < nvec; v += 128) {
      uint4 xv[ML_TOK];
#pragma unroll
      for (int t = 0; t < ML_TOK; ++t) xv[t] = rows[t][v];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (e0 + j < E) {
          const uint4 w = __ldg(reinterpret_cast<const uint4*>(wr + static_cast<int64_t>(e0 + j) * D) + v);
          const float2 w0 = unpack_bf16(w.x), w1 = unpack_bf16(w.y), w2 = unpack_bf16(w.z), w3 = unpack_bf16(w.w);
#pragma unroll
          for (int t = 0; t < ML_TOK; ++t) {
            const float2 a = unpack_bf16(xv[t].x), b = unpack_bf16(xv[t].y), c = unpack_bf16(xv[t].z), d = unpack_bf16(xv[t].w);
            acc[t][j] += ((a.x * w0.x + a.y * w0.y) + (b.x * w1.x + b.y * w1.y)) + ((c.x * w2.x + c.y * w2.y) + (d.x * w3.x + d.y * w3.y));
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < ML_TOK; ++t)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float s = ml_warp_sum(acc[t][j]);
        if (lane == 0 && e0 + j < E) part[warp][t][e0 + j] = s;
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ML_TOK * E; i += 128) {
    const int t = i / E, e = i - t * E;
    part[0][t][e] = (part[0][t][e] + part[1][t][e]) + (part[2][t][e] + part[3][t][e]);
  }
  __syncthreads();
  if (threadIdx.x < min(ML_TOK, T - t0)) {
    const float* lg = part[0][threadIdx.x];
    const int64_t out = static_cast<int64_t>(t0 + threadIdx.x) * k;
    int chosen[ML_MAX_K];
    float val[ML_MAX_K];
    for (int j = 0; j < k; ++j) {
      int best = -1;
      for (int e = 0; e < E; ++e) {
        bool taken = false;
        for (int i = 0; i < j; ++i) taken |= chosen[i] == e;
        if (!taken && (best < 0 || ml_before(lg[e], lg[best]))) best = e;
      }
      chosen[j] = best;
      val[j] = lg[best];
    }
    float den = 0.f;
    const float mx = val[0];
    for (int j = 0; j < k; ++j) { val[j] = expf(val[j] - mx); den += val[j]; }
    for (int j = 0; j < k; ++j) {
      idx[out + j] = chosen[j];
      gates[out + j] = val[j] / den;
    }
  }
}

// One block per expert: histogram of all choices, then this expert's rows in token order.
__global__ void __launch_bounds__(1024)
    ml_plan_kernel(const int* __restrict__ idx, int n, int E, int* __restrict__ plan, int* __restrict__ pos,
                   int* __restrict__ row_of) {
  __shared__ int hist[GG_MAX_E];
  __shared__ int warp_cnt[32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < GG_MAX_E) hist[threadIdx.x] = 0;
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const int v = i < n ? idx[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, v);
    if (v >= 0 && lane == __ffs(same) - 1) atomicAdd(&hist[v], __popc(same));
  }
  __syncthreads();
  int start = 0;
  for (int i = 0; i < e; ++i) start += (hist[i] + GG_PAD - 1) / GG_PAD * GG_PAD;
  if (e == 0 && threadIdx.x == 0) {
    int s = 0, tiles = 0;
    for (int i = 0; i < GG_MAX_E; ++i) {
      const int c = i < E ? hist[i] : 0;
      plan[GG_START + i] = s;
      plan[GG_COUNT + i] = c;
      plan[GG_TILE + i] = tiles;
      s += (c + GG_PAD - 1) / GG_PAD * GG_PAD;
      tiles += (c + 255) / 256;
    }
    plan[GG_TILE + GG_MAX_E] = tiles;
  }
  // every thread owns a run of consecutive choices: ranks follow from a scan of the runs' counts
  const int run = (n + 1023) / 1024;
  const int i0 = min(n, static_cast<int>(threadIdx.x) * run), i1 = min(n, i0 + run);
  int mine = 0;
  for (int i = i0; i < i1; ++i) mine += idx[i] == e;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warp_cnt[warp] = incl;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += warp_cnt[w];
  int at = start + before + incl - mine;
  for (int i = i0; i < i1; ++i)
    if (idx[i] == e) {
      pos[i] = at;
      row_of[at] = i;
      ++at;
    }
  const int c = hist[e], padded = (c + GG_PAD - 1) / GG_PAD * GG_PAD;
  for (int i = c + threadIdx.x; i < padded; i += 1024) row_of[start + i] = -1;
}

__device__ __forceinline__ int ml_total_rows(const int* plan, int E) {
  return plan[GG_START + E - 1] + (plan[GG_COUNT + E - 1] + GG_PAD - 1) / GG_PAD * GG_PAD;
}

// Rows of x (and of a second tensor) in grouped order. One block per row; memory bound.
__global__ void __launch_bounds__(128)
    ml_gather_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ xs, const __nv_bfloat16* __restrict__ y,
                     __nv_bfloat16* __restrict__ ys, const int* __restrict__ row_of, const int* __restrict__ plan, int E, int k,
                     int D) {
  const int r = blockIdx.x;
  if (r >= ml_total_rows(plan, E)) return;
  const int f = row_of[r];
  const int nvec = D / 8;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const int64_t src = static_cast<int64_t>(f < 0 ? 0 : f / k) * nvec, dst = static_cast<int64_t>(r) * nvec;
  const uint4* x4 = reinterpret_cast<const uint4*>(x) + src;
  const uint4* y4 = reinterpret_cast<const uint4*>(y) + src;
  for (int v = threadIdx.x; v < nvec; v += 128) {
    reinterpret_cast<uint4*>(xs)[dst + v] = f < 0 ? zero : x4[v];
    if (ys) reinterpret_cast<uint4*>(ys)[dst + v] = f < 0 ? zero : y4[v];
  }
}

// h = silu(gate) * up over the grouped rows; one block per row, memory bound.
__global__ void __launch_bounds__(256)
    ml_swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h, const int* __restrict__ plan, int E,
                     int F) {
  const int r = blockIdx.x;
  if (r >= ml_total_rows(plan, E)) return;
  const int fv = F / 8;
  const uint4* g4 = reinterpret_cast<const uint4*>(gu) + static_cast<int64_t>(r) * 2 * fv;
  uint4* h4 = reinterpret_cast<uint4*>(h) + static_cast<int64_t>(r) * fv;
#pragma unroll 4
  for (int v = threadIdx.x; v < fv; v += 256) {
    const uint4 g = g4[v], u = g4[fv + v];
    const uint32_t gg[4] = {g.x, g.y, g.z, g.w}, uu[4] = {u.x, u.y, u.z, u.w};
    uint32_t oo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = unpack_bf16(gg[j]), b = unpack_bf16(uu[j]);
      oo[j] = pack_bf16(a.x / (1.f + __expf(-a.x)) * b.x, a.y / (1.f + __expf(-a.y)) * b.y);
    }
    h4[v] = make_uint4(oo[0], oo[1], oo[2], oo[3]);
  }
}

// One block per grouped row: reads gate | up and u = dy W_down; overwrites them with the gradients of
// gate | up (for gate * u) and with gate_weight * h, and writes <u, h>, the gradient of the gate weight.
__global__ void __launch_bounds__(256)
    ml_swiglu_bwd_kernel(__nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ u, const float* __restrict__ gates,
                         float* __restrict__ dgates, const int* __restrict__ row_of, const int* __restrict__ plan, int E, int F) {
  __shared__ float red[8];
  const int r = blockIdx.x;
  if (r >= ml_total_rows(plan, E)) return;
  const int f = row_of[r];
  const int fv = F / 8;
  uint4* g4 = reinterpret_cast<uint4*>(gu) + static_cast<int64_t>(r) * 2 * fv;
  uint4* u4 = reinterpret_cast<uint4*>(u) + static_cast<int64_t>(r) * fv;
  if (f < 0) {          // a zero row stays one whatever the weights hold
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int v = threadIdx.x; v < fv; v += 256) g4[v] = g4[fv + v] = u4[v] = zero;
    return;
  }
  const float w = gates[f];
  float dot = 0.f;
#pragma unroll 2
  for (int v = threadIdx.x; v < fv; v += 256) {
    const uint4 g = g4[v], p = g4[fv + v], d = u4[v];
    const uint32_t gg[4] = {g.x, g.y, g.z, g.w}, pp[4] = {p.x, p.y, p.z, p.w}, dd[4] = {d.x, d.y, d.z, d.w};
    uint32_t og[4], ou[4], oh[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = unpack_bf16(gg[j]), b = unpack_bf16(pp[j]), c = unpack_bf16(dd[j]);
      const float s0 = 1.f / (1.f + __expf(-a.x)), s1 = 1.f / (1.f + __expf(-a.y));
      const float i0 = a.x * s0, i1 = a.y * s1;              // silu(gate)
      const float h0 = i0 * b.x, h1 = i1 * b.y;
      dot += c.x * h0 + c.y * h1;
      const float e0 = w * c.x, e1 = w * c.y;
      og[j] = pack_bf16(e0 * b.x * (s0 * (1.f + a.x * (1.f - s0))), e1 * b.y * (s1 * (1.f + a.y * (1.f - s1))));
      ou[j] = pack_bf16(e0 * i0, e1 * i1);
      oh[j] = pack_bf16(w * h0, w * h1);
    }
    g4[v] = make_uint4(og[0], og[1], og[2], og[3]);
    g4[fv + v] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
    u4[v] = make_uint4(oh[0], oh[1], oh[2], oh[3]);
  }
  dot = ml_warp_sum(dot);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < 8; ++i) s += red[i];
    dgates[f] = s;
  }
}

// y[t] = sum_j weight_j * rows[pos_j] in fp32, choices in ascending order of their experts. Forward:
// the weights are the gates. Backward (dl given): weights of 1, plus the router's part
// sum_j dl_j * wr[expert_j], where dl is the gradient of the chosen logits; it is stored for ml_dwr_kernel.
__global__ void __launch_bounds__(128)
    ml_combine_kernel(const __nv_bfloat16* __restrict__ rows, const int* __restrict__ idx, const int* __restrict__ pos,
                      const float* __restrict__ gates, const float* __restrict__ dgates, const __nv_bfloat16* __restrict__ wr,
                      float* __restrict__ dl, __nv_bfloat16* __restrict__ y, int k, int D) {
  const int64_t t = blockIdx.x;
  int e[ML_MAX_K], p[ML_MAX_K];
  float w[ML_MAX_K];
  float mean = 0.f;
  for (int j = 0; j < k; ++j) {
    e[j] = idx[t * k + j];
    p[j] = pos[t * k + j];
    w[j] = gates[t * k + j];
    if (dl) mean += w[j] * dgates[t * k + j];
  }
  if (dl)
    for (int j = 0; j < k; ++j) {
      w[j] = w[j] * (dgates[t * k + j] - mean);
      if (threadIdx.x == 0) dl[t * k + j] = w[j];
    }
  for (int i = 1; i < k; ++i)
    for (int j = i; j > 0 && e[j] < e[j - 1]; --j) {
      const int te = e[j], tp = p[j];
      const float tw = w[j];
      e[j] = e[j - 1]; p[j] = p[j - 1]; w[j] = w[j - 1];
      e[j - 1] = te; p[j - 1] = tp; w[j - 1] = tw;
    }
  const int nvec = D / 8;
  for (int v = threadIdx.x; v < nvec; v += 128) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int j = 0; j < k; ++j) {
      const uint4 a = reinterpret_cast<const uint4*>(rows)[static_cast<int64_t>(p[j]) * nvec + v];
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
      const float s = dl ? 1.f : w[j];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = unpack_bf16(aw[i]);
        acc[2 * i] += s * f.x;
        acc[2 * i + 1] += s * f.y;
      }
    }
    if (dl)
      for (int j = 0; j < k; ++j) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(wr) + static_cast<int64_t>(e[j]) * nvec + v);
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = unpack_bf16(aw[i]);
          acc[2 * i] += w[j] * f.x;
          acc[2 * i + 1] += w[j] * f.y;
        }
      }
    reinterpret_cast<uint4*>(y)[t * nvec + v] = make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]),
                                                           pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
  }
}

// Router weight gradient: partial[s][e][:] = sum over slice s of the group's rows of dl[row] * x[row].
__global__ void __launch_bounds__(128)
    ml_dwr_kernel(const __nv_bfloat16* __restrict__ xs, const float* __restrict__ dl, const int* __restrict__ row_of,
                  const int* __restrict__ plan, float* __restrict__ partial, int E, int D) {
  const int e = blockIdx.z, s = blockIdx.y;
  const int v = blockIdx.x * 128 + threadIdx.x, nvec = D / 8;
  if (v >= nvec) return;
  const int c = plan[GG_COUNT + e], first = plan[GG_START + e];
  const int r0 = static_cast<int>(static_cast<int64_t>(c) * s / ML_DWR_SPLIT);
  const int r1 = static_cast<int>(static_cast<int64_t>(c) * (s + 1) / ML_DWR_SPLIT);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int r = first + r0; r < first + r1; ++r) {
    const float w = dl[row_of[r]];
    const uint4 a = reinterpret_cast<const uint4*>(xs)[static_cast<int64_t>(r) * nvec + v];
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpack_bf16(aw[i]);
      acc[2 * i] += w * f.x;
      acc[2 * i + 1] += w * f.y;
    }
  }
  float4* o = reinterpret_cast<float4*>(partial + (static_cast<int64_t>(s) * E + e) * D + v * 8);
  o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

__global__ void __launch_bounds__(256)
    ml_dwr_sum_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dwr, int64_t n) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll
  for (int p = 0; p < ML_DWR_SPLIT; ++p) s += partial[p * n + i];
  dwr[i] = __float2bfloat16(s);
}

// Workspace of one pass; every part starts on a 256-byte boundary.
struct MoeSpace {
  int64_t used = 0;
  char* base;
  int *idx, *pos, *row_of, *plan;
  float *gates, *dgates, *dl, *dwr_part;
  __nv_bfloat16 *xs, *ys, *gu, *h, *rows;
  int cap;
  template <class P>
  void take(P*& p, int64_t count) {
    p = reinterpret_cast<P*>(base + used);
    used += (count * static_cast<int64_t>(sizeof(P)) + 255) / 256 * 256;
  }
  MoeSpace(void* ws, int T, int D, int F, int E, int k, bool backward) : base(static_cast<char*>(ws)) {
    const int64_t n = static_cast<int64_t>(T) * k;
    cap = static_cast<int>(n + static_cast<int64_t>(E) * (GG_PAD - 1) + GG_PAD - 1) / GG_PAD * GG_PAD;
    take(idx, n);
    take(pos, n);
    take(row_of, cap);
    take(plan, GG_PLAN);
    take(gates, n);
    take(xs, static_cast<int64_t>(cap) * D);
    take(gu, static_cast<int64_t>(cap) * 2 * F);
    take(h, static_cast<int64_t>(cap) * F);
    take(rows, static_cast<int64_t>(cap) * D);
    dgates = dl = dwr_part = nullptr;
    ys = nullptr;
    if (backward) {
      take(ys, static_cast<int64_t>(cap) * D);
      take(dgates, n);
      take(dl, n);
      take(dwr_part, static_cast<int64_t>(ML_DWR_SPLIT) * E * D);
    }
  }
};

static int moe_check(int T, int D, int F, int E, int k) {
  if (T < 1 || D < 8 || D % 8 || F < 8 || F % 8 || E < 1 || E > GG_MAX_E || k < 1 || k > ML_MAX_K || k > E) return -2;
  if (static_cast<int64_t>(T) * k + static_cast<int64_t>(E) * GG_PAD > (1 << 30)) return -2;
  return 0;
}

static int moe_group(const MoeSpace& w, const void* x, const void* wr, const void* dy, int T, int D, int E, int k,
                     cudaStream_t stream) {
  ml_route_kernel<<<(T + ML_TOK - 1) / ML_TOK, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(wr), T,
                                                   D, E, k, w.idx, w.gates);
  ml_plan_kernel<<<E, 1024, 0, stream>>>(w.idx, T * k, E, w.plan, w.pos, w.row_of);
  ml_gather_kernel<<<w.cap, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), w.xs, static_cast<const __nv_bfloat16*>(dy),
                                              dy ? w.ys : nullptr, w.row_of, w.plan, E, k, D);
  MM_LAUNCHED(3);
  return 0;
}

}  // namespace mm

extern "C" {

// Bytes of workspace for a pass over T tokens, or -2 when the sizes are outside what these kernels take.
int64_t mm_moe_workspace(int T, int D, int F, int E, int k, int backward) {
  using namespace mm;
  if (moe_check(T, D, F, E, k)) return -2;
  return MoeSpace(nullptr, T, D, F, E, k, backward != 0).used;
}

// The router alone: the k experts of every token and their gates, as the two passes below choose them.
// x [T, D], wr [E, D] bf16, contiguous and 16-byte aligned; idx, gates [T, k].
int mm_moe_route(const void* x, const void* wr, int* idx, float* gates, int T, int D, int E, int k, cudaStream_t stream) {
  using namespace mm;
  const int rc = moe_check(T, D, 8, E, k);
  if (rc) return rc;
  ml_route_kernel<<<(T + ML_TOK - 1) / ML_TOK, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x),
                                                                static_cast<const __nv_bfloat16*>(wr), T, D, E, k, idx, gates);
  MM_LAUNCHED(1);
  return 0;
}

// y[T, D] = sum over the k chosen experts of gate * W_down (silu(W_gate x) * W_up x). All tensors bf16,
// contiguous and 16-byte aligned: x [T, D], wr [E, D], wgu [E, 2, F, D], wdown [E, D, F]; ws: 256-byte aligned.
int mm_moe_fwd(const void* x, const void* wr, const void* wgu, const void* wdown, void* y, void* ws, int T, int D, int F, int E,
               int k, cudaStream_t stream) {
  using namespace mm;
  int rc = moe_check(T, D, F, E, k);
  if (rc) return rc;
  const MoeSpace w(ws, T, D, F, E, k, false);
  if ((rc = moe_group(w, x, wr, nullptr, T, D, E, k, stream))) return rc;
  if ((rc = grouped_rows(w.xs, wgu, 0, w.gu, w.cap, E, 2 * F, D, w.plan, stream))) return rc;
  ml_swiglu_kernel<<<w.cap, 256, 0, stream>>>(w.gu, w.h, w.plan, E, F);
  if ((rc = grouped_rows(w.h, wdown, 0, w.rows, w.cap, E, D, F, w.plan, stream))) return rc;
  ml_combine_kernel<<<T, 128, 0, stream>>>(w.rows, w.idx, w.pos, w.gates, nullptr, nullptr, nullptr,
                                           static_cast<__nv_bfloat16*>(y), k, D);
  MM_LAUNCHED(2);
  return 0;
}

// Gradients of mm_moe_fwd (routing and expert activations are computed again).
int mm_moe_bwd(const void* dy, const void* x, const void* wr, const void* wgu, const void* wdown, void* dx, void* dwr, void* dwgu,
               void* dwdown, void* ws, int T, int D, int F, int E, int k, cudaStream_t stream) {
  using namespace mm;
  int rc = moe_check(T, D, F, E, k);
  if (rc) return rc;
  const MoeSpace w(ws, T, D, F, E, k, true);
  if ((rc = moe_group(w, x, wr, dy, T, D, E, k, stream))) return rc;
  if ((rc = grouped_rows(w.xs, wgu, 0, w.gu, w.cap, E, 2 * F, D, w.plan, stream))) return rc;
  if ((rc = grouped_rows(w.ys, wdown, 1, w.h, w.cap, E, F, D, w.plan, stream))) return rc;
  ml_swiglu_bwd_kernel<<<w.cap, 256, 0, stream>>>(w.gu, w.h, w.gates, w.dgates, w.row_of, w.plan, E, F);
  if ((rc = grouped_wgrad(w.ys, w.h, dwdown, w.cap, E, D, F, w.plan, stream))) return rc;
  if ((rc = grouped_wgrad(w.gu, w.xs, dwgu, w.cap, E, 2 * F, D, w.plan, stream))) return rc;
  if ((rc = grouped_rows(w.gu, wgu, 1, w.rows, w.cap, E, D, 2 * F, w.plan, stream))) return rc;
  ml_combine_kernel<<<T, 128, 0, stream>>>(w.rows, w.idx, w.pos, w.gates, w.dgates, static_cast<const __nv_bfloat16*>(wr), w.dl,
                                           static_cast<__nv_bfloat16*>(dx), k, D);
  ml_dwr_kernel<<<dim3((D / 8 + 127) / 128, ML_DWR_SPLIT, E), 128, 0, stream>>>(w.xs, w.dl, w.row_of, w.plan, w.dwr_part, E, D);
  const int64_t n = static_cast<int64_t>(E) * D;
  ml_dwr_sum_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(w.dwr_part, static_cast<__nv_bfloat16*>(dwr), n);
  MM_LAUNCHED(4);
  return 0;
}

}  // extern "C"
