// Causal grouped-query attention over the paged cache on the CUDA cores, float32
// arithmetic, for any head size: one block of threads per (token, query head).
//
// The keys a token sees are the positions lo..pos of its own request, lo = 0 or
// pos+1-window.  They are taken in blocks of 32 counted from lo, which go to PARTS parts in turn, each with an online
// softmax of its own, and the parts are put together in their order, so the result at a position depends
// neither on how the tokens were cut into steps nor on which pages hold them.  This kernel is the attention of the
// true 32-bit path and the fallback of the bfloat16 path.
//
// Options beside the plain softmax over a causal window: `chunk` > 0 hides every key whose
// position lies in another block of `chunk` positions than the query's (blocks counted from
// position 0 of the request); SIGMOID replaces the softmax by unnormalised weights
// sigmoid(score * head_scale[h] + head_bias[h]) (either array may be missing); `gate` multiplies
// the output element by element with sigmoid(gate[token, head * vd + d]), or, with GATE_PER_HEAD, every
// element of head h with the one number sigmoid(gate[token, h]).  The values may have another size than the
// keys (`vcache.head_dim`), and with v_pool == k_pool and a value size of at most the key size they are the
// leading dimensions of the cached keys (a latent cache: one vector per token serves as key and as value).
// Reference: hostfog/hfee internal/llm/forward.go:146-178 (scores scaled after the
// dot, softmax over 0..pos, weighted sum of values), internal/ggml/ops.go:136-150.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int PARTS = 8;         // results that are put together: block b of 32 keys goes to part b mod PARTS
constexpr int MAX_HD = 640;      // key size
constexpr int MAX_VD = 512;      // value size
constexpr int GATE_NONE = 0, GATE_ELEMENT = 1, GATE_PER_HEAD = 2;

// Bound by the latency of its loads: a block of 32 keys is one trip for the keys (a lane's key is read 16 bytes at a time, and its
// share of a value four numbers at a time, where VEC says that rows start on 16-byte boundaries) and the values of AHEAD keys at a time,
// the first of them requested with the keys; values are read without a condition (a key or column that is not there reads one that is,
// and is not used), since a branch around each load ends the overlap.  A decode step has few (token, head) pairs, so the parts of one
// pair run side by side in eight warps (two tokens behind prompts of 150: 7.6 us a layer, with one warp a pair 52); the many pairs of a
// prompt portion have two warps each, since most of eight would have nothing to do.  DPL, the value dimensions a lane owns, is the
// smallest that covers the value size; the more it owns, the fewer keys it takes ahead, or the registers leave too few warps an SM:
// 285 tokens, 8 heads of 256 on 2: 136 us (float32), 90 us (bfloat16); eight ahead, keys one number at a time and conditional
// values took 308 and 579, one key at a time in one warp a pair 526 and 503.
template <int N, typename T> struct alignas(N * sizeof(T)) PieceOf { T v[N]; };

template <typename T, bool SIGMOID, int DPL, bool VEC, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 2 ? 32 / DPL : DPL == 2 ? 4 : 1)
attention_simt_kernel(const T* __restrict__ q, int ld_q, const T* __restrict__ k_pool,
                      const T* __restrict__ v_pool, PagedCache cache, PagedCache vcache, int vd,
                      const int* __restrict__ positions,
                      const int* __restrict__ slot_of_token, T* __restrict__ out, int ld_o, int n, int heads,
                      float scale, int window, int chunk, const float* __restrict__ head_scale,
                      const float* __restrict__ head_bias, const T* __restrict__ gate, long long ld_gate,
                      int gate_mode, const float* __restrict__ dist_r1, const float* __restrict__ dist_r2, float out_scale,
                      const float* __restrict__ sink, int keep_first, float softcap) {
  constexpr int AHEAD = DPL <= 4 ? 8 : 32 / DPL;
  constexpr int VW = VEC ? (DPL < 4 ? DPL : 4) : 1, KW = 16 / (int)sizeof(T);      // numbers of a piece of a value, of a key
  pdl_wait();
  pdl_launch_dependents();
  __shared__ __align__(16) float q_s[MAX_HD];
  __shared__ float o_s[PARTS][DPL * 32], m_s[PARTS], l_s[PARTS];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int i = blockIdx.x / heads, h = blockIdx.x % heads;
  int hd = cache.head_dim;
  int kvh = h / (heads / cache.kv_heads);
  int pos = positions[i], slot = slot_of_token[i];
  int lo = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;
  if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
  const float h_scale = (SIGMOID && head_scale != nullptr) ? head_scale[h] : 1.f;
  const float h_bias = (SIGMOID && head_bias != nullptr) ? head_bias[h] : 0.f;
  const float r1 = dist_r1 != nullptr ? dist_r1[h] : 0.f, r2 = dist_r1 != nullptr ? dist_r2[h] : 0.f;

  const T* qrow = q + (long long)i * ld_q + (long long)h * hd;
  for (int d = threadIdx.x; d < hd; d += WARPS * 32) q_s[d] = to_f32<T>(qrow[d]);
  __syncthreads();

  // the first keep_first positions stay visible behind the window: they are visited first, [0, kept), then [lo, pos]
  const int kept = min(keep_first, lo);
  const int front_blocks = (kept + 31) / 32, blocks = front_blocks + (pos - lo) / 32 + 1;
  const int parts = min(PARTS, blocks);
  float o[DPL], m = 0.f, l = 0.f;
  for (int part = warp; part < parts; part += WARPS) {
#pragma unroll
    for (int j = 0; j < DPL; ++j) o[j] = 0.f;
    // a sink is one more term exp(sink[h]) of the denominator that has no key and no value
    const bool sunk = !SIGMOID && sink != nullptr && part == 0;
    m = sunk ? sink[h] : -INFINITY;
    l = sunk ? 1.f : 0.f;
    for (int block = part; block < blocks; block += PARTS) {
      const bool front = block < front_blocks;
      const int base = front ? block * 32 : lo + (block - front_blocks) * 32;
      const int end = front ? kept - 1 : pos;                  // last key of the range this block of 32 lies in
      const int count = min(32, end + 1 - base);
      const int key = base + lane;
      const long long k_at = key <= end ? paged_offset(cache, slot, key, kvh) : 0, v_at = key <= end ? paged_offset(vcache, slot, key, kvh) : 0;
      float v[AHEAD][DPL];
      auto request = [&](int t0) {
#pragma unroll
        for (int t = 0; t < AHEAD; ++t) {
          const T* vr = v_pool + __shfl_sync(0xffffffffu, v_at, min(t0 + t, count - 1));
#pragma unroll
          for (int j = 0; j < DPL / VW; ++j) {
            const int d = (lane + 32 * j) * VW;
            const PieceOf<VW, T> x = *reinterpret_cast<const PieceOf<VW, T>*>(vr + (d < vd ? d : 0));
#pragma unroll
            for (int e = 0; e < VW; ++e) v[t][j * VW + e] = to_f32<T>(x.v[e]);
          }
        }
      };
      request(0);
      float s = -INFINITY;
      if (key <= end) {
        const T* kr = k_pool + k_at;
        float acc = 0.f;
        if constexpr (VEC) {
#pragma unroll 4
          for (int d = 0; d < hd; d += KW) {
            const PieceOf<KW, T> x = *reinterpret_cast<const PieceOf<KW, T>*>(kr + d);
#pragma unroll
            for (int e = 0; e < KW; ++e) acc = fmaf(q_s[d + e], to_f32<T>(x.v[e]), acc);
          }
        } else {
          for (int d = 0; d < hd; ++d) acc = fmaf(q_s[d], to_f32<T>(kr[d]), acc);
        }
        s = acc * scale;
        if (softcap > 0.f) s = softcap * tanhf(s / softcap);
        if (dist_r1 != nullptr) s -= r1 * log1pf(r2 * (float)(pos - key));
      }
      float p;
      if constexpr (SIGMOID) {
        p = key <= end ? 1.f / (1.f + expf(-(s * h_scale + h_bias))) : 0.f;
      } else {
        // a part may have seen no finite score yet (its block can be one key): its weights are 0, not exp(inf - inf)
        const float m_new = fmaxf(m, warp_max(s)), m_use = m_new == -INFINITY ? 0.f : m_new;
        p = key <= end ? expf(s - m_use) : 0.f;
        const float alpha = expf(m - m_use);    // exp(-inf) = 0 on the first block
        l = l * alpha + warp_sum(p);
#pragma unroll
        for (int j = 0; j < DPL; ++j) o[j] *= alpha;
        m = m_new;
      }
      for (int t0 = 0; t0 < count; t0 += AHEAD) {
        if (t0 > 0) request(t0);
#pragma unroll
        for (int t = 0; t < AHEAD; ++t) {
          if (t0 + t >= count) break;
          const float pt = __shfl_sync(0xffffffffu, p, t0 + t);
#pragma unroll
          for (int j = 0; j < DPL; ++j) o[j] = fmaf(pt, v[t][j], o[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < DPL; ++j) o_s[part][lane + 32 * j] = o[j];
    if (lane == 0) { m_s[part] = m; l_s[part] = l; }
  }
  __syncthreads();
  if (warp != 0) return;
  m = m_s[0];
  for (int w = 1; w < parts; ++w) m = fmaxf(m, m_s[w]);
  if (m == -INFINITY) m = 0.f;
  l = 0.f;
#pragma unroll
  for (int j = 0; j < DPL; ++j) o[j] = 0.f;
  for (int w = 0; w < parts; ++w) {
    const float share = SIGMOID ? 1.f : expf(m_s[w] - m);
    l += l_s[w] * share;
#pragma unroll
    for (int j = 0; j < DPL; ++j) o[j] = fmaf(o_s[w][lane + 32 * j], share, o[j]);
  }
  T* orow = out + (long long)i * ld_o + (long long)h * vd;
  float inv = (SIGMOID ? 1.f : 1.f / l) * out_scale;
  const T* grow = gate_mode == GATE_ELEMENT ? gate + (long long)i * ld_gate + (long long)h * vd : nullptr;
  if (gate_mode == GATE_PER_HEAD) inv *= 1.f / (1.f + expf(-to_f32<T>(gate[(long long)i * ld_gate + h])));
#pragma unroll
  for (int j = 0; j < DPL; ++j) {
    const int d = (lane + 32 * (j / VW)) * VW + j % VW;
    if (d < vd) {
      float v = o[j] * inv;
      if (grow != nullptr) v *= 1.f / (1.f + expf(-to_f32<T>(grow[d])));
      orow[d] = from_f32<T>(v);
    }
  }
}

}  // namespace

namespace {
template <typename T, bool SIGMOID, int DPL, bool VEC>
void launch_one(const void* q, int ld_q, const void* k_pool, const void* v_pool, const PagedCache& c, const PagedCache& vc,
                int vd, const int* positions, const int* slot_of_token, void* out, int ld_o, int n, int heads, float scale,
                int window, int chunk, const float* head_scale, const float* head_bias, const void* gate, long long ld_gate,
                int gate_mode, const float* dist_r1, const float* dist_r2, float out_scale, const float* sink, int keep_first,
                float softcap, cudaStream_t stream) {
  auto run = [&](auto warps) {
    constexpr int WARPS = decltype(warps)::value;
    hfee_launch(attention_simt_kernel<T, SIGMOID, DPL, VEC, WARPS>, dim3((unsigned)n * (unsigned)heads), dim3(WARPS * 32), 0, stream, (const T*)q,
                ld_q, (const T*)k_pool, (const T*)v_pool, c, vc, vd, positions, slot_of_token, (T*)out, ld_o, n, heads, scale, window, chunk,
                head_scale, head_bias, (const T*)gate, ld_gate, gate_mode, dist_r1, dist_r2, out_scale, sink, keep_first, softcap);
  };
  if ((long long)n * heads <= 8LL * hfee_sm_count()) run(std::integral_constant<int, 8>{});      // a full SM holds eight such blocks
  else run(std::integral_constant<int, 2>{});
}

template <typename T, bool SIGMOID, typename... Args>
void launch_weights(const void* q, int ld_q, const void* k_pool, const void* v_pool, const PagedCache& c, const PagedCache& vc, int vd,
                    Args... args) {
  // whole 16-byte pieces of keys, whole pieces of four values (rows follow one another in a page, so pools and sizes decide)
  const bool vec = c.head_dim % (16 / (int)sizeof(T)) == 0 && vd % 4 == 0 && ((uintptr_t)k_pool | (uintptr_t)v_pool) % 16 == 0;
  auto with = [&](auto dpl) {
    constexpr int DPL = decltype(dpl)::value;
    if (vec) launch_one<T, SIGMOID, DPL, true>(q, ld_q, k_pool, v_pool, c, vc, vd, args...);
    else launch_one<T, SIGMOID, DPL, false>(q, ld_q, k_pool, v_pool, c, vc, vd, args...);
  };
  if (vd <= 64) with(std::integral_constant<int, 2>{});
  else if (vd <= 128) with(std::integral_constant<int, 4>{});
  else if (vd <= 256) with(std::integral_constant<int, 8>{});
  else with(std::integral_constant<int, MAX_VD / 32>{});
}

template <typename T, typename... Args>
void launch_simt(int sigmoid, Args... args) {
  if (sigmoid) launch_weights<T, true>(args...);
  else launch_weights<T, false>(args...);
}
}  // namespace

// weights: 0 = softmax over the visible keys, 1 = sigmoid(score * head_scale[h] + head_bias[h]) per key.
// value_dim: size of a value; v_pool is [pages][kv_heads][page_size][value_dim], or, with values_in_keys, the key
// pool itself, whose leading value_dim dimensions are the values.  gate_mode: 0 none, 1 one number per output
// element ([n, heads * value_dim]), 2 one number per head ([n, heads]); the output is multiplied by its sigmoid.
// dist_r1, dist_r2 (per head, or both null): r1[h] * ln(1 + r2[h] * (query position - key position)) is taken off the
// score before the softmax.  out_scale multiplies the output.  sink (per head, or null): the softmax's denominator also
// holds exp(sink[h]).  keep_first: that many positions from the start stay visible behind a window.  softcap > 0: the scaled
// score becomes softcap * tanh(score / softcap).
HFEE_API int hfee_attention_simt_capped(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                          const int* block_table, int max_pages, int page_size, const int* positions,
                                          const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                          int head_dim, int value_dim, int values_in_keys, float scale, int window,
                                          int chunk, int weights, const float* head_scale, const float* head_bias,
                                          const void* gate, long long ld_gate, int gate_mode, const float* dist_r1,
                                          const float* dist_r2, float out_scale, const float* sink, int keep_first,
                                          float softcap, int dtype, cudaStream_t stream) {
  HFEE_REQUIRE(keep_first >= 0 && (keep_first == 0 || chunk == 0), "attention_simt: kept first positions go with a window");
  HFEE_REQUIRE(sink == nullptr || weights == 0, "attention_simt: a sink goes with the softmax");
  HFEE_REQUIRE((dist_r1 == nullptr) == (dist_r2 == nullptr), "attention_simt: the distance penalty needs both of its arrays");
  HFEE_REQUIRE(dist_r1 == nullptr || weights == 0, "attention_simt: the distance penalty goes with the softmax");
  if (n == 0) return HFEE_OK;
  HFEE_REQUIRE(head_dim > 0 && head_dim <= MAX_HD, "attention_simt: head_dim %d is outside 1..%d", head_dim, MAX_HD);
  HFEE_REQUIRE(value_dim > 0 && value_dim <= MAX_VD, "attention_simt: value_dim %d is outside 1..%d", value_dim, MAX_VD);
  HFEE_REQUIRE(!values_in_keys || value_dim <= head_dim, "attention_simt: values inside keys need value_dim <= head_dim");
  HFEE_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0,
               "attention_simt: heads %d must be a multiple of kv_heads %d", heads, kv_heads);
  HFEE_REQUIRE(page_size > 0 && max_pages > 0, "attention_simt: bad cache sizes");
  HFEE_REQUIRE(window >= 0 && chunk >= 0 && (weights == 0 || weights == 1), "attention_simt: bad mask or weight option");
  HFEE_REQUIRE(gate_mode >= GATE_NONE && gate_mode <= GATE_PER_HEAD && (gate_mode == GATE_NONE) == (gate == nullptr),
               "attention_simt: gate and gate_mode %d do not fit", gate_mode);
  HFEE_REQUIRE(gate_mode != GATE_ELEMENT || ld_gate >= (long long)heads * value_dim, "attention_simt: ld_gate is too small");
  HFEE_REQUIRE(gate_mode != GATE_PER_HEAD || ld_gate >= heads, "attention_simt: ld_gate is too small");
  PagedCache c, vc;
  HFEE_REQUIRE(make_paged_cache(&c, block_table, max_pages, page_size, kv_heads, head_dim),
               "page_size %d must be a power of two", page_size);
  if (values_in_keys) {
    vc = c;
    v_pool = k_pool;
  } else {
    make_paged_cache(&vc, block_table, max_pages, page_size, kv_heads, value_dim);
  }
  if (dtype == HFEE_F32)
    launch_simt<float>(weights, q, ld_q, k_pool, v_pool, c, vc, value_dim, positions, slot_of_token, out, ld_o, n, heads, scale,
                       window, chunk, head_scale, head_bias, gate, ld_gate, gate_mode, dist_r1, dist_r2, out_scale, sink, keep_first,
                       softcap, stream);
  else if (dtype == HFEE_BF16)
    launch_simt<__nv_bfloat16>(weights, q, ld_q, k_pool, v_pool, c, vc, value_dim, positions, slot_of_token, out, ld_o, n, heads,
                               scale, window, chunk, head_scale, head_bias, gate, ld_gate, gate_mode, dist_r1, dist_r2,
                               out_scale, sink, keep_first, softcap, stream);
  else
    return hfee_fail(HFEE_ERR_ARG, "attention_simt: unknown dtype %d", dtype);
  return hfee_check_launch("attention_simt");
}

HFEE_API int hfee_attention_simt_sink(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                      const int* block_table, int max_pages, int page_size, const int* positions,
                                      const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                      int head_dim, int value_dim, int values_in_keys, float scale, int window,
                                      int chunk, int weights, const float* head_scale, const float* head_bias,
                                      const void* gate, long long ld_gate, int gate_mode, const float* dist_r1,
                                      const float* dist_r2, float out_scale, const float* sink, int dtype,
                                      cudaStream_t stream) {
  return hfee_attention_simt_capped(q, ld_q, k_pool, v_pool, block_table, max_pages, page_size, positions, slot_of_token, out,
                                    ld_o, n, heads, kv_heads, head_dim, value_dim, values_in_keys, scale, window, chunk,
                                    weights, head_scale, head_bias, gate, ld_gate, gate_mode, dist_r1, dist_r2, out_scale, sink,
                                    0, 0.f, dtype, stream);
}

HFEE_API int hfee_attention_simt_distance(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                          const int* block_table, int max_pages, int page_size, const int* positions,
                                          const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                          int head_dim, int value_dim, int values_in_keys, float scale, int window,
                                          int chunk, int weights, const float* head_scale, const float* head_bias,
                                          const void* gate, long long ld_gate, int gate_mode, const float* dist_r1,
                                          const float* dist_r2, float out_scale, int dtype, cudaStream_t stream) {
  return hfee_attention_simt_sink(q, ld_q, k_pool, v_pool, block_table, max_pages, page_size, positions, slot_of_token, out,
                                  ld_o, n, heads, kv_heads, head_dim, value_dim, values_in_keys, scale, window, chunk,
                                  weights, head_scale, head_bias, gate, ld_gate, gate_mode, dist_r1, dist_r2, out_scale,
                                  nullptr, dtype, stream);
}

HFEE_API int hfee_attention_simt_general(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                         const int* block_table, int max_pages, int page_size, const int* positions,
                                         const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                         int head_dim, int value_dim, int values_in_keys, float scale, int window,
                                         int chunk, int weights, const float* head_scale, const float* head_bias,
                                         const void* gate, long long ld_gate, int gate_mode, int dtype,
                                         cudaStream_t stream) {
  return hfee_attention_simt_distance(q, ld_q, k_pool, v_pool, block_table, max_pages, page_size, positions, slot_of_token,
                                      out, ld_o, n, heads, kv_heads, head_dim, value_dim, values_in_keys, scale, window,
                                      chunk, weights, head_scale, head_bias, gate, ld_gate, gate_mode, nullptr, nullptr,
                                      1.f, dtype, stream);
}

HFEE_API int hfee_attention_simt_masked(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                        const int* block_table, int max_pages, int page_size, const int* positions,
                                        const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                        int head_dim, float scale, int window, int chunk, int weights,
                                        const float* head_scale, const float* head_bias, const void* gate,
                                        long long ld_gate, int dtype, cudaStream_t stream) {
  HFEE_REQUIRE(head_dim > 0 && head_dim <= MAX_VD, "attention_simt: head_dim %d is outside 1..%d", head_dim, MAX_VD);
  return hfee_attention_simt_general(q, ld_q, k_pool, v_pool, block_table, max_pages, page_size, positions, slot_of_token,
                                     out, ld_o, n, heads, kv_heads, head_dim, head_dim, 0, scale, window, chunk, weights,
                                     head_scale, head_bias, gate, ld_gate, gate != nullptr ? GATE_ELEMENT : GATE_NONE,
                                     dtype, stream);
}

HFEE_API int hfee_attention_simt(const void* q, int ld_q, const void* k_pool, const void* v_pool,
                                 const int* block_table, int max_pages, int page_size, const int* positions,
                                 const int* slot_of_token, void* out, int ld_o, int n, int heads, int kv_heads,
                                 int head_dim, float scale, int window, int dtype, cudaStream_t stream) {
  return hfee_attention_simt_masked(q, ld_q, k_pool, v_pool, block_table, max_pages, page_size, positions, slot_of_token,
                                    out, ld_o, n, heads, kv_heads, head_dim, scale, window, 0, 0, nullptr, nullptr,
                                    nullptr, 0, dtype, stream);
}
