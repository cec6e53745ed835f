// The kernels a decode step needs between the NF4 linears: token embedding, per-head RMSNorm + RoPE
// + KV-cache append of the new token, and single-token attention over the cache. They follow the
// reference's operators as the Qwen3 NF4 backend calls them (src/models/Qwen3Bnb4Backend.cpp:298-439):
//   ops::embedding_lookup      src/ops/ElementwiseOps.cpp:14-27
//   ops::decode_prepare_qkv    src/ops/ElementwiseOps.cpp:105-215
//   ops::attention_decode      src/ops/AttentionOps.cpp:73-166 (the baseline form: whole window)
// Same arithmetic and the same bf16 roundings (normalised q/k are rounded before the rotation, the
// rotated values again; scores, softmax and the value sum stay fp32), simple kernels: these are
// not on the named hot path, they make the linears' callers runnable end to end.
#include <cooperative_groups.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "nf4_common.cuh"
#include "nf4_internal.h"

namespace nf4 {
namespace {

__global__ void embedding_kernel(const uint16_t* __restrict__ table, const int* __restrict__ ids,
                                 int hidden, long long vocab, uint16_t* __restrict__ out) {
    const int s = blockIdx.x;
    long long id = ids[s];
    if (id < 0 || id >= vocab) id = 0;  // (the reference reads out of range; a clamped row is the safe form)
    const uint16_t* row = table + id * hidden;
    for (int h = threadIdx.x; h < hidden; h += blockDim.x) out[(size_t)s * hidden + h] = row[h];
}

// Sum over 128 threads in the order of a work-group tree reduction (strides 64, 32, ..., 1); every warp
// works it out for itself from the shared values.
__device__ __forceinline__ float block_sum_128(float v, float* scratch) {
    const int lane = threadIdx.x & 31;
    scratch[threadIdx.x] = v;
    __syncthreads();
    float s = (scratch[lane] + scratch[lane + 64]) + (scratch[lane + 32] + scratch[lane + 96]);
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) s += __shfl_down_sync(0xffffffffu, s, stride);
    return __shfl_sync(0xffffffffu, s, 0);
}

// One block of 128 threads per query head and per key head; a key head's block also appends k and v to
// the cache at position pos. The normalised row stays in shared memory until it is rotated (a row too long
// for what every launch may use stays where it is). Latency-bound:
// 4.8 us (cold L2) against 6.3 us with a nine-barrier reduction, the row through global memory and k behind
// q in one block. The kernel is resident while the launch before still writes q, k, v and the position: they
// are read from L2 (a non-coherent load of data that changes in the kernel's lifetime is undefined).
constexpr int kPrepareShared = 20480;  // values of a row that fit beside the 512 static bytes in 48 KB

__global__ void __launch_bounds__(128)
prepare_qkv_kernel(uint16_t* q, uint16_t* k, const uint16_t* v, const float* __restrict__ rope_freq,
                   const uint16_t* __restrict__ q_norm_w, const uint16_t* __restrict__ k_norm_w,
                   uint16_t* __restrict__ k_cache, uint16_t* __restrict__ v_cache, int max_seq_len, int pos,
                   const int* pos_dev, int n_q, int head_dim, float eps) {
    __shared__ float scratch[128];
    extern __shared__ uint16_t prepare_row[];  // [head_dim] up to kPrepareShared
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the launch before may still write q, k, v or the position
    if (pos_dev) pos = __ldcg(pos_dev);
    if (pos < 0 || pos >= max_seq_len) return;  // (the host refuses such a step; nothing is written)
    const bool is_q = (int)blockIdx.x < n_q;
    const int head = is_q ? blockIdx.x : blockIdx.x - n_q;
    uint16_t* x = (is_q ? q : k) + (size_t)head * head_dim;
    uint16_t* normed = head_dim <= kPrepareShared ? prepare_row : x;
    const uint16_t* w = is_q ? q_norm_w : k_norm_w;
    const int half = head_dim / 2;
    float ss = 0.0f;
    for (int d = threadIdx.x; d < head_dim; d += 128) {
        const float a = bf16_bits_to_f32(__ldcg(x + d));
        ss += a * a;
    }
    const float rms = sqrtf(block_sum_128(ss, scratch) / (float)head_dim + eps);
    for (int d = threadIdx.x; d < head_dim; d += 128)
        normed[d] = f32_to_bf16_bits((bf16_bits_to_f32(__ldcg(x + d)) / rms) * bf16_bits_to_f32(w[d]));
    __syncthreads();
    const size_t at = ((size_t)head * max_seq_len + pos) * head_dim;
    for (int d = threadIdx.x; d < half; d += 128) {
        const float angle = (float)pos * rope_freq[d];
        const float c = cosf(angle), s = sinf(angle);
        const float a = bf16_bits_to_f32(normed[d]), b = bf16_bits_to_f32(normed[d + half]);
        const uint16_t lo = f32_to_bf16_bits(a * c - b * s), hi = f32_to_bf16_bits(b * c + a * s);
        x[d] = lo;
        x[d + half] = hi;
        if (!is_q) {
            k_cache[at + d] = lo;
            k_cache[at + d + half] = hi;
        }
    }
    if (is_q) return;
    for (int d = threadIdx.x; d < head_dim; d += 128) v_cache[at + d] = __ldcg(v + (size_t)head * head_dim + d);
}

// One block per query head: scores over the cached positions in shared memory, softmax, value sum.
__global__ void __launch_bounds__(256)
attention_decode_kernel(const uint16_t* __restrict__ q, const uint16_t* __restrict__ k_cache,
                        const uint16_t* __restrict__ v_cache, uint16_t* __restrict__ out,
                        int heads_per_kv, int head_dim, int cached_len, const int* __restrict__ pos_dev,
                        int max_seq_len) {
    extern __shared__ float att_smem[];
    if (pos_dev) cached_len = min(*pos_dev + 1, cached_len);  // (the launch holds `cached_len` scores at most)
    if (cached_len <= 0) return;
    float* qf = att_smem;                  // [head_dim]
    float* score = att_smem + head_dim;    // [cached_len]
    __shared__ float red[8];
    const int head = blockIdx.x, kv_head = head / heads_per_kv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int d = tid; d < head_dim; d += 256) qf[d] = bf16_bits_to_f32(q[(size_t)head * head_dim + d]);
    __syncthreads();
    const float scale = 1.0f / sqrtf((float)head_dim);
    const uint16_t* kb = k_cache + (size_t)kv_head * max_seq_len * head_dim;
    const uint16_t* vb = v_cache + (size_t)kv_head * max_seq_len * head_dim;
    float mx = -1e30f;
    for (int t = tid; t < cached_len; t += 256) {
        const uint16_t* row = kb + (size_t)t * head_dim;
        float sum = 0.0f;
        for (int d = 0; d < head_dim; ++d) sum += qf[d] * bf16_bits_to_f32(row[d]);
        sum *= scale;
        score[t] = sum;
        mx = fmaxf(mx, sum);
    }
    auto block_reduce = [&](float v, bool is_max) {
        for (int sh = 16; sh > 0; sh >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, v, sh);
            v = is_max ? fmaxf(v, o) : v + o;
        }
        if (lane == 0) red[warp] = v;
        __syncthreads();
        float r = red[0];
        for (int w = 1; w < 8; ++w) r = is_max ? fmaxf(r, red[w]) : r + red[w];
        __syncthreads();
        return r;
    };
    mx = block_reduce(mx, true);
    float den = 0.0f;
    for (int t = tid; t < cached_len; t += 256) {
        const float e = __expf(score[t] - mx);
        score[t] = e;
        den += e;
    }
    den = block_reduce(den, false);
    for (int t = tid; t < cached_len; t += 256) score[t] = score[t] / den;
    __syncthreads();
    for (int d = tid; d < head_dim; d += 256) {
        float acc = 0.0f;
        for (int t = 0; t < cached_len; ++t) acc += score[t] * bf16_bits_to_f32(vb[(size_t)t * head_dim + d]);
        out[(size_t)head * head_dim + d] = f32_to_bf16_bits(acc);
    }
}

// The same attention for head sizes 64, 128 and 256 on a cluster of up to eight CTAs per HG query heads
// that share a key/value head, every sum in the order of the kernel above, so that both give the same
// bits (a decode step amplifies a changed rounding layer by layer):
//   scores  each CTA takes a contiguous part of the positions; K rows arrive as 16-byte pieces in shared
//           memory, a thread adds up one row's products, and the score goes to every CTA of the cluster
//   softmax every CTA for all positions (thread t: t, t + 256, ...)
//   values  each CTA takes HD / S dimensions of all positions, one chain of additions per head and
//           dimension; its slice of V streams through two shared-memory tiles, the first one while the
//           scores are computed
// Bound by latency at a decode step's lengths (4 KB per position of eight key/value heads): the value
// chain alone is one dependent addition per position. The one-block-per-head form reads whole rows per
// thread, uncoalesced, on as many SMs as there are heads. Decode step of 36 layers, 32 heads of 128 over
// 1001 positions: 8.58 ms with that form, 2.44 ms with this one.
constexpr int kAttThreads = 256;
constexpr int kAttVBytes = 32768;  // one tile of V
template <int HD>
constexpr int kAttKRows = HD == 256 ? 64 : 128;
template <int HD>
constexpr int kAttKPitch = HD * 2 + 16;  // eight rows' 16-byte pieces fall into different banks

template <int HD, int HG>
size_t attention_cluster_smem(int cached_len) {
    return (size_t)HG * HD * 4 + (size_t)kAttKRows<HD> * kAttKPitch<HD> + 2 * kAttVBytes +
           (size_t)HG * ((size_t)(cached_len + 3) / 4 * 4) * 4;
}

__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <int HD, int HG>
__global__ void __launch_bounds__(kAttThreads)
attention_cluster_kernel(const uint16_t* q, const uint16_t* k_cache, const uint16_t* v_cache, uint16_t* out,
                         int heads_per_kv, int cached_len, const int* pos_dev, int max_seq_len) {
    namespace cg = cooperative_groups;
    constexpr int TK = kAttKRows<HD>, KP = kAttKPitch<HD>;
    extern __shared__ __align__(16) uint8_t att_cl[];
    __shared__ float red[HG][8];
    const int pitch = (cached_len + 3) / 4 * 4;
    float* s_q = reinterpret_cast<float*>(att_cl);                 // [HG][HD]
    uint8_t* s_k = att_cl + HG * HD * 4;                           // [TK][KP]
    uint8_t* s_v = s_k + TK * KP;                                  // two tiles of [rows][dims]
    float* s_score = reinterpret_cast<float*>(s_v + 2 * kAttVBytes);  // [HG][pitch]
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the launch before writes q and the newest position
    // (everything that the launch before may have written is read from L2: __ldcg, cp.async.cg)
    if (pos_dev) cached_len = min(__ldcg(pos_dev) + 1, cached_len);  // (the launch holds `cached_len` scores at most)
    if (cached_len <= 0) return;                              // (the whole grid)
    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int head0 = (int)(blockIdx.x / S) * HG, kv_head = head0 / heads_per_kv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint16_t* kb = k_cache + (size_t)kv_head * max_seq_len * HD;
    const uint16_t* vb = v_cache + (size_t)kv_head * max_seq_len * HD;
    const int per = (cached_len + S - 1) / S;
    const int t_begin = rank * per, t_end = min(cached_len, t_begin + per);
    const int dims = HD / S, TV = kAttVBytes / 2 / dims;
    auto load_k = [&](int t0) {
        const int rows = min(TK, t_end - t0);
        for (int i = tid; i < rows * (HD / 8); i += kAttThreads) {
            const int row = i / (HD / 8), piece = i % (HD / 8);
            cp_async_16(s_k + row * KP + piece * 16, kb + (size_t)(t0 + row) * HD + piece * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto load_v = [&](int tile) {
        const int t0 = tile * TV, rows = min(TV, cached_len - t0), pieces = dims / 8;
        uint8_t* dst = s_v + (tile & 1) * kAttVBytes;
        for (int i = tid; i < rows * pieces; i += kAttThreads) {
            const int row = i / pieces, piece = i - row * pieces;
            cp_async_16(dst + i * 16, vb + (size_t)(t0 + row) * HD + rank * dims + piece * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (t_begin < t_end) load_k(t_begin);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    load_v(0);
    for (int i = tid; i < HG * HD; i += kAttThreads) s_q[i] = bf16_bits_to_f32(__ldcg(q + (size_t)head0 * HD + i));
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster runs

    // ---- scores ----
    const float scale = 1.0f / sqrtf((float)HD);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    for (int t0 = t_begin; t0 < t_end; t0 += TK) {
        if (t0 > t_begin) {
            __syncthreads();
            load_k(t0);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        for (int i = tid; i < TK * HG; i += kAttThreads) {
            const int h = i / TK, t = t0 + i % TK;  // (a warp's threads share the head)
            if (t < t_end) {
                const uint8_t* row = s_k + (i % TK) * KP;
                const float4* qh = reinterpret_cast<const float4*>(s_q + h * HD);
                float sum = 0.0f;
#pragma unroll 4
                for (int d = 0; d < HD / 8; ++d) {
                    const uint4 r = *reinterpret_cast<const uint4*>(row + d * 16);
                    const float4 a = qh[2 * d], b = qh[2 * d + 1];
                    sum = fmaf(a.x, __uint_as_float(r.x << 16), sum);
                    sum = fmaf(a.y, __uint_as_float(r.x & 0xffff0000u), sum);
                    sum = fmaf(a.z, __uint_as_float(r.y << 16), sum);
                    sum = fmaf(a.w, __uint_as_float(r.y & 0xffff0000u), sum);
                    sum = fmaf(b.x, __uint_as_float(r.z << 16), sum);
                    sum = fmaf(b.y, __uint_as_float(r.z & 0xffff0000u), sum);
                    sum = fmaf(b.z, __uint_as_float(r.w << 16), sum);
                    sum = fmaf(b.w, __uint_as_float(r.w & 0xffff0000u), sum);
                }
                sum *= scale;
                for (int c = 0; c < S; ++c) *cluster.map_shared_rank(s_score + h * pitch + t, c) = sum;
            }
        }
    }
    cluster.sync();  // every score is everywhere; nobody looks into another CTA from here on

    // ---- softmax ----
    auto block_reduce = [&](float (&v)[HG], bool is_max) {
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            for (int sh = 16; sh > 0; sh >>= 1) {
                const float o = __shfl_xor_sync(0xffffffffu, v[h], sh);
                v[h] = is_max ? fmaxf(v[h], o) : v[h] + o;
            }
            if (lane == 0) red[h][warp] = v[h];
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            float r = red[h][0];
            for (int w = 1; w < 8; ++w) r = is_max ? fmaxf(r, red[h][w]) : r + red[h][w];
            v[h] = r;
        }
        __syncthreads();
    };
    float mx[HG], den[HG];
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        mx[h] = -1e30f;
        den[h] = 0.0f;
        for (int t = tid; t < cached_len; t += kAttThreads) mx[h] = fmaxf(mx[h], s_score[h * pitch + t]);
    }
    block_reduce(mx, true);
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        for (int t = tid; t < cached_len; t += kAttThreads) {
            const float e = __expf(s_score[h * pitch + t] - mx[h]);
            s_score[h * pitch + t] = e;
            den[h] += e;
        }
    }
    block_reduce(den, false);
#pragma unroll
    for (int h = 0; h < HG; ++h)
        for (int t = tid; t < cached_len; t += kAttThreads) s_score[h * pitch + t] = s_score[h * pitch + t] / den[h];

    // ---- values ----
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // (at most 4 * 256 dimensions and 256 threads)
    const int tiles = (cached_len + TV - 1) / TV;
    for (int tile = 0; tile < tiles; ++tile) {
        if (tile + 1 < tiles) {
            load_v(tile + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int t0 = tile * TV, rows = min(TV, cached_len - t0);
        const uint16_t* v = reinterpret_cast<const uint16_t*>(s_v + (tile & 1) * kAttVBytes);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = tid + u * kAttThreads;
            if (i < HG * dims) {
                const float* ph = s_score + (i / dims) * pitch + t0;
                const uint16_t* vd = v + i % dims;
                float a = acc[u];
                int t = 0;
#pragma unroll 4
                for (; t + 4 <= rows; t += 4) {
                    const float4 w = *reinterpret_cast<const float4*>(ph + t);
                    a = fmaf(w.x, bf16_bits_to_f32(vd[t * dims]), a);
                    a = fmaf(w.y, bf16_bits_to_f32(vd[(t + 1) * dims]), a);
                    a = fmaf(w.z, bf16_bits_to_f32(vd[(t + 2) * dims]), a);
                    a = fmaf(w.w, bf16_bits_to_f32(vd[(t + 3) * dims]), a);
                }
                for (; t < rows; ++t) a = fmaf(ph[t], bf16_bits_to_f32(vd[t * dims]), a);
                acc[u] = a;
            }
        }
        __syncthreads();  // the tile's buffer is filled again two tiles later
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = tid + u * kAttThreads;
        if (i < HG * dims) out[(size_t)(head0 + i / dims) * HD + rank * dims + i % dims] = f32_to_bf16_bits(acc[u]);
    }
}

constexpr size_t kAttMaxSmem = 220 * 1024;
constexpr size_t kAttTwoSmem = 112 * 1024;  // two CTAs on an SM (228 KB, 1 KB and the static arrays of each among them)

struct AttentionPlan {
    void (*fn)(const uint16_t*, const uint16_t*, const uint16_t*, uint16_t*, int, int, const int*, int) = nullptr;
    size_t smem = 0;
    int hg = 0;
    cudaError_t err = cudaSuccess;
};

// What the launches of one instantiation on one device need to know, found out once.
struct AttentionDevice {
    cudaError_t err = cudaSuccess;
    int fit[2][9] = {};  // clusters of 1, 2, 4 or 8 CTAs that run at once, one or two CTAs on an SM
};

template <int HD, int HG>
const AttentionDevice& attention_device(int device) {
    static std::once_flag once[64];
    static AttentionDevice devs[64];
    AttentionDevice& d = devs[device & 63];
    std::call_once(once[device & 63], [&] {
        d.err = cudaFuncSetAttribute(attention_cluster_kernel<HD, HG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kAttMaxSmem);
        for (int two = 0; two < 2; ++two) {
            for (unsigned ctas = 1; ctas <= 8 && d.err == cudaSuccess; ctas *= 2) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(ctas * 1024);
                cfg.blockDim = dim3(kAttThreads);
                cfg.dynamicSmemBytes = two ? kAttTwoSmem : kAttMaxSmem;
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = ctas;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
                cfg.attrs = attr;
                cfg.numAttrs = 1;
                d.err = cudaOccupancyMaxActiveClusters(&d.fit[two][ctas], attention_cluster_kernel<HD, HG>, &cfg);
            }
        }
    });
    return d;
}

// Takes the group size if it divides the heads and holds the scores; whether all of its clusters run at once.
template <int HD, int HG>
bool attention_plan(int heads, int per_kv, int cached_len, unsigned ctas, int device, AttentionPlan* plan) {
    const size_t smem = attention_cluster_smem<HD, HG>(cached_len);
    if (per_kv % HG != 0 || smem > kAttMaxSmem) return false;
    const AttentionDevice& d = attention_device<HD, HG>(device);
    plan->fn = attention_cluster_kernel<HD, HG>;
    plan->smem = smem;
    plan->hg = HG;
    plan->err = d.err;
    return heads / HG <= d.fit[smem <= kAttTwoSmem ? 1 : 0][ctas];
}

// Head groups of four, two or one share what they read, but a CTA's work is a chain of latencies: the smallest
// group whose clusters all run at once, and where none does the largest that holds its scores. us per launch by
// group size (24 caches in turn, best of the rule in brackets):
//   32 heads of 128 on 8 key/value heads, 1000 positions: 18.9, 16.7, 13.8 in groups of four, two, one (one);
//   4000 positions, where 15 clusters of eight run at once: 58.8, 98.7, 118 (four); 64 heads, 1000 positions:
//   36.6, 18.3 in groups of four and two (two)
template <int HD>
bool attention_plan_of(int heads, int per_kv, int cached_len, unsigned ctas, int device, AttentionPlan* plan) {
    plan->fn = nullptr;
    if (!attention_plan<HD, 1>(heads, per_kv, cached_len, ctas, device, plan) &&
        !attention_plan<HD, 2>(heads, per_kv, cached_len, ctas, device, plan))
        attention_plan<HD, 4>(heads, per_kv, cached_len, ctas, device, plan);
    return plan->fn != nullptr;
}

struct BackendDevGuard {
    int prev = -1;
    cudaError_t err = cudaSuccess;
    explicit BackendDevGuard(int device) {
        err = cudaGetDevice(&prev);
        if (err == cudaSuccess && prev != device) err = cudaSetDevice(device);
    }
    ~BackendDevGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

}  // namespace
}  // namespace nf4

using nf4::fail;

AILA_NF4_API AilaNf4Status aila_embedding_lookup(const void* table_bf16, int64_t vocab_size,
                                                 const int32_t* token_ids_device, int seq_len,
                                                 int hidden_size, void* out_bf16, int device,
                                                 void* stream) {
    if (!table_bf16 || !token_ids_device || !out_bf16) return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "NULL argument");
    if (seq_len <= 0 || hidden_size <= 0 || vocab_size <= 0)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "seq_len, hidden_size and vocab_size must be positive");
    nf4::BackendDevGuard guard(device);
    if (guard.err != cudaSuccess) return nf4::cuda_fail(guard.err, "cudaSetDevice");
    nf4::embedding_kernel<<<(unsigned)seq_len, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint16_t*>(table_bf16), token_ids_device, hidden_size, (long long)vocab_size,
        static_cast<uint16_t*>(out_bf16));
    NF4_CUDA(cudaGetLastError());
    return AILA_NF4_OK;
}

AILA_NF4_API AilaNf4Status aila_decode_prepare_qkv(void* q_bf16, void* k_bf16, const void* v_bf16,
                                                   const float* rope_freq, const void* q_norm_weight_bf16,
                                                   const void* k_norm_weight_bf16, void* k_cache_bf16,
                                                   void* v_cache_bf16, int max_seq_len, int start_pos,
                                                   const int32_t* position_device, int num_heads_q,
                                                   int num_kv_heads, int head_dim, float eps, int device,
                                                   void* stream) {
    if (!q_bf16 || !k_bf16 || !v_bf16 || !rope_freq || !q_norm_weight_bf16 || !k_norm_weight_bf16 ||
        !k_cache_bf16 || !v_cache_bf16)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "NULL argument");
    if (num_heads_q <= 0 || num_kv_heads <= 0 || num_kv_heads > num_heads_q || num_heads_q % num_kv_heads != 0)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "query heads must be a positive multiple of the key/value heads");
    if (head_dim <= 0 || head_dim % 2 != 0) return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "head_dim must be positive and even");
    if (start_pos < 0 || start_pos >= max_seq_len)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "context window exceeded (start_pos=" + std::to_string(start_pos) +
                                                       ", max_seq_len=" + std::to_string(max_seq_len) + ")");
    nf4::BackendDevGuard guard(device);
    if (guard.err != cudaSuccess) return nf4::cuda_fail(guard.err, "cudaSetDevice");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(num_heads_q + num_kv_heads));
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = head_dim <= nf4::kPrepareShared ? (size_t)head_dim * 2 : 0;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nf4::overlapped_launches() ? 1 : 0;
    NF4_CUDA(cudaLaunchKernelEx(&cfg, nf4::prepare_qkv_kernel, static_cast<uint16_t*>(q_bf16),
                                static_cast<uint16_t*>(k_bf16), static_cast<const uint16_t*>(v_bf16), rope_freq,
                                static_cast<const uint16_t*>(q_norm_weight_bf16),
                                static_cast<const uint16_t*>(k_norm_weight_bf16),
                                static_cast<uint16_t*>(k_cache_bf16), static_cast<uint16_t*>(v_cache_bf16), max_seq_len,
                                start_pos, position_device, num_heads_q, head_dim, eps));
    return AILA_NF4_OK;
}

AILA_NF4_API AilaNf4Status aila_attention_decode(const void* q_bf16, const void* k_cache_bf16,
                                                 const void* v_cache_bf16, void* out_bf16, int num_heads,
                                                 int num_kv_heads, int head_dim, int cached_len,
                                                 const int32_t* position_device, int max_seq_len, int device,
                                                 void* stream) {
    if (!q_bf16 || !k_cache_bf16 || !v_cache_bf16 || !out_bf16) return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "NULL argument");
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads != 0 || head_dim <= 0)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "query heads must be a positive multiple of the key/value heads");
    if (cached_len <= 0 || cached_len > max_seq_len)
        return fail(AILA_NF4_ERR_INVALID_ARGUMENT, "cached_len out of range");
    const size_t smem = ((size_t)cached_len + (size_t)head_dim) * sizeof(float);
    if (smem > 200 * 1024)
        return fail(AILA_NF4_ERR_UNSUPPORTED, "attention_decode keeps one score per cached position in shared memory: "
                                              "at most about 51,000 positions");
    nf4::BackendDevGuard guard(device);
    if (guard.err != cudaSuccess) return nf4::cuda_fail(guard.err, "cudaSetDevice");
    // Rows of K and V in 16-byte pieces need the alignment. CTAs per head group: one per 64 positions the
    // launch can hold, at most the portable cluster of eight.
    const unsigned ctas = cached_len <= 64 ? 1 : cached_len <= 128 ? 2 : cached_len <= 256 ? 4 : 8;
    nf4::AttentionPlan plan;
    const int per_kv = num_heads / num_kv_heads;
    if (((reinterpret_cast<uintptr_t>(k_cache_bf16) | reinterpret_cast<uintptr_t>(v_cache_bf16)) & 15) == 0 &&
        ((head_dim == 64 && nf4::attention_plan_of<64>(num_heads, per_kv, cached_len, ctas, device, &plan)) ||
         (head_dim == 128 && nf4::attention_plan_of<128>(num_heads, per_kv, cached_len, ctas, device, &plan)) ||
         (head_dim == 256 && nf4::attention_plan_of<256>(num_heads, per_kv, cached_len, ctas, device, &plan)))) {
        if (plan.err != cudaSuccess) return nf4::cuda_fail(plan.err, "cudaFuncSetAttribute(attention)");
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(num_heads / plan.hg) * ctas);
        cfg.blockDim = dim3(nf4::kAttThreads);
        cfg.dynamicSmemBytes = plan.smem;
        cfg.stream = static_cast<cudaStream_t>(stream);
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = nf4::overlapped_launches() ? 2 : 1;
        NF4_CUDA(cudaLaunchKernelEx(&cfg, plan.fn, static_cast<const uint16_t*>(q_bf16),
                                    static_cast<const uint16_t*>(k_cache_bf16),
                                    static_cast<const uint16_t*>(v_cache_bf16), static_cast<uint16_t*>(out_bf16),
                                    per_kv, cached_len, position_device, max_seq_len));
        return AILA_NF4_OK;
    }
    static bool raised[64] = {false};
    if (smem > 48 * 1024 && device >= 0 && device < 64 && !raised[device]) {
        NF4_CUDA(cudaFuncSetAttribute(nf4::attention_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      200 * 1024));
        raised[device] = true;
    }
    nf4::attention_decode_kernel<<<(unsigned)num_heads, 256, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint16_t*>(q_bf16), static_cast<const uint16_t*>(k_cache_bf16),
        static_cast<const uint16_t*>(v_cache_bf16), static_cast<uint16_t*>(out_bf16), num_heads / num_kv_heads,
        head_dim, cached_len, position_device, max_seq_len);
    NF4_CUDA(cudaGetLastError());
    return AILA_NF4_OK;
}
