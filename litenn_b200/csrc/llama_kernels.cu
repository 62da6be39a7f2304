// Glue kernels of the LLaMA decoder around the quantized linears: embedding row
// dequantization, RMSNorm, interleaved RoPE, fp16 KV cache, attention, SwiGLU, residual
// adds and greedy argmax.  Semantics follow the reference graph builders:
//   RMSNorm   x / sqrt(mean(x^2) + eps) * w, statistics in double
//             (src/LiteNN/ComputePrimitives.h:795-821)
//   RoPE      interleaved pairs (x[2i], x[2i+1]), angle = pos * theta^(-2i/d), tables made in
//             double and cast to fp32, rotation in fp32 (src/LiteNN/Layer/RoPE.h:22-114)
//   attention scores = q.k * 1/sqrt(head_dim), causal, max-shifted softmax, probs.V
//             (src/LiteNN/Layer/FlashAttnExt.h:100-229; tools/gguf/LLaMABuilder.cpp:350-404);
//             GQA maps head h to kv head h / (heads / kv_heads) (LLaMABuilder.cpp:524)
//   SwiGLU    down(silu(gate(x)) * up(x)), silu(x) = x / (1 + exp(-x))
//             (src/LiteNN/Layer/SwiGLU.h:54-64; Layer/Activation.h:20-33,52-59)
// The KV cache holds rotated keys and values as fp16 (the benchmark configuration's choice;
// the reference keeps them in the model dtype, LLaMABuilder.cpp:847-849).
// These kernels are latency-sized (one token of a 4096-wide model); the weight streaming
// lives in qmm_gemv.cu / qmm_gemm.cu.
#include <algorithm>

#include <cuda_bf16.h>
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include "llama_device.cuh"
#include "llama_kernels.h"
#include "qmm_layout.cuh"
#include "qmm_pack.cuh"

namespace qmm {

namespace {

__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_sync()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ double block_sum_double(double v, double* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    }
    __syncthreads();
    if (lane == 0) {
        red[warp] = v;
    }
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < nw; ++i) {
        t += red[i];
    }
    return t;
}

// ---- decode (one token) -------------------------------------------------------------------------

// h[d] = dequantized row `token` of the raw (not repacked) embedding payload.  First kernel of a prompt and of a batched step:
// like embed_pack_kernel it waits before it lets its dependents launch.
__global__ void embed_row_kernel(int fmt, const uint8_t* __restrict__ raw, const int* __restrict__ tokens, int n_rows,
                                 int d, float* __restrict__ h)
{
    pdl_sync();
    pdl_trigger();
    const int elems = block_elems(fmt), bytes = block_bytes(fmt);
    const int64_t row_bytes = (int64_t)(d / elems) * bytes;
    for (int r = blockIdx.y; r < n_rows; r += gridDim.y) {
        const uint8_t* row = raw + (int64_t)__ldcg(tokens + r) * row_bytes;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d; i += gridDim.x * blockDim.x) {
            h[(int64_t)r * d + i] = dequant_raw_element(fmt, row + (i / elems) * bytes, i % elems);
        }
    }
}

__device__ __forceinline__ double warp_sum_double(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    }
    return v;
}

// What every producer of a matvec input leaves behind for element e of the residual stream `hv`:
// the stream itself, hv * w as the packed activations of the matvec that follows the RMSNorm,
// and the 32-block's sum of squares (the consumer applies 1/rms to its row sums).  One warp per
// 32-block, one element per lane.
__device__ __forceinline__ void emit_block32(float hv, int group, int e, const float* __restrict__ w,
                                             float* __restrict__ h_out, uint8_t* __restrict__ packed,
                                             double* __restrict__ ss_out)
{
    if (h_out) {
        h_out[e] = hv;
    }
    const double sq = warp_sum_double((double)hv * (double)hv);
    if ((threadIdx.x & 31) == 0) {
        ss_out[group] = sq;
    }
    warp_pack_block32(hv * w[e], packed + (size_t)(group >> 3) * XPK1_REC, group & 7);
}

// First kernel of a decoded token: the embedding row of *token becomes the residual stream, and
// the first block's attention-norm input is packed.  It waits for the previous token's last
// kernel BEFORE it lets its own dependents launch: that kernel sets the token and advances the
// position, which every later kernel of this token may read as soon as it starts.
__global__ void __launch_bounds__(128) embed_pack_kernel(int fmt, const uint8_t* __restrict__ raw,
                                                         const int* __restrict__ token, int d,
                                                         const float* __restrict__ w, float* __restrict__ h,
                                                         uint8_t* __restrict__ packed, double* __restrict__ ss_out)
{
    pdl_sync();
    pdl_trigger();
    const int group = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int e = group * 32 + (threadIdx.x & 31);
    if (group * 32 >= d) {
        return;
    }
    const int elems = block_elems(fmt), bytes = block_bytes(fmt);
    const uint8_t* row = raw + (int64_t)(*token) * (int64_t)(d / elems) * bytes;
    const float hv = dequant_raw_element(fmt, row + (e / elems) * bytes, e % elems);
    emit_block32(hv, group, e, w, h, packed, ss_out);
}

__device__ __forceinline__ uint2 ld_sys_v2(const uint2* p)
{
    uint2 q;
    asm volatile("ld.relaxed.sys.global.v2.u32 {%0, %1}, [%2];" : "=r"(q.x), "=r"(q.y) : "l"(p) : "memory");
    return q;
}

__device__ __forceinline__ void st_sys_v2(uint2* p, uint32_t a, uint32_t b)
{
    asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// hv = h_in + add (add optional), then emit_block32.  The stand-alone form of the matvec's
// EPI_RESID_PACK epilogue, for the places where the addend is not one matvec's row sums:
//   - tensor parallelism (TP): `add` is only this rank's addend; the other ranks' addends arrive
//     in pg.recv as {value, exchange number} packets stored by their matvec kernels (PeerScatter,
//     qmm_common.cuh).  A lane requests the packets of all peers at once, polls the ones that
//     have not arrived (bounded), and adds the addends in rank order, so every rank computes
//     bit-identical sums without a collective launch;
//   - the last row of a prefill, whose addend comes from the GEMM path.
// h_out may equal h_in (each element is touched by one lane only).
template <bool TP>
__global__ void __launch_bounds__(128) resid_pack_kernel(const float* __restrict__ h_in, const float* __restrict__ add,
                                                         const float* __restrict__ w, int d, float* __restrict__ h_out,
                                                         uint8_t* __restrict__ packed, double* __restrict__ ss_out,
                                                         PeerGather pg)
{
    pdl_trigger();
    // the position was advanced by the previous token's last kernel, which completed before this
    // token's first kernel let anything else launch (embed_pack_kernel)
    unsigned int epoch = 0;
    if (TP) {
        epoch = (unsigned int)(*pg.pos * pg.sites + pg.site + 1);
    }
    pdl_sync();
    const int group = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int e = group * 32 + (threadIdx.x & 31);
    if (group * 32 >= d) {
        return;
    }
    float a = 0.0f;
    if (TP) {
        constexpr int MAXR = 8;
        bool ok = *reinterpret_cast<volatile int*>(pg.status) == 0;  // after one timeout nothing waits again
        uint2 pk[MAXR];
#pragma unroll
        for (int r = 0; r < MAXR; ++r) {
            if (r < pg.tp_size && r != pg.tp_rank) {
                pk[r] = ld_sys_v2(pg.recv + (size_t)r * d + e);
            }
        }
        const float own = __ldcg(add + e);
#pragma unroll
        for (int r = 0; r < MAXR; ++r) {
            if (r < pg.tp_size) {
                if (r == pg.tp_rank) {
                    a += own;
                } else {
                    unsigned int spin = 0;
                    while (ok && pk[r].y != epoch) {
                        if (++spin > pg.spin_limit) {
                            ok = false;
                            atomicExch(pg.status, 5);  // a peer's addend never came; the sum is incomplete
                            break;
                        }
                        pk[r] = ld_sys_v2(pg.recv + (size_t)r * d + e);
                    }
                    a += __uint_as_float(pk[r].x);
                }
            }
        }
    } else if (add) {
        a = __ldcg(add + e);
    }
    emit_block32(__ldcg(h_in + e) + a, group, e, w, h_out, packed, ss_out);
}

// cos/sin tables [max_seq][rope_dim/2], computed in double and cast (Layer/RoPE.h:22-39).
__global__ void rope_table_kernel(int max_seq, int rope_dim, double theta, float* __restrict__ rope_cos,
                                  float* __restrict__ rope_sin)
{
    const int half = rope_dim / 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)max_seq * half;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int pos = (int)(i / half), dim = (int)(i % half);
        const double inv_freq = pow(theta, -2.0 * (double)dim / (double)rope_dim);
        const double ang = (double)pos * inv_freq;
        rope_cos[i] = (float)cos(ang);
        rope_sin[i] = (float)sin(ang);
    }
}

// RoPE on q and k of one token at position *pos, K/V appended to the fp16 cache.
//   qkv: [n_heads*hd | n_kv*hd | n_kv*hd] fp32 (q rotated in place)
//   cache_k / cache_v: [n_kv][max_seq][hd] fp16
__global__ void rope_kv_kernel(float* __restrict__ qkv, const int* __restrict__ pos_ptr, int pos_add, int n_heads,
                               int n_kv, int hd, int rope_dim, const float* __restrict__ rope_cos,
                               const float* __restrict__ rope_sin, int max_seq, __half* __restrict__ cache_k,
                               __half* __restrict__ cache_v, int row_stride)
{
    pdl_trigger();
    pdl_sync();
    const int row = blockIdx.y;  // token within the batch (prefill) or 0
    const int pos = *pos_ptr + pos_add + row;
    float* base = qkv + (int64_t)row * row_stride;
    const int pairs_q = n_heads * hd / 2, pairs_k = n_kv * hd / 2;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < pairs_q + pairs_k + n_kv * hd; p += gridDim.x * blockDim.x) {
        if (p < pairs_q + pairs_k) {
            const bool is_k = p >= pairs_q;
            const int pp = is_k ? p - pairs_q : p;
            const int head = pp / (hd / 2), i = pp % (hd / 2);
            float* x = base + (is_k ? n_heads * hd : 0) + head * hd + 2 * i;
            float a = x[0], b = x[1];
            if (2 * i < rope_dim) {
                const float c = rope_cos[(int64_t)pos * (rope_dim / 2) + i];
                const float s = rope_sin[(int64_t)pos * (rope_dim / 2) + i];
                const float ra = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s));
                const float rb = __fadd_rn(__fmul_rn(a, s), __fmul_rn(b, c));
                a = ra;
                b = rb;
            }
            if (is_k) {
                __half* dst = cache_k + ((int64_t)head * max_seq + pos) * hd + 2 * i;
                dst[0] = __float2half_rn(a);
                dst[1] = __float2half_rn(b);
            } else {
                x[0] = a;
                x[1] = b;
            }
        } else {
            const int e = p - pairs_q - pairs_k;
            const int head = e / hd, i = e % hd;
            cache_v[((int64_t)head * max_seq + pos) * hd + i] = __float2half_rn(base[(n_heads + n_kv) * hd + e]);
        }
    }
}

// CTAs per 256-wide context chunk = key splits / 4.  One sequence wants the most splits a portable cluster
// allows (cluster sizes 4 and 16 measured slower than 8: 39.2 / 38.1 / 36.6 us per block of the 7B shape); a
// batch of sequences already fills the SMs with (sequence, chunk) pairs, and fewer, longer splits keep its
// CTAs in one wave.
constexpr int attn_cluster_for(int batch)
{
    return batch >= 8 ? 2 : batch >= 3 ? 4 : 8;
}

// Decode attention of one token in one launch: RoPE of q and of the new key, K/V append to
// the fp16 cache, attention over the cache, merge and activation packing.
// A cluster of CTAs owns one 256-wide chunk of the context vector (256/hd heads).  Inside a
// CTA warp w serves head (w % HH) of the chunk and key split (rank * NSUB + w / HH); every warp
// rotates its own copy of q, takes batches of 8 cached keys (all loads of a batch are issued
// before any use) and keeps an online softmax.  The last split also takes the new position,
// whose key and value come straight from the qkv vector (rounded to fp16 as the cache holds
// them) and are stored to the cache by the first head of each kv group.  Partials are merged
// per CTA in shared memory and stored into rank 0's shared memory (distributed shared memory);
// rank 0 merges the CTAs' partials and writes the packed chunk.
template <int DPL, int ATTN_CLUSTER>  // head dims per lane = hd / 32 (2 or 4); CTAs per 256-wide context chunk
__global__ void __launch_bounds__(256) attn_fused_kernel(const float* __restrict__ qkv, const int* __restrict__ pos_ptr,
                                                         int n_heads, int n_kv, int rope_dim,
                                                         const float* __restrict__ rope_cos,
                                                         const float* __restrict__ rope_sin, int max_seq,
                                                         __half* __restrict__ cache_k, __half* __restrict__ cache_v,
                                                         uint8_t* __restrict__ packed, AttnBatch ab)
{
    constexpr int hd = 32 * DPL;
    // batched decode: blockIdx.y is the sequence; each has its own qkv row, position and cache
    qkv += (int64_t)blockIdx.y * ab.qkv_stride;
    pos_ptr += blockIdx.y;
    cache_k += (int64_t)blockIdx.y * ab.cache_stride;
    cache_v += (int64_t)blockIdx.y * ab.cache_stride;
    constexpr int HH = 256 / hd;  // heads per chunk
    constexpr int NSUB = 8 / HH;  // key splits per CTA
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // Shared memory is kept small (13 KB) on purpose: this kernel is launched while the qkv matvec
    // still fills the SMs, and it can only start its preloads early if a CTA fits beside them.
    __shared__ float sm[8][hd + 2];                      // per-warp partials of this CTA
    __shared__ float parts[ATTN_CLUSTER][HH][hd + 2];    // rank 0's copy collects every CTA's merged partials
    __shared__ float vals[256];
    pdl_trigger();
    // Everything up to pdl_sync() reads only what earlier tokens left behind (the position, the
    // rotation tables, the cached keys and values), so it runs while the qkv GEMV is finishing.  All of that is in place
    // because the first kernel of a step waits for the step before and only then releases what follows it.
    const int rank = (int)cluster.block_rank();
    const int chunk = blockIdx.x / ATTN_CLUSTER;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hl = warp % HH, sub = warp / HH;
    const int head = chunk * HH + hl;
    const int nsplit = ATTN_CLUSTER * NSUB, split = rank * NSUB + sub;
    const int pos = *pos_ptr;
    const int per = (pos + nsplit - 1) / nsplit;
    const int k0 = split * per, k1 = min(pos, k0 + per);
    const int group = n_heads / n_kv, kvh = head < n_heads ? head / group : 0;
    const __half* kb = cache_k + (int64_t)kvh * max_seq * hd + lane * DPL;
    const __half* vb = cache_v + (int64_t)kvh * max_seq * hd + lane * DPL;
    float cs_[DPL / 2], sn_[DPL / 2];
#pragma unroll
    for (int j = 0; j < DPL / 2; ++j) {
        const int i = lane * (DPL / 2) + j;
        const bool rot = 2 * i < rope_dim;
        cs_[j] = rot ? rope_cos[(int64_t)pos * (rope_dim / 2) + i] : 1.0f;
        sn_[j] = rot ? rope_sin[(int64_t)pos * (rope_dim / 2) + i] : 0.0f;
    }
    // The first 16 keys of this warp's split go to registers now; longer splits are prefetched
    // to L2 and loaded in the loop below.
    KvBatch<DPL> pre0, pre1;
    if (head < n_heads) {
        kv_batch_load<DPL>(pre0, kb, vb, k0, k1);
        kv_batch_load<DPL>(pre1, kb, vb, k0 + 8, k1);
        // one 128-byte line per lane and step: this warp's rows of K and of V are contiguous
        const char* kl = reinterpret_cast<const char*>(cache_k + ((int64_t)kvh * max_seq + k0 + 16) * hd);
        const char* vl = reinterpret_cast<const char*>(cache_v + ((int64_t)kvh * max_seq + k0 + 16) * hd);
        const int bytes = (k1 - k0 - 16) * hd * (int)sizeof(__half);
        for (int o = lane * 128; o < bytes; o += 32 * 128) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(kl + o));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(vl + o));
        }
    }
    pdl_sync();
    float acc[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        acc[i] = 0.0f;
    }
    float m = -INFINITY, l = 0.0f;
    if (head < n_heads) {
        const float scale = rsqrtf((float)hd);
        const bool takes_new = split == nsplit - 1;
        float2 qx[DPL / 2], kx[DPL / 2], vx[DPL / 2];
#pragma unroll
        for (int j = 0; j < DPL / 2; ++j) {
            qx[j] = *reinterpret_cast<const float2*>(qkv + head * hd + lane * DPL + 2 * j);
            if (takes_new) {
                kx[j] = *reinterpret_cast<const float2*>(qkv + (n_heads + kvh) * hd + lane * DPL + 2 * j);
                vx[j] = *reinterpret_cast<const float2*>(qkv + (n_heads + n_kv + kvh) * hd + lane * DPL + 2 * j);
            }
        }
        float qv[DPL];
#pragma unroll
        for (int j = 0; j < DPL / 2; ++j) {
            const float2 x = qx[j];
            const bool rot = 2 * (lane * (DPL / 2) + j) < rope_dim;
            const float ra = rot ? __fsub_rn(__fmul_rn(x.x, cs_[j]), __fmul_rn(x.y, sn_[j])) : x.x;
            const float rb = rot ? __fadd_rn(__fmul_rn(x.x, sn_[j]), __fmul_rn(x.y, cs_[j])) : x.y;
            qv[2 * j] = ra * scale;
            qv[2 * j + 1] = rb * scale;
        }
        kv_batch_apply<DPL>(pre0, qv, k0, k1, m, l, acc);
        kv_batch_apply<DPL>(pre1, qv, k0 + 8, k1, m, l, acc);
        for (int kbase = k0 + 16; kbase < k1; kbase += 8) {
            KvBatch<DPL> cur;
            kv_batch_load<DPL>(cur, kb, vb, kbase, k1);
            kv_batch_apply<DPL>(cur, qv, kbase, k1, m, l, acc);
        }
        if (takes_new) {  // the new position
            __half kn[DPL], vn[DPL];
#pragma unroll
            for (int j = 0; j < DPL / 2; ++j) {
                const float2 x = kx[j];
                const float2 v = vx[j];
                const bool rot = 2 * (lane * (DPL / 2) + j) < rope_dim;
                const float ra = rot ? __fsub_rn(__fmul_rn(x.x, cs_[j]), __fmul_rn(x.y, sn_[j])) : x.x;
                const float rb = rot ? __fadd_rn(__fmul_rn(x.x, sn_[j]), __fmul_rn(x.y, cs_[j])) : x.y;
                kn[2 * j] = __float2half_rn(ra);
                kn[2 * j + 1] = __float2half_rn(rb);
                vn[2 * j] = __float2half_rn(v.x);
                vn[2 * j + 1] = __float2half_rn(v.y);
            }
            if (head % group == 0) {
                __half* kd = cache_k + ((int64_t)kvh * max_seq + pos) * hd + lane * DPL;
                __half* vd = cache_v + ((int64_t)kvh * max_seq + pos) * hd + lane * DPL;
#pragma unroll
                for (int i = 0; i < DPL; i += 2) {
                    *reinterpret_cast<__half2*>(kd + i) = *reinterpret_cast<const __half2*>(&kn[i]);
                    *reinterpret_cast<__half2*>(vd + i) = *reinterpret_cast<const __half2*>(&vn[i]);
                }
            }
            float dot = 0.0f;
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                dot += qv[i] * __half2float(kn[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                dot += __shfl_xor_sync(0xFFFFFFFFu, dot, o);
            }
            const float mb = fmaxf(m, dot);
            const float corr = __expf(m - mb), p = __expf(dot - mb);
            l = l * corr + p;
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                acc[i] = acc[i] * corr + p * __half2float(vn[i]);
            }
            m = mb;
        }
    }
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        sm[warp][lane * DPL + i] = acc[i];
    }
    if (lane == 0) {
        sm[warp][hd] = m;
        sm[warp][hd + 1] = l;
    }
    __syncthreads();
    {   // merge this CTA's key splits per head and hand the result to rank 0 of the cluster
        const int h2 = threadIdx.x / hd, e = threadIdx.x % hd;
        float M = -INFINITY;
#pragma unroll
        for (int s2 = 0; s2 < NSUB; ++s2) {
            M = fmaxf(M, sm[h2 + HH * s2][hd]);
        }
        float a = 0.0f, L = 0.0f;
#pragma unroll
        for (int s2 = 0; s2 < NSUB; ++s2) {
            const float mw = sm[h2 + HH * s2][hd];
            const float f = mw == -INFINITY ? 0.0f : __expf(mw - M);
            a += sm[h2 + HH * s2][e] * f;
            L += sm[h2 + HH * s2][hd + 1] * f;
        }
        float* dst = cluster.map_shared_rank(&parts[0][0][0], 0) + (rank * HH + h2) * (hd + 2);
        dst[e] = a;
        if (e == 0) {
            dst[hd] = M;
            dst[hd + 1] = L;
        }
    }
    cluster.sync();  // remote stores above are visible to rank 0 after this
    if (rank != 0) {
        return;
    }
    {
        const int h2 = threadIdx.x / hd, e = threadIdx.x % hd;
        float M = -INFINITY;
#pragma unroll
        for (int r = 0; r < ATTN_CLUSTER; ++r) {
            M = fmaxf(M, parts[r][h2][hd]);
        }
        float a = 0.0f, L = 0.0f;
#pragma unroll
        for (int r = 0; r < ATTN_CLUSTER; ++r) {
            const float mp = parts[r][h2][hd];
            const float f = mp == -INFINITY ? 0.0f : __expf(mp - M);
            a += parts[r][h2][e] * f;
            L += parts[r][h2][hd + 1] * f;
        }
        vals[threadIdx.x] = L > 0.0f ? a / L : 0.0f;
    }
    __syncthreads();
    if (ab.packed) {  // batched decode: this sequence's row of the chunk's record
        if (threadIdx.x < 64) {
            const int e = 4 * threadIdx.x;  // two warps, 128 activations each
            const float4 v = make_float4(vals[e], vals[e + 1], vals[e + 2], vals[e + 3]);
            pack_row_block4(v, ab.packed + (size_t)chunk * xpack_row_rec_bytes(ab.ncp), ab.ncp, blockIdx.y, e >> 5, true);
        }
        return;
    }
    if (threadIdx.x < 32) {
        float r8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            r8[i] = vals[8 * threadIdx.x + i];
        }
        warp_pack_chunk(r8, packed + (size_t)chunk * XPK1_REC);
    }
}

// Greedy argmax, first stage (lowest index wins ties): CTA b writes its (value bits, index)
// candidate to best_pair[2b..2b+1].
__global__ void __launch_bounds__(1024) argmax_kernel(const float* __restrict__ logits, int n, int index_offset,
                                                      int* __restrict__ best_pair, int64_t row_stride)
{
    __shared__ float sv[32];
    __shared__ int si[32];
    pdl_trigger();
    pdl_sync();
    logits += (int64_t)blockIdx.y * row_stride;  // batched decode: one row of logits per sequence
    best_pair += (int64_t)blockIdx.y * 2 * gridDim.x;
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = logits[i];
        if (v > bv || (v == bv && i < bi)) {
            bv = v;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
        const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    if ((threadIdx.x & 31) == 0) {
        sv[threadIdx.x >> 5] = bv;
        si[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            if (sv[w] > bv || (sv[w] == bv && si[w] < bi)) {
                bv = sv[w];
                bi = si[w];
            }
        }
        best_pair[2 * blockIdx.x] = __float_as_int(bv);
        best_pair[2 * blockIdx.x + 1] = bi == 0x7FFFFFFF ? bi : bi + index_offset;
    }
}

// Picks the winner among this rank's `n_local` (value, index) candidates, and with tensor
// parallelism among the ranks' winners: every rank stores its winner as two packets
// {value bits, number} {index, number} into each peer's buffer (number = position + 1) and polls
// the peers' packets (bounded).  Ties go to the lowest index, so all ranks agree.  Then stores
// the token and advances the position.  One warp.
__global__ void __launch_bounds__(32) commit_token_kernel(const int* __restrict__ pairs, int n_local, ArgmaxExchange ax,
                                                          int* __restrict__ token, int* __restrict__ pos,
                                                          int* __restrict__ out_tokens, int* __restrict__ out_count,
                                                          TokenReport report)
{
    pdl_trigger();
    pdl_sync();
    const int lane = threadIdx.x;
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    for (int i = lane; i < n_local; i += 32) {
        const float v = __int_as_float(pairs[2 * i]);
        const int ix = pairs[2 * i + 1];
        if (v > bv || (v == bv && ix < bi)) {
            bv = v;
            bi = ix;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
        const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    if (ax.tp_size > 1) {
        const unsigned int number = (unsigned int)(*pos + 1);
        if (lane < ax.tp_size && lane != ax.tp_rank) {
            uint2* dst = ax.peer[lane] + 2 * ax.tp_rank;
            st_sys_v2(dst, __float_as_uint(bv), number);
            st_sys_v2(dst + 1, (uint32_t)bi, number);
        }
        float cv = -INFINITY;
        int ci = 0x7FFFFFFF;
        if (lane == ax.tp_rank) {
            cv = bv;
            ci = bi;
        } else if (lane < ax.tp_size) {
            bool ok = *reinterpret_cast<volatile int*>(ax.status) == 0;
            const uint2* src = ax.recv + 2 * lane;
            uint2 a = ld_sys_v2(src), b = ld_sys_v2(src + 1);
            unsigned int spin = 0;
            while (ok && (a.y != number || b.y != number)) {
                if (++spin > ax.spin_limit) {
                    ok = false;
                    atomicExch(ax.status, 6);  // a peer's arg-max candidate never came
                    break;
                }
                a = ld_sys_v2(src);
                b = ld_sys_v2(src + 1);
            }
            if (ok) {
                cv = __uint_as_float(a.x);
                ci = (int)b.x;
            }
        }
        bv = cv;
        bi = ci;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
            const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) {
                bv = ov;
                bi = oi;
            }
        }
    }
    if (lane == 0) {
        *token = bi;
        out_tokens[*out_count] = bi;
        *out_count += 1;
        *pos += 1;
        if (report.host) {
            // the token and the two status words in host-visible memory: a caller that takes one token at a
            // time reads them after the stream has drained, without a copy of its own
            report.host[0] = bi;
            report.host[1] = *reinterpret_cast<const volatile int*>(report.model_status);
            report.host[2] = *reinterpret_cast<const volatile int*>(report.library_status);
        }
    }
}

// Batched decode: one warp per sequence picks the winner among the ranks' candidates of its row
// (pairs[rank][row][2 * per_rank]; lowest index wins ties), stores the row's next token, appends it to
// the step-major output list and advances the row's position.
__global__ void __launch_bounds__(512) commit_batch_kernel(const int* __restrict__ pairs, int per_rank, int ranks,
                                                           int batch, int* __restrict__ tokens, int* __restrict__ pos,
                                                           int* __restrict__ out_tokens, int* __restrict__ out_steps)
{
    pdl_trigger();
    pdl_sync();
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    if (row < batch) {
        for (int i = lane; i < per_rank * ranks; i += 32) {
            const int r = i / per_rank, c = i % per_rank;
            const int* p = pairs + ((int64_t)r * batch + row) * 2 * per_rank + 2 * c;
            const float v = __int_as_float(p[0]);
            const int ix = p[1];
            if (v > bv || (v == bv && ix < bi)) {
                bv = v;
                bi = ix;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
        const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) {
            bv = ov;
            bi = oi;
        }
    }
    const int step = *out_steps;
    __syncthreads();  // every warp has read the step count before it moves
    if (row < batch && lane == 0) {
        tokens[row] = bi;
        out_tokens[(int64_t)step * batch + row] = bi;
        pos[row] += 1;
    }
    if (threadIdx.x == 0) {
        *out_steps = step + 1;
    }
}

// ---- prefill (many tokens) ------------------------------------------------------------------------

// Where a row kernel puts four neighbouring values of its row.  All threads of a warp call it; `ok` marks the ones that
// hold values.
struct RowOutBf16 {  // bf16 rows for the GEMM
    __nv_bfloat16* p;
    int64_t width;
    __device__ __forceinline__ void put(int64_t row, int i4, const float4& v, bool ok) const
    {
        if (ok) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
            *reinterpret_cast<uint2*>(p + row * width + 4 * (int64_t)i4) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
    }
};
struct RowOutPacked {  // the row's part of the matvec's packed activations; rows are a multiple of 32 wide
    uint8_t* p;
    int ncp;
    __device__ __forceinline__ void put(int64_t row, int i4, const float4& v, bool ok) const
    {
        pack_row_block4(v, p + (size_t)(i4 >> 6) * xpack_row_rec_bytes(ncp), ncp, (int)row, (i4 >> 3) & 7, ok);
    }
};

// Per row: h += add (optional); rmsnorm(h) * w, as bf16 for the GEMM or packed for the matvec of a batch.
// One CTA per row (d a multiple of 4); a thread keeps its float4 pieces of the row in registers between the
// two passes (up to 8 pieces = d <= 8192 with 256 threads; longer rows re-read h), and all of a pass's loads
// are issued before the first is used: with scalar loads in a 16-trip loop the kernel took 18 us for 16 rows.
// Statistics and the scale by the weight in double, one cast (ComputePrimitives.h:755-816); one double
// reciprocal per row instead of a division per element (within one unit in the last place of the double
// quotient, so the fp32 result is the reference's).
template <typename Out>
__global__ void __launch_bounds__(256) resid_rmsnorm_rows_kernel(float* __restrict__ h, const float* __restrict__ add,
                                                                 const float* __restrict__ w, float eps, int d,
                                                                 Out out)
{
    pdl_trigger();
    pdl_sync();
    constexpr int KEEP = 8;
    __shared__ double red[32];
    const int64_t row = blockIdx.x;
    float4* hr = reinterpret_cast<float4*>(h + row * d);
    const float4* ar = add ? reinterpret_cast<const float4*>(add + row * d) : nullptr;
    const int n4 = d >> 2;
    float4 keep[KEEP];
    double ss = 0.0;
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        const int i = threadIdx.x + j * 256;
        keep[j] = i < n4 ? hr[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (ar) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = threadIdx.x + j * 256;
            if (i < n4) {
                const float4 a = __ldcg(ar + i);
                keep[j].x += a.x;
                keep[j].y += a.y;
                keep[j].z += a.z;
                keep[j].w += a.w;
                hr[i] = keep[j];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        ss += (double)keep[j].x * (double)keep[j].x + (double)keep[j].y * (double)keep[j].y +
              (double)keep[j].z * (double)keep[j].z + (double)keep[j].w * (double)keep[j].w;
    }
    for (int i = threadIdx.x + KEEP * 256; i < n4; i += 256) {  // rows longer than 8192
        float4 v = hr[i];
        if (ar) {
            const float4 a = __ldcg(ar + i);
            v = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
            hr[i] = v;
        }
        ss += (double)v.x * (double)v.x + (double)v.y * (double)v.y + (double)v.z * (double)v.z + (double)v.w * (double)v.w;
    }
    ss = block_sum_double(ss, red);
    const double inv = 1.0 / sqrt(ss / (double)d + (double)eps);
    const float4* wr = reinterpret_cast<const float4*>(w);
    auto emit = [&](int i, const float4& v) {
        const bool ok = i < n4;
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (ok) {
            const float4 ww = wr[i];
            o = make_float4((float)(((double)v.x * inv) * (double)ww.x), (float)(((double)v.y * inv) * (double)ww.y),
                            (float)(((double)v.z * inv) * (double)ww.z), (float)(((double)v.w * inv) * (double)ww.w));
        }
        out.put(row, i, o, ok);
    };
#pragma unroll
    for (int j = 0; j < KEEP; ++j) {
        if (j * 256 < n4) {
            emit(threadIdx.x + j * 256, keep[j]);
        }
    }
    for (int i0 = KEEP * 256; i0 < n4; i0 += 256) {
        const int i = i0 + threadIdx.x;
        emit(i, i < n4 ? hr[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    }
}

// ---- prefill attention -------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

// D += A(16x16, fp16) * B(16x8, fp16), fp32 accumulate
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Two fp32 values as sums of N fp16 parts, the largest first.  fp16 ends at 2^-24: three parts hold every bit of a value
// of at least 1/2, of smaller ones what lies above that.
template <int N>
__device__ __forceinline__ void split_f16x2(float a, float b, uint32_t (&o)[N])
{
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        a -= f.x;
        b -= f.y;
        o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

__device__ __forceinline__ void store_ctx(__nv_bfloat16* p, float a, float b)
{
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}
__device__ __forceinline__ void store_ctx(float* p, float a, float b)  // tests look at the sums before they are rounded
{
    *reinterpret_cast<float2*>(p) = make_float2(a, b);
}

// (The prefill attention kernels take plain pointers: what they read is written by kernels that may still run when they start,
// and loads of read-only data need not stay behind the dependency wait.)
// Causal attention for rows row0..row0+ROWS-1 of one head (those below m) by one warp, fp32 arithmetic throughout: it
// reuses each loaded batch of eight keys for all of its rows; a row simply ignores the keys beyond its own position.
// Online softmax per row, one rescale per batch.
template <int DPL, int ROWS, typename OutT>
__device__ __forceinline__ void attn_rows(const float* qkv, int row_stride, int m, int pos0, int n_heads,
                                          int n_kv, int max_seq, const __half* cache_k,
                                          const __half* cache_v, OutT* ctx, int row0, int head)
{
    constexpr int hd = 32 * DPL;
    const int lane = threadIdx.x & 31;
    const int kvh = head / (n_heads / n_kv);
    const float scale = rsqrtf((float)hd);
    float qv[ROWS][DPL], acc[ROWS][DPL], mx[ROWS], l[ROWS];
    int keys[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int row = min(row0 + r, m - 1);  // a ragged last group repeats the last row (stored once)
        keys[r] = pos0 + row + 1;
        mx[r] = -INFINITY;
        l[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            qv[r][i] = qkv[(int64_t)row * row_stride + head * hd + lane * DPL + i] * scale;
            acc[r][i] = 0.0f;
        }
    }
    const __half* kb = cache_k + (int64_t)kvh * max_seq * hd + lane * DPL;
    const __half* vb = cache_v + (int64_t)kvh * max_seq * hd + lane * DPL;
    const int n_keys = keys[ROWS - 1];
    KvBatch<DPL> a, b;
    kv_batch_load<DPL>(a, kb, vb, 0, n_keys);
    for (int kbase = 0; kbase < n_keys; kbase += 16) {
        if (kbase + 8 < n_keys) {
            kv_batch_load<DPL>(b, kb, vb, kbase + 8, n_keys);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            kv_batch_apply<DPL>(a, qv[r], kbase, keys[r], mx[r], l[r], acc[r]);
        }
        if (kbase + 16 < n_keys) {
            kv_batch_load<DPL>(a, kb, vb, kbase + 16, n_keys);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            kv_batch_apply<DPL>(b, qv[r], kbase + 8, keys[r], mx[r], l[r], acc[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (row0 + r < m) {
#pragma unroll
            for (int i = 0; i < DPL; i += 2) {
                store_ctx(ctx + (int64_t)(row0 + r) * n_heads * hd + head * hd + lane * DPL + i, acc[r][i] / l[r],
                          acc[r][i + 1] / l[r]);
            }
        }
    }
}

// Sixteen rows again, for attn_prefill_kernel; kept out of line, so that its registers are not that kernel's.
template <int HD, typename OutT>
__device__ __noinline__ void attn_rows_again(const float* qkv, int row_stride, int m, int pos0, int n_heads, int n_kv,
                                             int max_seq, const __half* cache_k, const __half* cache_v, OutT* ctx, int row0,
                                             int head)
{
    for (int r = row0; r < min(row0 + 16, m); r += 4) {
        attn_rows<HD / 32, 4>(qkv, row_stride, m, pos0, n_heads, n_kv, max_seq, cache_k, cache_v, ctx, r, head);
    }
}

// Causal attention over the fp16 cache for rows 0..m-1 at positions pos0+row, on the tensor cores.  A CTA owns 64
// query rows of one head (16 per warp) and walks the keys in tiles of 64, which cp.async brings into shared memory one
// tile ahead; online softmax per row, output bf16 ctx[m][n_heads*hd].
// Queries and probabilities are fp32 and go through the fp16 MMA in parts (K and V are fp16, so those are exact): a query
// as three parts, which hold all of its bits, a probability as two, which hold 23.  A power of two per row keeps the
// split away from fp16's range limits: the row's largest query value is brought to 2^14..2^15, probabilities are taken
// times 2^14.  The MMA truncates what it adds, so its chains are kept short and start with the smallest parts: 32
// dimensions of a score, one tile of keys of a context value; fp32 additions, which round, put these together.
// Error against 64 bits before the rounding to bf16 (2-norm, 300 / 1999 tokens, HD 128, scores of about 1): 1.6e-7 /
// 1.4e-7 here, 2.1e-7 / 6.2e-7 in the fp32 row kernel below; two parts and one chain for everything had 5.5e-7 / 2.9e-6.
// Scores of about 16: 4.1e-7 / 5.3e-7, 4.2e-7 / 5.4e-7 and 1.3e-6 / 1.6e-6.
// Bound: the MMA pipe (65 % of all cycles at 1999 rows), about 16 cycles per m16n8k16 and scheduler, five MMAs where plain
// fp16 takes two.  1999 rows, 32 heads, HD 128: 309 us, 272 with two parts of a query, 247 with two parts and long chains.
// Four rows per warp with fp32 arithmetic and shuffles are issue-bound: 512 rows 250 us against 40.
// A masked key's V row takes part in the product with probability 0, and a query or a key that overflowed fp16 meets the
// parts one by one, so infinities and NaN spread further here than they should.  They always leave a mark on the row's own
// sums, and a warp that finds one does its rows again in fp32, key by key.
template <int HD, typename OutT>
__global__ void __launch_bounds__(128, HD == 128 ? 2 : 3)  // what its shared memory lets an SM hold at HD = 128
    attn_prefill_kernel(const float* qkv, int row_stride, int m,
                                                           int pos0, int n_heads, int n_kv, int max_seq,
                                                           const __half* cache_k,
                                                           const __half* cache_v, OutT* ctx)
{
    constexpr int KT = 64;                 // keys per tile
    constexpr int ROW = HD * 2;            // bytes of a key row
    constexpr int CH = ROW / 16;           // 16-byte pieces of it; piece c of row r sits at c ^ (r & 7)
    constexpr int TILE = KT * ROW;
    constexpr int KS = HD / 16;            // k steps of a score
    constexpr int QP = 3, PP = 2;          // parts of a query and of a probability
    constexpr int KG = 2, JG = 2;          // k steps of one MMA chain, 16-wide column groups of V at a time
    constexpr float P_SCALE = 16384.0f;
    extern __shared__ __align__(128) uint8_t att_smem[];  // [2 buffers][K tile | V tile], query fragments
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int head = blockIdx.y, kvh = head / (n_heads / n_kv);
    const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 64;  // the longest rows first
    const int n_keys = pos0 + min(row0 + 64, m);                   // keys the last row of this CTA sees
    const int tiles = (n_keys + KT - 1) / KT;
    const __half* kb = cache_k + (int64_t)kvh * max_seq * HD;
    const __half* vb = cache_v + (int64_t)kvh * max_seq * HD;

    auto fetch = [&](int tile) {
        const uint32_t dst = smem_addr(att_smem) + (tile & 1) * 2 * TILE;
#pragma unroll
        for (int i = 0; i < KT * CH / 128; ++i) {
            const int idx = threadIdx.x + i * 128;
            const int r = idx / CH, c = idx % CH;
            const int key = min(tile * KT + r, n_keys - 1);  // beyond the last key: any row that exists
            const uint32_t o = dst + r * ROW + ((c ^ (r & 7)) * 16);
            cp_async16(o, kb + (int64_t)key * HD + c * 8);
            cp_async16(o + TILE, vb + (int64_t)key * HD + c * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);

    // this thread's rows of the warp's 16: g and g + 8; their A fragments wait in shared memory, where only this thread
    // reads them: [part][k step][lane]
    int rows[2];
    uint4* qfrag = reinterpret_cast<uint4*>(att_smem + 4 * TILE) + warp * (QP * KS * 32) + lane;
    float unscale[2];
    {
        const float scale = rsqrtf((float)HD);
        float2 x[2][HD / 8];
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            rows[rs] = row0 + warp * 16 + g + 8 * rs;
            const float* q = qkv + (int64_t)min(rows[rs], m - 1) * row_stride + head * HD + 2 * t;
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                x[rs][i] = *reinterpret_cast<const float2*>(q + 8 * i);
                x[rs][i].x *= scale;
                x[rs][i].y *= scale;
                amax = fmaxf(amax, fmaxf(fabsf(x[rs][i].x), fabsf(x[rs][i].y)));
            }
            amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
            const int e = max((int)((__float_as_uint(amax) >> 23) & 255u) - 127, -100);
            const float up = __uint_as_float((uint32_t)(127 + 14 - e) << 23);
            unscale[rs] = __uint_as_float((uint32_t)(127 - 14 + e) << 23);
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                x[rs][i].x *= up;
                x[rs][i].y *= up;
            }
        }
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            uint32_t a[4][QP];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 v = x[i & 1][2 * k + (i >> 1)];
                split_f16x2<QP>(v.x, v.y, a[i]);
            }
#pragma unroll
            for (int p = 0; p < QP; ++p) {
                qfrag[(p * KS + k) * 32] = make_uint4(a[0][p], a[1][p], a[2][p], a[3][p]);
            }
        }
    }
    float acc[HD / 8][4], mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < HD / 8; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[j][i] = 0.0f;
        }
    }

    for (int tile = 0; tile < tiles; ++tile) {
        if (tile + 1 < tiles) {
            fetch(tile + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t ks = smem_addr(att_smem) + (tile & 1) * 2 * TILE, vs = ks + TILE;

        // scores of 16 rows x 64 keys
        float sc[KT / 8][4];
#pragma unroll
        for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sc[j][i] = 0.0f;
            }
        }
#pragma unroll
        for (int k0 = 0; k0 < KS; k0 += KG) {
            uint32_t b[KG][KT / 16][4];
#pragma unroll
            for (int kg = 0; kg < KG; ++kg) {
#pragma unroll
                for (int j2 = 0; j2 < KT / 16; ++j2) {
                    const int r = 16 * j2 + (lane >> 4) * 8 + (lane & 7);
                    ldmatrix_x4(b[kg][j2], ks + r * ROW + (((2 * (k0 + kg) + ((lane >> 3) & 1)) ^ (r & 7)) * 16));
                }
            }
            float d[KT / 8][4] = {};
#pragma unroll
            for (int p = QP - 1; p >= 0; --p) {
#pragma unroll
                for (int kg = 0; kg < KG; ++kg) {
                    const uint4 v = qfrag[(p * KS + k0 + kg) * 32];
                    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < KT / 8; ++j) {
                        mma_f16(d[j], q, b[kg][j >> 1][2 * (j & 1)], b[kg][j >> 1][2 * (j & 1) + 1]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    sc[j][i] += d[j][i];
                }
            }
        }
        const bool masked = tile * KT + KT - 1 > pos0 + row0 + warp * 16;  // some row of the warp ends inside the tile
        float corr[2], sum[2] = {0.0f, 0.0f};
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            float mb = mx[rs];
#pragma unroll
            for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float& s = sc[j][2 * rs + i];
                    s *= unscale[rs];
                    if (masked && tile * KT + 8 * j + 2 * t + i > pos0 + rows[rs]) {
                        s = -INFINITY;
                    }
                    mb = fmaxf(mb, s);
                }
            }
            mb = fmaxf(mb, __shfl_xor_sync(0xFFFFFFFFu, mb, 1));
            mb = fmaxf(mb, __shfl_xor_sync(0xFFFFFFFFu, mb, 2));
            corr[rs] = __expf(mx[rs] - mb);
            mx[rs] = mb;
#pragma unroll
            for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float p = __expf(sc[j][2 * rs + i] - mb);
                    sum[rs] += p;
                    sc[j][2 * rs + i] = p * P_SCALE;
                }
            }
            l[rs] = l[rs] * corr[rs] + sum[rs];
        }
        // probabilities times V: the score fragments are the A operand as they lie
        uint32_t pf[KT / 16][4][PP];
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                split_f16x2<PP>(sc[2 * kk + (i >> 1)][2 * (i & 1)], sc[2 * kk + (i >> 1)][2 * (i & 1) + 1], pf[kk][i]);
            }
        }
#pragma unroll
        for (int j0 = 0; j0 < HD / 16; j0 += JG) {
            uint32_t b[JG][KT / 16][4];
#pragma unroll
            for (int jg = 0; jg < JG; ++jg) {
#pragma unroll
                for (int kk = 0; kk < KT / 16; ++kk) {
                    const int r = 16 * kk + ((lane >> 3) & 1) * 8 + (lane & 7);
                    ldmatrix_x4_trans(b[jg][kk], vs + r * ROW + (((2 * (j0 + jg) + (lane >> 4)) ^ (r & 7)) * 16));
                }
            }
            float d[JG][2][4] = {};
#pragma unroll
            for (int p = PP - 1; p >= 0; --p) {
#pragma unroll
                for (int kk = 0; kk < KT / 16; ++kk) {
                    const uint32_t a[4] = {pf[kk][0][p], pf[kk][1][p], pf[kk][2][p], pf[kk][3][p]};
#pragma unroll
                    for (int jg = 0; jg < JG; ++jg) {
                        mma_f16(d[jg][0], a, b[jg][kk][0], b[jg][kk][1]);
                        mma_f16(d[jg][1], a, b[jg][kk][2], b[jg][kk][3]);
                    }
                }
            }
#pragma unroll
            for (int jg = 0; jg < JG; ++jg) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float& o = acc[2 * (j0 + jg) + h][i];
                        o = fmaf(o, corr[i >> 1], d[jg][h][i]);
                    }
                }
            }
        }
        __syncthreads();  // the buffer is refilled two tiles from now
    }
    pdl_trigger();  // not earlier: the next GEMM's CTAs would take the SMs that this grid leaves free, two to an SM
    bool finite = true;
#pragma unroll
    for (int rs = 0; rs < 2; ++rs) {
        float tot = l[rs];
        tot += __shfl_xor_sync(0xFFFFFFFFu, tot, 1);
        tot += __shfl_xor_sync(0xFFFFFFFFu, tot, 2);
        tot *= P_SCALE;
        finite = finite && isfinite(tot);
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) {
            finite = finite && isfinite(acc[j][2 * rs]) && isfinite(acc[j][2 * rs + 1]);
        }
        if (rows[rs] < m) {
            OutT* out = ctx + (int64_t)rows[rs] * n_heads * HD + head * HD + 2 * t;
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) {
                store_ctx(out + 8 * j, acc[j][2 * rs] / tot, acc[j][2 * rs + 1] / tot);
            }
        }
    }
    if (!__all_sync(0xFFFFFFFFu, finite)) {
        __syncwarp();  // the lanes' own stores of these rows come first
        attn_rows_again<HD>(qkv, row_stride, m, pos0, n_heads, n_kv, max_seq, cache_k, cache_v, ctx, row0 + 16 * warp, head);
    }
}

// A few rows at a time, where a 64-row tile of the kernel above would be mostly padding: one warp per four rows of a
// head.  Bound by the L2 reads of K and V (every row streams the whole prefix of its head).
template <int DPL, int ROWS, typename OutT>
__global__ void __launch_bounds__(128) attn_prefill_rows_kernel(const float* qkv, int row_stride, int m,
                                                                int pos0, int n_heads, int n_kv, int max_seq,
                                                                const __half* cache_k,
                                                                const __half* cache_v,
                                                                OutT* ctx)
{
    pdl_trigger();
    pdl_sync();
    const int groups = (m + ROWS - 1) / ROWS;
    const int64_t wid = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (wid < (int64_t)groups * n_heads) {
        // the longest rows first: the last CTAs to start are the shortest
        attn_rows<DPL, ROWS>(qkv, row_stride, m, pos0, n_heads, n_kv, max_seq, cache_k, cache_v, ctx,
                             (groups - 1 - (int)(wid / n_heads)) * ROWS, (int)(wid % n_heads));
    }
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename OutT>
cudaError_t attn_prefill(const float* qkv, int m, int pos0, int n_heads, int n_kv, int hd, int max_seq,
                         const __half* cache_k, const __half* cache_v, OutT* ctx, int rows_max, cudaStream_t st)
{
    const int row_stride = (n_heads + 2 * n_kv) * hd;
    if (m <= rows_max && (hd == 64 || hd == 128)) {
        constexpr int ROWS = 4;
        const unsigned ctas = (unsigned)(((m + ROWS - 1) / ROWS * n_heads + 3) / 4);
        auto kernel = hd == 64 ? attn_prefill_rows_kernel<2, ROWS, OutT> : attn_prefill_rows_kernel<4, ROWS, OutT>;
        return launch_pdl(kernel, dim3(ctas), dim3(128), 0, st, qkv, row_stride, m, pos0, n_heads, n_kv, max_seq, cache_k, cache_v,
                          ctx);
    }
    const dim3 grid((unsigned)((m + 63) / 64), (unsigned)n_heads);
    auto launch = [&](auto kernel) -> cudaError_t {
        const int smem = (4 * 64 + 3 * 64) * hd * 2;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            return e;
        }
        // not ahead of the kernel before: its 112 KB per CTA would keep that kernel's own CTAs waiting (128 tokens, four 7B-shape
        // blocks 733 us against 762)
        kernel<<<grid, 128, smem, st>>>(qkv, row_stride, m, pos0, n_heads, n_kv, max_seq, cache_k, cache_v, ctx);
        return cudaGetLastError();
    };
    return hd == 64    ? launch(attn_prefill_kernel<64, OutT>)
           : hd == 128 ? launch(attn_prefill_kernel<128, OutT>)
                       : cudaErrorInvalidValue;
}

// silu(gate) * up, packed for ffn_down, from gu[m][2*ffn], whose columns are the gate|up weight's rows: groups of 8 gate
// channels followed by the same 8 channels of up (the matvec's SwiGLU epilogue wants both halves of a channel in one
// 16-row tile).  A thread takes four neighbouring channels; grid (channels / 1024, rows).
__global__ void __launch_bounds__(256) silu_mul_rows_kernel(const float* __restrict__ gu, int ffn, RowOutPacked out)
{
    pdl_trigger();
    pdl_sync();
    const int i4 = blockIdx.x * 256 + threadIdx.x;
    const bool ok = 4 * i4 < ffn;
    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ok) {
        const float* p = gu + (int64_t)blockIdx.y * 2 * ffn + (i4 >> 1) * 16 + (i4 & 1) * 4;
        const float4 g = *reinterpret_cast<const float4*>(p), u = *reinterpret_cast<const float4*>(p + 8);
        o = make_float4((g.x * (1.0f / (1.0f + expf(-g.x)))) * u.x, (g.y * (1.0f / (1.0f + expf(-g.y)))) * u.y,
                        (g.z * (1.0f / (1.0f + expf(-g.z)))) * u.z, (g.w * (1.0f / (1.0f + expf(-g.w)))) * u.w);
    }
    out.put(blockIdx.y, i4, o, ok);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, int cluster, cudaStream_t stream,
                               Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace

cudaError_t ll_rope_tables(int max_seq, int rope_dim, double theta, float* rope_cos, float* rope_sin, cudaStream_t st)
{
    rope_table_kernel<<<64, 256, 0, st>>>(max_seq, rope_dim, theta, rope_cos, rope_sin);
    return cudaGetLastError();
}

cudaError_t ll_embed_rows(int fmt, const uint8_t* raw, const int* tokens, int n_rows, int d, float* h, cudaStream_t st)
{
    return launch_pdl(embed_row_kernel, dim3((d + 255) / 256, n_rows < 1024 ? n_rows : 1024), dim3(256), 0, st, fmt, raw, tokens,
                      n_rows, d, h);
}

cudaError_t ll_embed_pack(int fmt, const uint8_t* raw, const int* token, int d, const float* w, float* h,
                          uint8_t* packed, double* ss_out, cudaStream_t st)
{
    if ((d & 31) != 0) {
        return cudaErrorInvalidValue;
    }
    return launch_pdl(embed_pack_kernel, dim3((d / 32 + 3) / 4), dim3(128), 0, st, fmt, raw, token, d, w, h, packed, ss_out);
}

cudaError_t ll_resid_pack(const float* h_in, const float* add, const float* w, int d, float* h_out, uint8_t* packed,
                          double* ss_out, const PeerGather& pg, cudaStream_t st)
{
    if ((d & 31) != 0 || pg.tp_size > 8) {
        return cudaErrorInvalidValue;
    }
    const dim3 grid((d / 32 + 3) / 4), block(128);
    if (pg.tp_size > 1) {
        if (!add) {
            return cudaErrorInvalidValue;
        }
        return launch_pdl(resid_pack_kernel<true>, grid, block, 0, st, h_in, add, w, d, h_out, packed, ss_out, pg);
    }
    return launch_pdl(resid_pack_kernel<false>, grid, block, 0, st, h_in, add, w, d, h_out, packed, ss_out, pg);
}

cudaError_t ll_rope_kv(float* qkv, const int* pos, int pos_add, int rows, int n_heads, int n_kv, int hd, int rope_dim,
                       const float* rope_cos, const float* rope_sin, int max_seq, __half* cache_k, __half* cache_v,
                       cudaStream_t st)
{
    const int row_stride = (n_heads + 2 * n_kv) * hd;
    const int work = (n_heads + n_kv) * hd / 2 + n_kv * hd;
    return launch_pdl(rope_kv_kernel, dim3((work + 255) / 256, rows), dim3(256), 0, st, qkv, pos, pos_add, n_heads,
                      n_kv, hd, rope_dim, rope_cos, rope_sin, max_seq, cache_k, cache_v, row_stride);
}

cudaError_t ll_attn_fused(const float* qkv, const int* pos, int n_heads, int n_kv, int hd, int rope_dim,
                          const float* rope_cos, const float* rope_sin, int max_seq, __half* cache_k, __half* cache_v,
                          uint8_t* packed, int batch, const AttnBatch& ab, cudaStream_t st)
{
    const int chunks = (n_heads * hd + 255) / 256;
    const int cl = attn_cluster_for(batch);
    const dim3 grid(chunks * cl, batch), block(256);
#define QMM_ATTN_LAUNCH(DPL, CL)                                                                                         \
    return launch_pdl_cluster(attn_fused_kernel<DPL, CL>, grid, block, CL, st, qkv, pos, n_heads, n_kv, rope_dim, rope_cos, \
                              rope_sin, max_seq, cache_k, cache_v, packed, ab)
    if (hd == 64) {
        if (cl == 2) { QMM_ATTN_LAUNCH(2, 2); }
        if (cl == 4) { QMM_ATTN_LAUNCH(2, 4); }
        QMM_ATTN_LAUNCH(2, 8);
    }
    if (hd == 128) {
        if (cl == 2) { QMM_ATTN_LAUNCH(4, 2); }
        if (cl == 4) { QMM_ATTN_LAUNCH(4, 4); }
        QMM_ATTN_LAUNCH(4, 8);
    }
#undef QMM_ATTN_LAUNCH
    return cudaErrorInvalidValue;
}

cudaError_t ll_argmax(const float* logits, int n, int index_offset, int ctas, int* best_pair, int rows,
                      int64_t row_stride, cudaStream_t st)
{
    return launch_pdl(argmax_kernel, dim3(ctas, rows), dim3(1024), 0, st, logits, n, index_offset, best_pair, row_stride);
}

cudaError_t ll_commit_batch(const int* pairs, int per_rank, int ranks, int batch, int* tokens, int* pos, int* out_tokens,
                            int* out_steps, cudaStream_t st)
{
    if (batch < 1 || batch > 16) {
        return cudaErrorInvalidValue;
    }
    return launch_pdl(commit_batch_kernel, dim3(1), dim3(32 * batch), 0, st, pairs, per_rank, ranks, batch, tokens, pos,
                      out_tokens, out_steps);
}

cudaError_t ll_commit_token(const int* pairs, int n_local, const ArgmaxExchange& ax, int* token, int* pos,
                            int* out_tokens, int* out_count, const TokenReport& report, cudaStream_t st)
{
    if (ax.tp_size > 8) {
        return cudaErrorInvalidValue;
    }
    return launch_pdl(commit_token_kernel, dim3(1), dim3(32), 0, st, pairs, n_local, ax, token, pos, out_tokens, out_count,
                      report);
}

cudaError_t ll_resid_rmsnorm_rows(float* h, const float* add, const float* w, float eps, int d, int64_t m,
                                  __nv_bfloat16* xn, cudaStream_t st)
{
    return launch_pdl(resid_rmsnorm_rows_kernel<RowOutBf16>, dim3((unsigned)m), dim3(256), 0, st, h, add, w, eps, d,
                      RowOutBf16{xn, d});
}

cudaError_t ll_resid_rmsnorm_rows_packed(float* h, const float* add, const float* w, float eps, int d, int m,
                                         uint8_t* packed, cudaStream_t st)
{
    return launch_pdl(resid_rmsnorm_rows_kernel<RowOutPacked>, dim3((unsigned)m), dim3(256), 0, st, h, add, w, eps, d,
                      RowOutPacked{packed, m == 1 ? 0 : xpack_ncp(m)});
}

cudaError_t ll_attn_prefill(const float* qkv, int m, int pos0, int n_heads, int n_kv, int hd, int max_seq,
                            const __half* cache_k, const __half* cache_v, __nv_bfloat16* ctx, int rows_max,
                            cudaStream_t st)
{
    return attn_prefill(qkv, m, pos0, n_heads, n_kv, hd, max_seq, cache_k, cache_v, ctx, rows_max, st);
}

cudaError_t ll_silu_mul_rows_packed(const float* gu, int m, int ffn, uint8_t* packed, cudaStream_t st)
{
    const dim3 grid((unsigned)((ffn / 4 + 255) / 256), (unsigned)m);
    return launch_pdl(silu_mul_rows_kernel, grid, dim3(256), 0, st, gu, ffn,
                      RowOutPacked{packed, m == 1 ? 0 : xpack_ncp(m)});
}

}  // namespace qmm
