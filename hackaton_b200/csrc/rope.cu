// Rotary embedding + grouped-query expansion on the packed q / k / v projections, forward and
// backward in one launch each: the arithmetic of the reference's qkv_kernel
// (solution/attention.py:36-146).
//   forward : q, k rotated (fp32 arithmetic, one rounding to fp16); every k and v head written
//             REP = heads / kv_heads times, so that the attention that follows sees `heads` heads;
//             output rows either packed (N, heads, D) or padded (B, heads, T, D)
//   backward: the copies' gradients summed (fp32), the inverse rotation for q and k, written
//             packed (N, heads * D) in the projections' type
// with y1 = x1*c1 - x2*s1, y2 = x2*c2 + x1*s2 over the two halves of a head (c1/c2, s1/s2: the two
// halves of the cos / sin rows of the token's position).
// Many tokens: a work item is four q heads, or one k and one v head, of one token; dim / 16 threads share it, each with
// 8 consecutive elements of both halves (16-byte accesses for fp16). Its threads read the token's cos / sin
// row once for all its heads (as an item per head those rows, 1 KB of fp32 each, were more L1 traffic
// than the heads) and request all inputs of the q heads, or three copies' gradients, before using one.
// q items of all tokens come first, so that a CTA holds items of one kind. Pure streaming, HBM bound:
// 16,384 packed tokens, 12 / 2 heads of 128, 218 MB: forward 41.8 -> 36.7 us (0.91 of the copy
// bandwidth), backward 49.6 -> 38.8 (0.86); 28 / 4 heads 91.2 -> 80.9 and 104.8 -> 84.7.
#include <cuda_fp16.h>

#include "kernels.h"
#include "ptx.cuh"

namespace nf4 {

struct F8 {
    float v[8];
};

// Eight consecutive elements as they lie in memory, until they are used.
template <bool F32>
struct Raw8 {
    uint4 q[F32 ? 2 : 1];
    __device__ __forceinline__ void load(const void* p, long long idx) {
        const uint4* s = reinterpret_cast<const uint4*>(static_cast<const char*>(p) + idx * (F32 ? 4 : 2));
#pragma unroll
        for (int i = 0; i < (F32 ? 2 : 1); ++i) q[i] = __ldg(s + i);
    }
    __device__ __forceinline__ F8 get() const {
        F8 r;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(q);
#pragma unroll
        for (int i = 0; i < (F32 ? 8 : 4); ++i) {
            if (F32) {
                r.v[i] = __uint_as_float(w[i]);
            } else {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                r.v[(2 * i) % 8] = f.x;
                r.v[(2 * i + 1) % 8] = f.y;
            }
        }
        return r;
    }
};

template <bool F32>
__device__ __forceinline__ void rope_store8(void* p, long long idx, const F8& r) {
    if (F32) {
        float4* d = reinterpret_cast<float4*>(static_cast<float*>(p) + idx);
        d[0] = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
        d[1] = make_float4(r.v[4], r.v[5], r.v[6], r.v[7]);
    } else {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 h = __floats2half2_rn(r.v[2 * i], r.v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(static_cast<__half*>(p) + idx) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// a * b + sign * c * d, element by element
__device__ __forceinline__ F8 fma8(const F8& a, const F8& b, const F8& c, const F8& d, float sign) {
    F8 r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.v[i] = a.v[i] * b.v[i] + sign * (c.v[i] * d.v[i]);
    return r;
}

constexpr int ROPE_Q_HEADS = 4;   // q heads of a work item
constexpr int ROPE_COPIES = 3;    // copies of a k / v head whose loads are issued together in the backward

template <bool F32, bool BACKWARD, int CTAS>
__global__ void __launch_bounds__(256, CTAS)
qkv_rotate_kernel(const RopeArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    // 32-bit index arithmetic (the launcher checks that the thread count fits).
    const unsigned gid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned item = gid >> a.lps_shift;
    const int half = a.dim / 2;
    const int j = (int)(gid & ((1u << a.lps_shift) - 1u)) * 8;
    const unsigned q_parts = (unsigned)(a.heads + ROPE_Q_HEADS - 1) / ROPE_Q_HEADS;
    const unsigned q_items = (unsigned)a.tokens * q_parts;
    if (item >= q_items + (unsigned)a.tokens * (unsigned)a.kv_heads) return;
    const bool is_q = item < q_items;
    const unsigned parts = is_q ? q_parts : (unsigned)a.kv_heads;
    const unsigned rest = is_q ? item : item - q_items;
    const unsigned tok_u = rest / parts;
    const int part = (int)(rest - tok_u * parts);
    const long long tok = tok_u;
    const int b = a.b_idx[tok], t = a.t_idx[tok];
    // row (in units of heads) of output head h: packed (N, H, D) or padded (B, H, T, D)
    const long long head_base = a.padded ? (long long)b * a.heads * a.seq + t : tok * a.heads;
    const long long head_step = a.padded ? a.seq : 1;
    auto out_at = [&](int head) { return (head_base + head * head_step) * a.dim + j; };
    const long long cb = (long long)b * a.cos_stride_b + (long long)t * a.cos_stride_t;
    F8 c1, c2, s1, s2;
    auto load_angles = [&]() {
        Raw8<true> r[4];
        r[0].load(a.cos, cb + j); r[1].load(a.cos, cb + half + j);
        r[2].load(a.sin, cb + j); r[3].load(a.sin, cb + half + j);
        c1 = r[0].get(); c2 = r[1].get();
        s1 = r[2].get(); s2 = r[3].get();
    };
    if (is_q) {
        // all heads' loads go out before the first is used
        const int h0 = part * ROPE_Q_HEADS;
        Raw8<BACKWARD ? false : F32> x1[ROPE_Q_HEADS], x2[ROPE_Q_HEADS];
        const long long qi = tok * (long long)(a.heads * a.dim) + j;
#pragma unroll
        for (int i = 0; i < ROPE_Q_HEADS; ++i) {
            if (h0 + i >= a.heads) break;
            const long long at = BACKWARD ? out_at(h0 + i) : qi + (h0 + i) * a.dim;
            x1[i].load(a.q, at);
            x2[i].load(a.q, at + half);
        }
        load_angles();
#pragma unroll
        for (int i = 0; i < ROPE_Q_HEADS; ++i) {
            if (h0 + i >= a.heads) break;
            const F8 u = x1[i].get(), w = x2[i].get();
            if (!BACKWARD) {
                const long long at = out_at(h0 + i);
                rope_store8<false>(a.qo, at, fma8(u, c1, w, s1, -1.f));
                rope_store8<false>(a.qo, at + half, fma8(w, c2, u, s2, 1.f));
            } else {
                const long long at = qi + (h0 + i) * a.dim;
                rope_store8<F32>(a.qo, at, fma8(u, c1, w, s2, 1.f));
                rope_store8<F32>(a.qo, at + half, fma8(w, c2, u, s1, -1.f));
            }
        }
        return;
    }
    const int rep = a.heads / a.kv_heads, h0 = part * rep;
    const long long xi = tok * (long long)(a.kv_heads * a.dim) + part * a.dim + j;
    if (!BACKWARD) {
        Raw8<F32> k1, k2, v1, v2;
        k1.load(a.k, xi); k2.load(a.k, xi + half);
        v1.load(a.v, xi); v2.load(a.v, xi + half);
        load_angles();
        const F8 u = k1.get(), w = k2.get(), y1 = fma8(u, c1, w, s1, -1.f), y2 = fma8(w, c2, u, s2, 1.f);
        const F8 z1 = v1.get(), z2 = v2.get();
        for (int r = 0; r < rep; ++r) {
            const long long at = out_at(h0 + r);
            rope_store8<false>(a.ko, at, y1);
            rope_store8<false>(a.ko, at + half, y2);
            rope_store8<false>(a.vo, at, z1);
            rope_store8<false>(a.vo, at + half, z2);
        }
        return;
    }
    // backward: the copies' gradients summed in copy order, a few copies' loads ahead
    auto sum_copies = [&](const void* src, F8& d1, F8& d2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) d1.v[i] = d2.v[i] = 0.f;
        for (int r0 = 0; r0 < rep; r0 += ROPE_COPIES) {
            Raw8<false> u[ROPE_COPIES], w[ROPE_COPIES];
#pragma unroll
            for (int r = 0; r < ROPE_COPIES; ++r) {
                if (r0 + r >= rep) break;
                u[r].load(src, out_at(h0 + r0 + r));
                w[r].load(src, out_at(h0 + r0 + r) + half);
            }
#pragma unroll
            for (int r = 0; r < ROPE_COPIES; ++r) {
                if (r0 + r >= rep) break;
                const F8 f = u[r].get(), g = w[r].get();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    d1.v[i] += f.v[i];
                    d2.v[i] += g.v[i];
                }
            }
        }
    };
    F8 d1, d2;
    sum_copies(a.v, d1, d2);
    rope_store8<F32>(a.vo, xi, d1);
    rope_store8<F32>(a.vo, xi + half, d2);
    sum_copies(a.k, d1, d2);
    load_angles();
    rope_store8<F32>(a.ko, xi, fma8(d1, c1, d2, s2, 1.f));
    rope_store8<F32>(a.ko, xi + half, fma8(d2, c2, d1, s1, -1.f));
}

// Few tokens: an item per head (every q head, k head and v head of a token), so that the work spreads over
// more threads and no thread's chain is longer than one head's loads and stores.
constexpr int ROPE_SLOT_COPIES = 4;   // copies whose loads are issued together in the backward

template <bool F32, bool BACKWARD>
__global__ void __launch_bounds__(256, 4)
qkv_rotate_slot_kernel(const RopeArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    const int half = a.dim / 2;
    const unsigned gid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned item = gid >> a.lps_shift, slots = (unsigned)(a.heads + 2 * a.kv_heads);
    if (item >= (unsigned)a.tokens * slots) return;
    // Forward: a token's slots side by side. Backward: every token's q heads first, so that a CTA holds
    // items of one weight (k / v read all their copies).
    const unsigned q_items = (unsigned)a.tokens * (unsigned)a.heads;
    unsigned tok_u, slot_u;
    if (!BACKWARD) {
        tok_u = item / slots;
        slot_u = item - tok_u * slots;
    } else if (item < q_items) {
        tok_u = item / (unsigned)a.heads;
        slot_u = item - tok_u * (unsigned)a.heads;
    } else {
        const unsigned r = item - q_items, kv2 = 2u * (unsigned)a.kv_heads;
        tok_u = r / kv2;
        slot_u = (unsigned)a.heads + (r - tok_u * kv2);
    }
    const int j = (int)(gid & ((1u << a.lps_shift) - 1u)) * 8;
    const long long tok = tok_u;
    const int slot = (int)slot_u;
    const int b = a.b_idx[tok], t = a.t_idx[tok];
    const int rep = a.heads / a.kv_heads;
    const long long head_base = a.padded ? (long long)b * a.heads * a.seq + t : tok * a.heads;
    const long long head_step = a.padded ? a.seq : 1;
    auto out_at = [&](int head) { return (head_base + head * head_step) * a.dim + j; };
    auto load = [](const void* p, long long idx) {
        Raw8<BACKWARD ? false : F32> r;
        r.load(p, idx);
        return r.get();
    };
    const long long cb = (long long)b * a.cos_stride_b + (long long)t * a.cos_stride_t;
    F8 c1, c2, s1, s2;
    auto load_angles = [&]() {
        Raw8<true> r;
        r.load(a.cos, cb + j); c1 = r.get();
        r.load(a.cos, cb + half + j); c2 = r.get();
        r.load(a.sin, cb + j); s1 = r.get();
        r.load(a.sin, cb + half + j); s2 = r.get();
    };
    if (!BACKWARD && slot < a.heads + a.kv_heads) load_angles();
    if (slot < a.heads) {
        const long long xi = tok * (long long)(a.heads * a.dim) + slot * a.dim + j, yi = out_at(slot);
        if (!BACKWARD) {
            const F8 x1 = load(a.q, xi), x2 = load(a.q, xi + half);
            rope_store8<false>(a.qo, yi, fma8(x1, c1, x2, s1, -1.f));
            rope_store8<false>(a.qo, yi + half, fma8(x2, c2, x1, s2, 1.f));
        } else {
            const F8 d1 = load(a.q, yi), d2 = load(a.q, yi + half);
            load_angles();
            rope_store8<F32>(a.qo, xi, fma8(d1, c1, d2, s2, 1.f));
            rope_store8<F32>(a.qo, xi + half, fma8(d2, c2, d1, s1, -1.f));
        }
        return;
    }
    const bool is_k = slot < a.heads + a.kv_heads;
    const int head = slot - a.heads - (is_k ? 0 : a.kv_heads);
    const void* src = is_k ? a.k : a.v;
    void* dst = is_k ? a.ko : a.vo;
    const long long xi = tok * (long long)(a.kv_heads * a.dim) + head * a.dim + j;
    if (!BACKWARD) {
        const F8 x1 = load(src, xi), x2 = load(src, xi + half);
        const F8 y1 = is_k ? fma8(x1, c1, x2, s1, -1.f) : x1;
        const F8 y2 = is_k ? fma8(x2, c2, x1, s2, 1.f) : x2;
        for (int r = 0; r < rep; ++r) {
            rope_store8<false>(dst, out_at(head * rep + r), y1);
            rope_store8<false>(dst, out_at(head * rep + r) + half, y2);
        }
        return;
    }
    F8 d1, d2;
#pragma unroll
    for (int i = 0; i < 8; ++i) d1.v[i] = d2.v[i] = 0.f;
    for (int r0 = 0; r0 < rep; r0 += ROPE_SLOT_COPIES) {
        // the copies' loads go out together, the sums follow in copy order
        Raw8<false> u[ROPE_SLOT_COPIES], w[ROPE_SLOT_COPIES];
#pragma unroll
        for (int r = 0; r < ROPE_SLOT_COPIES; ++r) {
            u[r].q[0] = w[r].q[0] = make_uint4(0u, 0u, 0u, 0u);
            if (r0 + r < rep) {
                u[r].load(src, out_at(head * rep + r0 + r));
                w[r].load(src, out_at(head * rep + r0 + r) + half);
            }
        }
#pragma unroll
        for (int r = 0; r < ROPE_SLOT_COPIES; ++r) {
            if (r0 + r < rep) {
                const F8 f = u[r].get(), g = w[r].get();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    d1.v[i] += f.v[i];
                    d2.v[i] += g.v[i];
                }
            }
        }
    }
    if (is_k) load_angles();
    rope_store8<F32>(dst, xi, is_k ? fma8(d1, c1, d2, s2, 1.f) : d1);
    rope_store8<F32>(dst, xi + half, is_k ? fma8(d2, c2, d1, s1, -1.f) : d2);
}

// Few enough tokens for an item per head? In waves of its threads (four CTAs per SM): forward up to four, two where
// k and v are not copied; backward, where an item reads all copies in a row, one, two with fp32 gradients. us, an
// item per head against the kernel above: forward, q / kv heads 12 / 2, fp16, 256 tokens 2.2 / 3.7, 1024 3.8 / 5.1,
// 2048 6.0 / 7.6, 4096 10.1 / 10.2, 6000 14.6 / 13.2; 28 / 4, 512 4.1 / 5.0, 2048 11.5 / 12.4, 3000 17.8 / 15.4; 16 /
// 16, 512 4.1 / 4.5, 1024 6.7 / 6.2. Forward and backward together 12 / 2, 64 tokens 4.7 / 6.9, 1024 8.3 / 8.9, 3000
// 17.4 / 15.9; 28 / 4, 512 8.7 / 10.2, 3000 41.7 / 35.4; fp32 projections 12 / 2, 2048 15.0 / 15.6.
static bool rope_few(const RopeArgs& a) {
    const long long threads = a.tokens * (a.heads + 2 * a.kv_heads) * (a.dim / 16);
    const int waves = a.backward ? (a.proj_f32 ? 2 : 1) : (a.heads > a.kv_heads ? 4 : 2);
    return threads <= (long long)waves * a.sm_count * 4 * 256;
}

template <bool F32, bool BACKWARD, int CTAS>
static cudaError_t launch_rotate(RopeArgs a, cudaStream_t stream) {
    const int lps = a.dim / 16;   // threads per work item: 8 elements of each half
    a.lps_shift = 0;
    while ((1 << a.lps_shift) < lps) ++a.lps_shift;
    const long long slots = a.tokens * (a.heads + 2 * a.kv_heads) * lps;
    // (the limit of the 32-bit indices with an item per head)
    if ((1 << a.lps_shift) != lps || slots >= (1ll << 31)) return cudaErrorInvalidValue;
    if (rope_few(a))
        return launch_pdl(qkv_rotate_slot_kernel<F32, BACKWARD>, dim3((unsigned)((slots + 255) / 256)), dim3(256), 0,
                          stream, a);
    const long long threads =
        a.tokens * ((a.heads + ROPE_Q_HEADS - 1) / ROPE_Q_HEADS + a.kv_heads) * lps;
    return launch_pdl(qkv_rotate_kernel<F32, BACKWARD, CTAS>, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0,
                      stream, a);
}

cudaError_t launch_qkv_rotate(const RopeArgs& a, cudaStream_t stream) {
    if (a.tokens <= 0) return cudaSuccess;
    // Three CTAs per SM (80 registers, a few spilled) keep the most loads in flight; two (no spills) are
    // better where a forward item holds fp32 loads (8192 tokens of fp32 projections 25.3 us against 29.5).
    if (a.backward)
        return a.proj_f32 ? launch_rotate<true, true, 3>(a, stream) : launch_rotate<false, true, 3>(a, stream);
    return a.proj_f32 ? launch_rotate<true, false, 2>(a, stream) : launch_rotate<false, false, 3>(a, stream);
}

}  // namespace nf4
