// NF4 linear for a handful of token rows (the decode shapes of serving), both directions:
//   forward  (M <= 64): out_i[M, N_i] = act[M, K] . W_i^T (+ bias_i) (+ ext_a_i . ext_b_i^T)
//   backward (M <= 16): out[M, K]     = sum_i act_i[M, N_i] . W_i  (+ ext_a_i . ext_b_i)
// for a group of up to four weights that share K (forward: they also share the activations; gate and
// up can leave as silu(gate) * up).
// At these sizes the work is reading the packed weights once (0.52 B per weight); a 128-row
// tensor-core tile would be 50-99 % padding and the persistent tcgen05 kernel's set-up and
// epilogue would dominate. So: no TMEM. Warps bring the codes into private rings in shared memory,
// expand them and multiply with warp-level mma.sync (m16n8k16, fp32 accumulate).
//
// Forward: a warp owns 16 or 32 weight rows of one member of the group and a slice of the 64-deep
// k-blocks. The contraction index is visited in a permuted order that A (weights) and B (tokens)
// share, so a thread's 16 consecutive weights and 16 consecutive activations feed four k16 steps
// without any shuffle. A byte of codes is expanded by one look-up in a byte -> fp16-pair table, and
// the block scale is applied to each k-block's fp32 sums (one rounding less than scaling weights).
// The warps' partial tiles are added through shared memory; bias, the rank-16 LoRA term and the
// SwiGLU product are applied there.
// What bounds it: the L1 / shared-memory pipe (per 16 rows x 64 weights: 16 wavefronts of look-ups,
// 8 of codes through the ring, 2 of scales, 2 to 32 of activations) and, with few k-blocks per warp,
// the launch itself (1.65 us for an empty kernel in a chain). Measured in CUDA graphs over rotating
// layers, us per layer (q/k/v, o, gate / up + product, down), before (codes loaded straight into
// registers, table look-ups with bank conflicts or by byte permutes, product as a kernel of its own)
// -> now: 1536-wide network, 1 row 28.9 -> 18.6, 16 rows 32.6 -> 25.2, 32 rows 51.8 -> 36.4;
// 3584-wide, 1 row 87 -> 53, 16 rows 94.5 -> 66.7, 32 rows 125.6 -> 96.4. The weights alone
// at the copy bandwidth: 3.7 and 18.4 us.
//
// Backward: the contraction runs over weight rows, along which the codes are NOT contiguous. A
// warp owns one k-block (64 output columns) and a slab of weight rows; per step of 16 rows lane
// (g, t) decodes one 32-bit word (8 columns: word g of the k-block) of rows 2t, 2t+1, 2t+8, 2t+9
// and issues eight MMAs, one per column position c of its word: in MMA c the B operand's column
// g is "column c of word g", so the fragment a thread needs (two consecutive contraction rows of
// one column) is a byte-permute of two of its own decoded words. A (the upstream gradient,
// row-major over the contraction) is loaded as plain fragments. A thread ends up with 16
// consecutive output columns of tokens g and g + 8. Row slabs are summed in two steps: the
// warps of a CTA through shared memory, the CTAs of a k-block as fp32 planes in caller-provided
// scratch, which the last CTA of the k-block to finish (a ticket counter) adds in slab order
// (deterministic) and writes out as fp16.
//
// Both kernels ask for their slab of codes to be brought into L2 before they wait for the
// previous kernel of the stream (programmatic dependent launch): a prefetch reads no values, so
// it needs no ordering, and in a chain of small launches the weights of launch i + 1 travel
// from HBM while launch i runs.
//
// Both need the ready-made fp16 block-scale table (kernels.h, launch_prepare_scales) and
// N % 16 == 0; other calls take the tcgen05 kernel.
#include <cuda_fp16.h>

#include <atomic>

#include "decode.cuh"
#include "kernels.h"
#include "ptx.cuh"
#include "swiglu.cuh"

namespace nf4 {

constexpr int GV_ROWS = 16;
constexpr int GV_MAXP = GEMM_MAX_GROUP;
constexpr int GV_MAX_SMEM = 227 * 1024;

struct GemvProblem {
    const uint8_t* codes;
    const __half* scales16;  // [K / 64][N]
    const float* code16;
    const __half* bias;
    const __half* ext_a;     // forward: [M, 16] or null; backward: u [M, 16] or null
    const __half* ext_b;     // forward: lora_b [N, 16]; backward: lora_a [16, K]
    const __half* act;       // backward: this member's dY [M, N]
    __half* out;             // forward: this member's output
    long long ld_out, ld_act;
    int n_w;
    int first;               // forward: first set of this member; backward: first row slab
    int tiles;               // forward: tiles of this member
};

struct GemvParams {
    GemvProblem prob[GV_MAXP];
    const __half* act;       // forward: shared activations
    long long ld_act;
    float* planes;           // backward: [slabs][M][ldp] fp32
    long long ldp;
    int n_prob, m, k_w;
    int split_log, n_sets;   // forward: log2(warps per tile), CTA-sized sets of tiles of the whole group
    __half* hidden;          // forward with SwiGLU: the product
    int rows_per_slab;       // backward: weight rows per CTA (multiple of 16 * warps)
    int ticket_base;         // backward: first ticket of this launch, or -1 (reduction by a second kernel)
    int n_slabs;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The same with a zero accumulator going in (first step of a k-block whose sums are scaled
// afterwards).
__device__ __forceinline__ void mma_16816_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                uint32_t a3, uint32_t b0, uint32_t b1) {
    const float z = 0.f;
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(z));
}

// Forward decode by byte: a 256-entry table in shared memory maps a byte of codes to its two
// unscaled fp16 table values (first weight = high nibble in the low half). It is kept once per
// bank (lane l reads copy l), so a warp's 32 look-ups are one conflict-free wavefront. Where gate and
// up are multiplied together their two tables share 256-byte entries.
// The table sits at a fixed shared-memory address, so that the base is an immediate of the load:
// behind the 1 KB that the system reserves at the start of a block's shared memory (the kernel
// has no static shared memory, so its dynamic part starts right there).
constexpr uint32_t PAIR_AT = 2048;

// The table is written again when a CTA walks on to another member, so the compiler has to know that a look-up
// reads memory. IN_ORDER: volatile, which also keeps the look-ups in program order; an ordinary load may be moved
// between the barriers. A decode step of the 3584-wide network at 16 tokens (4 layers) takes 519 us in order and
// 534 with ordinary loads, one of the 1536-wide network at 32 tokens (10 layers) 529 and 518.
template <bool IN_ORDER>
__device__ __forceinline__ uint32_t pair_lookup(uint32_t offset) {
    if (!IN_ORDER) return *static_cast<const uint32_t*>(__cvta_shared_to_generic(offset + PAIR_AT));
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(offset), "n"(PAIR_AT));
    return v;
}

__device__ __forceinline__ RegLut load_reg_lut(const float* code16) {
    uint16_t bits[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) bits[i] = __half_as_ushort(__float2half_rn(__ldg(code16 + i)));
    return make_reg_lut(bits);
}

__device__ __forceinline__ int gemv_find(const GemvParams& p, int idx) {
    int r = 0;
#pragma unroll
    for (int i = 1; i < GV_MAXP; ++i)
        if (i < p.n_prob && idx >= p.prob[i].first) r = i;
    return r;
}

// Asks for `bytes` starting at `ptr` (16-byte aligned, multiple of 16) to be brought into L2, in
// pieces the bulk-prefetch instruction takes.
__device__ __forceinline__ void prefetch_span(const uint8_t* ptr, long long bytes) {
    constexpr long long PIECE = 32768;
    for (long long off = 0; off < bytes; off += PIECE) {
        const long long n = bytes - off < PIECE ? bytes - off : PIECE;
        bulk_prefetch_l2(ptr + off, (uint32_t)n);
    }
}

// Forward. A warp tile is MT * 16 weight rows of one member of the group (SWIGLU: the same 16 rows
// of gate and of up) times up to 32 tokens; 2^split_log warps share a tile, each with a contiguous
// slice of its k-blocks, and a CTA (of 16, 8 or 4 warps) holds the other tiles of a set. Every warp brings its
// own codes and scales through a private ring in shared memory (cp.async), laid out [k-block][row]
// [32 bytes], from which its fragments (rows g, g + 8; 8 bytes each) are read without conflicts: a
// direct load of such a fragment touches eight lines, which cost as much of the L1 pipe as the
// look-ups.
template <int NT, int MT, bool SWIGLU, int WL>
struct GemvShape {
    static constexpr int WARPS = 1 << WL, THREADS = WARPS * 32;
    static constexpr int KBS = MT == 1 ? 4 : 2;        // k-blocks per ring stage
    static constexpr int STAGES = NT == 1 && MT == 1 ? 3 : 2;
    static constexpr int SLOT = 2048 + 128;            // codes and scales of a stage: MT * KBS * (512 + 32)
    static constexpr int RING = STAGES * SLOT;         // per warp
    static constexpr int ROWS = GV_ROWS * MT;
    static constexpr int STRIDE = SWIGLU ? 256 : 128;  // bytes per table entry
    static constexpr int TABLE_BYTES = 256 * STRIDE;
    static constexpr int RED_BYTES = WARPS * NT * 8 * (ROWS + 1) * 4;   // takes the rings' place
    static constexpr int RINGS_BYTES = WARPS * RING;
    static constexpr int FIXED_BYTES = TABLE_BYTES + (RED_BYTES > RINGS_BYTES ? RED_BYTES : RINGS_BYTES);
};

// XS: the activations are staged in shared memory
template <int NT, int MT, bool SWIGLU, bool XS, int WL>
__global__ void __launch_bounds__(32 << WL, NT * MT == 1 || WL == 3 ? 2 : 1)
nf4_gemv_kernel(const __grid_constant__ GemvParams p) {
    using Shape = GemvShape<NT, MT, SWIGLU, WL>;
    constexpr int KBS = Shape::KBS, ROWS = Shape::ROWS, STAGES = Shape::STAGES;
    static_assert(!SWIGLU || MT == 2, "gate and up rows are the two row blocks of a tile");
    extern __shared__ __align__(256) uint8_t smem[];
    uint8_t* const table = smem + (PAIR_AT - (uint32_t)__cvta_generic_to_shared(smem));
    float (*red)[NT * 8][ROWS + 1] = reinterpret_cast<float (*)[NT * 8][ROWS + 1]>(table + Shape::TABLE_BYTES);
    __half* xs = reinterpret_cast<__half*>(table + Shape::FIXED_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t row_bytes = (uint32_t)p.k_w >> 1;
    const int nkb = p.k_w >> 6;
    const int slots_log = WL - p.split_log, slots = 1 << slots_log;  // tiles of a set
    const int slot = warp >> p.split_log, slice = warp & ((1 << p.split_log) - 1);
    const int kb_begin = (nkb * slice) >> p.split_log, kb_end = (nkb * (slice + 1)) >> p.split_log;

    // A set's tiles belong to one member (SWIGLU: to gate and up alike). Member of a set, weight of
    // row block mt, first row of row block mt of a tile:
    auto member_of = [&](int set) { return SWIGLU ? 0 : gemv_find(p, set); };
    auto problem = [&](int pi, int mt) -> const GemvProblem& { return p.prob[SWIGLU ? mt : pi]; };
    auto row_of = [&](int tile, int mt) { return SWIGLU ? tile * GV_ROWS : tile * ROWS + mt * GV_ROWS; };
    // On their way to L2 while the previous kernel of the stream is still running: the rows of codes
    // of a tile (one contiguous span) and its block scales (a 32-byte piece per k-block).
    {
        const int pi = member_of((int)blockIdx.x);
        const int tile0 = ((int)blockIdx.x - problem(pi, 0).first) << slots_log;
        const int valid = problem(pi, 0).tiles - tile0;
        if ((int)threadIdx.x < slots * MT) {
            const int sl = (int)threadIdx.x / MT, mt = (int)threadIdx.x % MT;
            if (sl < valid)
                prefetch_span(problem(pi, mt).codes + (size_t)row_of(tile0 + sl, mt) * row_bytes,
                              (long long)GV_ROWS * row_bytes);
        }
        if (slot < valid) {
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const GemvProblem& pr = problem(pi, mt);
                for (int kb = kb_begin + lane; kb < kb_end; kb += 32)
                    prefetch_l2(pr.scales16 + (size_t)kb * pr.n_w + row_of(tile0 + slot, mt));
            }
        }
    }
    grid_dep_wait();
    grid_dep_launch();

    // the tokens of this CTA (blockIdx.y: blocks of NT * 8)
    const int token0 = (int)blockIdx.y * NT * 8, tokens = min(p.m - token0, NT * 8);
    const __half* const act = p.act + token0 * p.ld_act;
    const uint32_t lane4 = lane * 4;
    auto pairs = [&](int mt, uint32_t w, uint32_t (&o)[8], int at) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            o[at + i] = pair_lookup<NT <= 2>(SWIGLU ? __byte_perm(w, lane4 + mt * 128, 0x7604u + (i << 4))
                                                    : __byte_perm(w, 0u, 0x4440u + i) * 128u + lane4);
    };
    const uint32_t ring = PAIR_AT + Shape::TABLE_BYTES + warp * Shape::RING;   // shared-memory address
    const uint8_t* const ring_ptr = table + Shape::TABLE_BYTES + warp * Shape::RING;

    int built = -1;   // the member whose pair table is in place
    for (int set = (int)blockIdx.x; set < p.n_sets; set += (int)gridDim.x) {
        const int pi = member_of(set);
        const int tile0 = (set - problem(pi, 0).first) << slots_log, tile = tile0 + slot;
        const bool build = pi != built;
        // the two table values of this thread's table entry: their loads share the first round trip
        constexpr int ENTRIES = 512 / Shape::THREADS;   // table entries (halves of, where SWIGLU) per thread
        const GemvProblem& tp = problem(pi, SWIGLU ? (threadIdx.x & 1) : 0);
        float code_hi[ENTRIES], code_lo[ENTRIES];
        if (build) {
#pragma unroll
            for (int i = 0; i < ENTRIES; ++i) {
                const int entry = (threadIdx.x + i * Shape::THREADS) >> 1;
                code_hi[i] = __ldg(tp.code16 + (entry >> 4));
                code_lo[i] = __ldg(tp.code16 + (entry & 15));
            }
        }
        if (XS && set == (int)blockIdx.x) {   // staged once, read by every warp
            const int chunks = p.k_w / 8;
            for (int token = 0; token < tokens; ++token) {
                const __half* src = act + (long long)token * p.ld_act;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs) + token * (p.k_w + 8) * 2;
                for (int c = threadIdx.x; c < chunks; c += Shape::THREADS) cp_async16(dst + c * 16, src + c * 8);
            }
        }
        cp_async_commit();

        const int count = tile < problem(pi, 0).tiles ? kb_end - kb_begin : 0;
        // Ring stage: lane = (row, 16-byte chunk) of KBS k-blocks (byte offsets: a member's codes are
        // below 4 GB); the first 8 lanes bring the scales, 16 bytes each.
        constexpr int CHUNKS = KBS * 2, ROWS_PER = 32 / CHUNKS;
        const int c_row = lane / CHUNKS, c_at = lane % CHUNKS;
        const uint32_t c_dst = (c_at >> 1) * 512 + c_row * 32 + (c_at & 1) * 16;
        const uint8_t* c_src[MT];
        uint32_t c_off[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            c_src[mt] = problem(pi, mt).codes;
            c_off[mt] = (uint32_t)(row_of(tile, mt) + c_row) * row_bytes + kb_begin * 32 + c_at * 16;
        }
        const int s_mt = lane / CHUNKS, s_kb = c_at >> 1;   // lanes 0 .. CHUNKS * MT - 1 = 0 .. 7
        const GemvProblem& sp = problem(pi, s_mt < MT ? s_mt : 0);
        const uint8_t* const s_src = reinterpret_cast<const uint8_t*>(
            sp.scales16 + (size_t)(kb_begin + s_kb) * sp.n_w + row_of(tile, s_mt)) + (c_at & 1) * 16;
        const uint32_t s_step = 2 * (uint32_t)sp.n_w;
        auto fill = [&](int i0, uint32_t at) {   // k-blocks i0 .. i0 + KBS - 1 of the slice
            if (i0 + (c_at >> 1) < count) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int r = 0; r < GV_ROWS / ROWS_PER; ++r)
                        cp_async16(at + mt * (KBS * 512) + c_dst + r * (ROWS_PER * 32),
                                   c_src[mt] + (c_off[mt] + i0 * 32 + r * ROWS_PER * row_bytes));
                if (lane < CHUNKS * MT)
                    cp_async16(at + 2048 + s_mt * (KBS * 32) + s_kb * 32 + (c_at & 1) * 16,
                               s_src + (size_t)i0 * s_step);
            }
            cp_async_commit();
        };
#pragma unroll
        for (int st = 0; st < STAGES - 1; ++st) fill(st * KBS, ring + st * Shape::SLOT);

        if (build) {
            // the 32 copies of an entry: by one thread per table, or half of them by each of the two;
            // 16-byte stores rotated over the banks
#pragma unroll
            for (int i = 0; i < ENTRIES; ++i) {
                const int entry = (threadIdx.x + i * Shape::THREADS) >> 1;
                const uint32_t pair = (uint32_t)__half_as_ushort(__float2half_rn(code_hi[i])) |
                                      ((uint32_t)__half_as_ushort(__float2half_rn(code_lo[i])) << 16);
                const uint4 v = make_uint4(pair, pair, pair, pair);
                uint4* dst = reinterpret_cast<uint4*>(table + entry * Shape::STRIDE) + (SWIGLU ? (threadIdx.x & 1) * 8 : 0);
                constexpr int STORES = SWIGLU ? 8 : 4;
                const int at = SWIGLU ? 0 : (threadIdx.x & 1) * 4;
#pragma unroll
                for (int j = 0; j < STORES; ++j) dst[at + ((j + entry) & (STORES - 1))] = v;
            }
            built = pi;
        }
        float acc[MT][NT][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
                acc[mt][nt][0] = acc[mt][nt][1] = acc[mt][nt][2] = acc[mt][nt][3] = 0.f;
        // Token nt * 8 + g, this thread's 16 columns of a k-block (tokens past the last one read the
        // last one's row again: their sums are not written).
        const long long x_ld = XS ? p.k_w + 8 : p.ld_act;
        const __half* x_at[NT];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
            x_at[nt] = (XS ? xs : act) + min(nt * 8 + g, tokens - 1) * x_ld + kb_begin * 64 + t * 16;
        cp_async_wait<STAGES - 1>();   // the staged activations
        __syncthreads();

        int read = 0, write = STAGES - 1;   // ring stages
        for (int i0 = 0; i0 < count; i0 += KBS) {
            cp_async_wait<STAGES - 2>();
            __syncwarp();      // the stage has landed for all lanes, and all have left the one before it
            fill(i0 + (STAGES - 1) * KBS, ring + write * Shape::SLOT);
            const uint8_t* const st = ring_ptr + read * Shape::SLOT;
            write = write + 1 == STAGES ? 0 : write + 1;
            read = read + 1 == STAGES ? 0 : read + 1;
#pragma unroll
            for (int j = 0; j < KBS; ++j) {
                if (i0 + j >= count) break;
                uint32_t wl[MT][8], wh[MT][8];
                float f_lo[MT], f_hi[MT];
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const uint8_t* c = st + (mt * KBS + j) * 512 + g * 32 + t * 8;
                    const uint2 lo = *reinterpret_cast<const uint2*>(c);
                    const uint2 hi = *reinterpret_cast<const uint2*>(c + 256);
                    const __half* sc = reinterpret_cast<const __half*>(st + 2048 + (mt * KBS + j) * 32) + g;
                    f_lo[mt] = __half2float(sc[0]);
                    f_hi[mt] = __half2float(sc[8]);
                    pairs(mt, lo.x, wl[mt], 0); pairs(mt, lo.y, wl[mt], 4);
                    pairs(mt, hi.x, wh[mt], 0); pairs(mt, hi.y, wh[mt], 4);
                }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    // the same 16 k of the token: k16 step j takes words 2j, 2j+1 of both operands
                    const uint4* xp = reinterpret_cast<const uint4*>(x_at[nt] + (i0 + j) * 64);
                    const uint4 x0 = xp[0], x1 = xp[1];
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        // unscaled sums of this k-block, then the rows' block scales (d0, d1: row g;
                        // d2, d3: row g + 8)
                        float blk[4];
                        mma_16816_first(blk, wl[mt][0], wh[mt][0], wl[mt][1], wh[mt][1], x0.x, x0.y);
                        mma_16816(blk, wl[mt][2], wh[mt][2], wl[mt][3], wh[mt][3], x0.z, x0.w);
                        mma_16816(blk, wl[mt][4], wh[mt][4], wl[mt][5], wh[mt][5], x1.x, x1.y);
                        mma_16816(blk, wl[mt][6], wh[mt][6], wl[mt][7], wh[mt][7], x1.z, x1.w);
                        acc[mt][nt][0] = fmaf(f_lo[mt], blk[0], acc[mt][nt][0]);
                        acc[mt][nt][1] = fmaf(f_lo[mt], blk[1], acc[mt][nt][1]);
                        acc[mt][nt][2] = fmaf(f_hi[mt], blk[2], acc[mt][nt][2]);
                        acc[mt][nt][3] = fmaf(f_hi[mt], blk[3], acc[mt][nt][3]);
                    }
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();   // the rings are idle: their place is the fold's
        // accumulator fragment: d0,d1 -> (weight row g, tokens 2t, 2t+1); d2,d3 -> (row g+8, same)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                red[warp][nt * 8 + 2 * t][mt * 16 + g] = acc[mt][nt][0];
                red[warp][nt * 8 + 2 * t + 1][mt * 16 + g] = acc[mt][nt][1];
                red[warp][nt * 8 + 2 * t][mt * 16 + g + 8] = acc[mt][nt][2];
                red[warp][nt * 8 + 2 * t + 1][mt * 16 + g + 8] = acc[mt][nt][3];
            }
        __syncthreads();
        constexpr int OUT_ROWS = SWIGLU ? GV_ROWS : ROWS;   // a power of two, like the slots
        const GemvProblem& pr = problem(pi, 0);
        for (int e = threadIdx.x; e < (tokens * OUT_ROWS) << slots_log; e += Shape::THREADS) {
            const int r = e % OUT_ROWS, sl = (e / OUT_ROWS) & (slots - 1), tok = (e / OUT_ROWS) >> slots_log;
            const int token = token0 + tok, w0 = sl << p.split_log;
            if (tile0 + sl >= pr.tiles) continue;
            float v = 0.f, u = 0.f;
#pragma unroll 4
            for (int w = 0; w < (1 << p.split_log); ++w) {
                v += red[w0 + w][tok][r];
                if (SWIGLU) u += red[w0 + w][tok][(GV_ROWS + r) % ROWS];
            }
            const int row = row_of(tile0 + sl, 0) + r;
            if (SWIGLU) {
                const __half hg = __float2half_rn(v), hu = __float2half_rn(u);
                const long long at = (long long)token * pr.ld_out + row;
                if (pr.out != nullptr) {
                    pr.out[at] = hg;
                    p.prob[1].out[at] = hu;
                }
                const float gf = __half2float(hg);
                p.hidden[at] = __float2half_rn(gf * sigmoid_fast(gf) * __half2float(hu));
                continue;
            }
            if (pr.ext_a != nullptr) {
                const __half2* xa = reinterpret_cast<const __half2*>(pr.ext_a + (long long)token * 16);
                const __half2* lb = reinterpret_cast<const __half2*>(pr.ext_b + (long long)row * 16);
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float2 a = __half22float2(__ldg(xa + j)), b = __half22float2(__ldg(lb + j));
                    s = fmaf(a.x, b.x, s);
                    s = fmaf(a.y, b.y, s);
                }
                v += s;
            }
            if (pr.bias != nullptr) v += __half2float(__ldg(pr.bias + row));
            pr.out[(long long)token * pr.ld_out + row] = __float2half_rn(v);
        }
        if (set + (int)gridDim.x < p.n_sets) __syncthreads();   // `red` is free again
    }
}

// ------------------------------------------------------------------------------------ backward

constexpr int GB_BATCH = 4;   // 16-row steps whose loads are in flight together

// One ticket per k-block of a launch in flight: the CTA that takes the last ticket of its k-block
// adds the slabs' planes and writes the result, so small problems need no second kernel. The
// tickets start at zero (module load) and the last arriver puts its ticket back to zero. Launches
// get their span of tickets in turn; TICKET_LAUNCHES launches may be in flight at once.
constexpr int TICKET_LAUNCHES = 64, TICKET_SPAN = 512;
__device__ unsigned g_gemv_tickets[TICKET_LAUNCHES * TICKET_SPAN];

// grid = (k-blocks, row slabs over the whole group); a CTA's warps take the 16-row steps of its
// slab in turn. The slab's sums go to an fp32 plane; the split-K reduction kernel adds the planes.
template <int GB_WARPS>
__global__ void __launch_bounds__(GB_WARPS * 32)
nf4_gemv_bwd_kernel(const __grid_constant__ GemvParams p) {
    const int kb = (int)blockIdx.x;
    const int slab = (int)blockIdx.y;
    const int pi = gemv_find(p, slab);
    const GemvProblem& pr = p.prob[pi];
    const int row0 = (slab - pr.first) * p.rows_per_slab;          // first row of the slab
    const int row_end = min(row0 + p.rows_per_slab, pr.n_w);
    const size_t row_bytes = (size_t)p.k_w >> 1;
    grid_dep_wait();
    grid_dep_launch();
    __shared__ float red[GB_WARPS][16][64 + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;

    const RegLut lut = load_reg_lut(pr.code16);
    float acc[8][4];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;

    // this lane's word of the k-block: columns kb*64 + 8g .. + 7
    const uint8_t* cbase = pr.codes + (size_t)kb * 32 + (size_t)g * 4;
    const __half* sbase = pr.scales16 + (size_t)kb * pr.n_w;
    const __half* a_lo = pr.act + (long long)g * pr.ld_act;        // token g
    const __half* a_hi = pr.act + (long long)(g + 8) * pr.ld_act;  // token g + 8
    const bool lo_ok = g < p.m, hi_ok = g + 8 < p.m;

    const int n_steps = (row_end - row0 + 15) / 16;   // n_w % 16 == 0: whole steps
    for (int s0 = warp * GB_BATCH; s0 < n_steps; s0 += GB_WARPS * GB_BATCH) {
        uint32_t code[GB_BATCH][4];
        uint32_t sc[GB_BATCH][2], av[GB_BATCH][4];
#pragma unroll
        for (int b = 0; b < GB_BATCH; ++b) {
            const int st = min(s0 + b, n_steps - 1);              // (tail: re-read, unused)
            const int n = row0 + st * 16 + 2 * t;                 // rows n, n+1, n+8, n+9
            const uint8_t* c0 = cbase + (size_t)n * row_bytes;
            code[b][0] = __ldg(reinterpret_cast<const uint32_t*>(c0));
            code[b][1] = __ldg(reinterpret_cast<const uint32_t*>(c0 + row_bytes));
            code[b][2] = __ldg(reinterpret_cast<const uint32_t*>(c0 + 8 * row_bytes));
            code[b][3] = __ldg(reinterpret_cast<const uint32_t*>(c0 + 9 * row_bytes));
            sc[b][0] = __ldg(reinterpret_cast<const uint32_t*>(sbase + n));      // scales of n, n+1
            sc[b][1] = __ldg(reinterpret_cast<const uint32_t*>(sbase + n + 8));  // of n+8, n+9
            av[b][0] = lo_ok ? __ldg(reinterpret_cast<const uint32_t*>(a_lo + n)) : 0u;
            av[b][1] = hi_ok ? __ldg(reinterpret_cast<const uint32_t*>(a_hi + n)) : 0u;
            av[b][2] = lo_ok ? __ldg(reinterpret_cast<const uint32_t*>(a_lo + n + 8)) : 0u;
            av[b][3] = hi_ok ? __ldg(reinterpret_cast<const uint32_t*>(a_hi + n + 8)) : 0u;
        }
#pragma unroll
        for (int b = 0; b < GB_BATCH; ++b) {
            if (s0 + b >= n_steps) break;
            uint32_t w[4][4];   // w[row][pair]: columns (2j, 2j+1) of the word, scaled
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t s32 = sc[b][r >> 1];
                const uint32_t dup = (r & 1) ? __byte_perm(s32, 0u, 0x3232u) : __byte_perm(s32, 0u, 0x1010u);
                const uint4 d = decode_word_reg(code[b][r], lut, *reinterpret_cast<const __half2*>(&dup));
                w[r][0] = d.x; w[r][1] = d.y; w[r][2] = d.z; w[r][3] = d.w;
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint32_t sel = (c & 1) ? 0x7632u : 0x5410u;
                const uint32_t b0 = __byte_perm(w[0][c >> 1], w[1][c >> 1], sel);  // rows n, n+1
                const uint32_t b1 = __byte_perm(w[2][c >> 1], w[3][c >> 1], sel);  // rows n+8, n+9
                mma_16816(acc[c], av[b][0], av[b][1], av[b][2], av[b][3], b0, b1);
            }
        }
    }

    // acc[c]: d0,d1 -> (token g, words 2t, 2t+1); d2,d3 -> (token g+8, same); column of (word j,
    // position c) = 8j + c
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        red[warp][g][16 * t + c] = acc[c][0];
        red[warp][g][16 * t + 8 + c] = acc[c][1];
        red[warp][g + 8][16 * t + c] = acc[c][2];
        red[warp][g + 8][16 * t + 8 + c] = acc[c][3];
    }
    __syncthreads();
    const size_t plane_elems = (size_t)p.m * (size_t)p.ldp;
    float* plane = p.planes + (size_t)slab * plane_elems;
    for (int e = threadIdx.x; e < 16 * 64; e += GB_WARPS * 32) {
        const int token = e >> 6, col = e & 63;
        if (token >= p.m) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < GB_WARPS; ++w) v += red[w][token][col];
        const int kcol = kb * 64 + col;
        if (pr.ext_a != nullptr && slab == pr.first) {   // u . lora_a, once per member
            float s = 0.f;
#pragma unroll
            for (int r = 0; r < 16; ++r)
                s = fmaf(__half2float(__ldg(pr.ext_a + (long long)token * 16 + r)),
                         __half2float(__ldg(pr.ext_b + (long long)r * p.k_w + kcol)), s);
            v += s;
        }
        __stcg(plane + (size_t)token * p.ldp + kcol, v);
    }
    if (p.ticket_base < 0) return;   // a reduction kernel follows
    // Last arriver of this k-block: every thread makes its plane writes visible device-wide, then
    // one thread takes the ticket.
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* ticket = g_gemv_tickets + p.ticket_base + kb;
        const unsigned old = atomicAdd(ticket, 1u);
        is_last = old == (unsigned)(p.n_slabs - 1) ? 1 : 0;
        if (is_last) *ticket = 0u;   // (nobody else touches it any more in this launch)
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    __half* out = p.prob[0].out;
    for (int e = threadIdx.x; e < 16 * 64; e += GB_WARPS * 32) {
        const int token = e >> 6, col = e & 63;
        if (token >= p.m) continue;
        const size_t off = (size_t)token * p.ldp + (size_t)(kb * 64 + col);
        float v = 0.f;
        for (int z = 0; z < p.n_slabs; ++z) v += __ldcg(p.planes + (size_t)z * plane_elems + off);
        out[(long long)token * p.prob[0].ld_out + kb * 64 + col] = __float2half_rn(v);
    }
}

// ------------------------------------------------------------------------------------ host side

static bool gemv_common_ok(const GemmArgs& a) {
    return a.scales16 != nullptr && a.n_w % GV_ROWS == 0 && a.k_w % 64 == 0 &&
           (reinterpret_cast<uintptr_t>(a.codes) & 15) == 0;
}

bool gemv_eligible(const GemmArgs& a) {
    // Measured against the tensor-core kernel: ahead up to 32 rows (four launches of a layer of the
    // 1536-wide network 36 against 52 us, of the 3584-wide one 96 against 126); up to 64 rows, as two
    // blocks of 32 tokens side by side, only where one block leaves SMs idle (64 rows, q/k/v of the
    // 1536-wide one 6.3 against 15.6; its gate / up 26 against 24).
    const bool small_enough = a.m <= 32 || (a.m <= 64 && a.n_w * a.k_w <= (1ll << 22));
    return !a.trans_w && a.m >= 1 && small_enough && gemv_common_ok(a) && a.n_w * (a.k_w / 2) < (1ll << 32) && a.ld_act % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(a.act) & 15) == 0;
}

bool gemv_bwd_eligible(const GemmArgs& a) {
    return a.trans_w && a.m >= 1 && a.m <= 16 && gemv_common_ok(a) && a.ld_act % 2 == 0 &&
           (reinterpret_cast<uintptr_t>(a.act) & 3) == 0 &&
           (reinterpret_cast<uintptr_t>(a.scales16) & 3) == 0;
}

static void fill_problem(GemvProblem& q, const GemmArgs& a) {
    q.codes = a.codes; q.scales16 = a.scales16; q.code16 = a.code16; q.bias = a.bias;
    q.ext_a = a.ext_a; q.ext_b = a.ext_b; q.act = a.act; q.out = a.out;
    q.ld_out = a.ld_out; q.ld_act = a.ld_act; q.n_w = (int)a.n_w; q.first = 0;
}

template <int NT, int MT, bool SWIGLU, bool XS, int WL>
static cudaError_t launch_gemv_x(const GemvParams& p, dim3 grid, size_t smem, cudaStream_t stream) {
    // the opt-in to more than 48 KB is a property of the kernel on a device: set once on each
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
        int reserved = 0;   // the pair table's fixed address has to lie behind it
        e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
        if (e != cudaSuccess) return e;
        if (reserved > (int)PAIR_AT) return cudaErrorInvalidConfiguration;
        e = cudaFuncSetAttribute(nf4_gemv_kernel<NT, MT, SWIGLU, XS, WL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 XS ? GV_MAX_SMEM : GemvShape<NT, MT, SWIGLU, WL>::FIXED_BYTES + (int)PAIR_AT);
        if (e != cudaSuccess) return e;
        done.fetch_or(bit, std::memory_order_release);
    }
    return launch_pdl(nf4_gemv_kernel<NT, MT, SWIGLU, XS, WL>, grid, dim3(32 << WL), smem, stream, p);
}

template <int NT, int MT, bool SWIGLU, int WL>
static cudaError_t launch_gemv_t(GemvParams p, int sms, cudaStream_t stream) {
    // Warps per tile: the fewest rounds of the busiest SM, then the fewest CTAs (the other half of
    // an SM's registers is where the next kernel of the stream sets itself up).
    const int nkb = p.k_w / 64, members = SWIGLU ? 1 : p.n_prob;
    auto sets_of = [&](int i, int sl) { return (((long long)p.prob[i].tiles << sl) + (1 << WL) - 1) / (1 << WL); };
    long long best = -1;
    for (int sl = 0; sl <= WL && (sl == 0 || (1 << sl) <= nkb); ++sl) {
        long long sets = 0;
        for (int i = 0; i < members; ++i) sets += sets_of(i, sl);
        const long long cost = (sets + sms - 1) / sms * ((1 << WL) >> sl);
        if (best < 0 || cost < best) {
            best = cost;
            p.split_log = sl;
            p.n_sets = (int)sets;
        }
    }
    int first = 0;
    for (int i = 0; i < members; ++i) {
        p.prob[i].first = first;
        first += (int)sets_of(i, p.split_log);
    }
    const dim3 grid((unsigned)(p.n_sets < 2 * sms ? p.n_sets : 2 * sms),
                    (unsigned)((p.m + NT * 8 - 1) / (NT * 8)));
    const size_t fixed = GemvShape<NT, MT, SWIGLU, WL>::FIXED_BYTES + PAIR_AT;
    if constexpr (NT == 1) {
        // Activations are staged (padded rows: 16-byte reads of eight rows meet no bank conflict) where
        // that is one row or several tiles of the CTA read them, and read through L1 otherwise. us:
        // one row, down_proj of 8960 columns 6.2 against 6.7; four rows, gate / up of the 3584-wide
        // network (8 tiles) 25.0 against 28.6, its q/k/v (2 tiles) 6.6 against 6.4. With more than
        // eight rows there was no gain.
        const size_t x_bytes = (size_t)p.m * (p.k_w + 8) * 2;
        if ((p.m == 1 || p.split_log <= WL - 2) && fixed + x_bytes <= (size_t)GV_MAX_SMEM)
            return launch_gemv_x<NT, MT, SWIGLU, true, WL>(p, grid, fixed + x_bytes, stream);
    }
    return launch_gemv_x<NT, MT, SWIGLU, false, WL>(p, grid, fixed, stream);
}

// CTAs of 2^WL warps; token blocks of 8, as many as there are up to four.
template <int MT, bool SWIGLU, int WL>
static cudaError_t launch_gemv_m(const GemvParams& p, int sms, cudaStream_t stream) {
    constexpr bool PAIRED = MT == 2;   // (tiles of 32 rows: not all token blocks, see launch_gemv_group)
    if constexpr (!PAIRED || SWIGLU)
        if (p.m <= 8) return launch_gemv_t<1, MT, SWIGLU, WL>(p, sms, stream);
    if (p.m <= 16) return launch_gemv_t<2, MT, SWIGLU, WL>(p, sms, stream);
    if constexpr (!PAIRED)
        if (p.m <= 24) return launch_gemv_t<3, MT, SWIGLU, WL>(p, sms, stream);
    if (p.m <= 32) return launch_gemv_t<4, MT, SWIGLU, WL>(p, sms, stream);
    // two blocks of tokens side by side: CTAs of 8 warps, two of which fit an SM
    if constexpr (!PAIRED && WL == 3)
        return p.m <= 48 ? launch_gemv_t<3, MT, SWIGLU, WL>(p, sms, stream)
                         : launch_gemv_t<4, MT, SWIGLU, WL>(p, sms, stream);
    return cudaErrorInvalidValue;
}

// Fills the parameters of a forward launch; `rows` = weight rows of a tile that come from one
// member.
static GemvParams gemv_forward_params(const GemmGroupArgs& ga, int rows) {
    const GemmArgs& a = ga.item[0];
    GemvParams p = {};
    p.n_prob = ga.count;
    p.act = a.act; p.ld_act = a.ld_act;
    p.m = (int)a.m; p.k_w = (int)a.k_w;
    for (int i = 0; i < ga.count; ++i) {
        fill_problem(p.prob[i], ga.item[i]);
        p.prob[i].tiles = (int)(ga.item[i].n_w / rows);
    }
    for (int i = ga.count; i < GV_MAXP; ++i) p.prob[i] = p.prob[0];
    return p;
}

cudaError_t launch_gemv_group(const GemmGroupArgs& ga, cudaStream_t stream) {
    const GemmArgs& a = ga.item[0];
    const int sms = a.sm_count > 0 ? a.sm_count : 148;
    long long rows = 0;
    bool wide = a.m > 8 && (a.m <= 16 || a.m > 24 || a.k_w >= 8192) && a.m <= 32;
    for (int i = 0; i < ga.count; ++i) {
        wide = wide && ga.item[i].n_w % 32 == 0;
        rows += ga.item[i].n_w;
    }
    const bool small = rows * a.k_w <= (1ll << 22), one_tile = rows <= (long long)GV_ROWS * sms;
    // Tiles of 32 rows read the activations half as often: they pay with more than 8 tokens where they
    // still occupy most SMs and a warp's slice of K is long (us, 32 against 16 rows: at 16 tokens 3584 x 18944
    // 21.9 against 27.0, 8960 x 1536 6.4 against 7.0, 1536 x 8960 12.2 against 8.6; at 32 tokens 4096 x 4096 10.9
    // against 11.6, 4096 x 1024 6.0 against 5.3). 17 to 24 tokens leave a fourth token block of them idle: 3584 x
    // 3584 at 24 tokens 10.0 against 8.9 with three, 3584 x 18944 30.5 against 31.8.
    if (wide && !small && rows / 32 * 4 >= 3ll * sms)
        return launch_gemv_m<2, false, 4>(gemv_forward_params(ga, 2 * GV_ROWS), sms, stream);
    const GemvParams p = gemv_forward_params(ga, GV_ROWS);
    // Small weights: a CTA's 32 KB pair table and the fold over its warps weigh more than the contraction, so
    // smaller CTAs, spread over more SMs (us, CTAs of 16 / 8 / 4 warps): 256 x 256, 8 tokens 2.9 / 1.9 / 1.7, 16
    // tokens 3.0 / 2.3 / 2.0; 512 x 512, 8 tokens 2.4 / 2.0 / 2.1, 32 tokens 3.9 / 2.9 / 3.0; 1024 x 1024, 8 tokens
    // 2.5 / 2.4 / 2.6, 32 tokens 3.8 / 3.6 / 3.7. Larger ones stay with 16 warps: by itself 1536 x 1536 at 16 tokens
    // takes 3.7 / 3.3 / 3.7, but two CTAs per SM leave the next kernel of a stream no room to set itself up, and a
    // decode step of the 1536-wide network got 2 % slower (4 % at 32 tokens).
    // More than 32 tokens, in two blocks: 1536 x 1536 at 40 tokens 5.4 with three token blocks each, 6.1 with four.
    if (a.m <= 32 && one_tile && p.k_w <= 4 * 64) return launch_gemv_m<1, false, 2>(p, sms, stream);
    if (a.m > 32 || (one_tile && p.k_w <= 16 * 64)) return launch_gemv_m<1, false, 3>(p, sms, stream);
    return launch_gemv_m<1, false, 4>(p, sms, stream);
}

bool gemv_swiglu_eligible(const GemmGroupArgs& ga) {
    if (ga.count != 2) return false;
    const GemmArgs &g = ga.item[0], &u = ga.item[1];
    return g.m <= 32 && g.n_w == u.n_w && g.k_w == u.k_w && g.bias == nullptr && u.bias == nullptr &&
           g.ext_a == nullptr && u.ext_a == nullptr && (g.out == nullptr) == (u.out == nullptr) &&
           gemv_eligible(g) && gemv_eligible(u);
}

cudaError_t launch_gemv_swiglu(const GemmGroupArgs& ga, __half* hidden, cudaStream_t stream) {
    const int sms = ga.item[0].sm_count > 0 ? ga.item[0].sm_count : 148;
    GemvParams p = gemv_forward_params(ga, GV_ROWS);
    p.hidden = hidden;
    return launch_gemv_m<2, true, 4>(p, sms, stream);
}

// Row slabs of the streaming backward: enough CTAs (k-blocks x slabs) for about three per SM, slabs
// of whole 16-row steps for every warp.
constexpr int GB_WARPS_PER_CTA = 8;

StreamBwdPlan plan_stream_bwd(long long m, const long long* n_w, int count, long long k_w, int sm_count) {
    StreamBwdPlan pl = {};
    const long long nkb = k_w / 64;
    long long total_rows = 0;
    for (int i = 0; i < count; ++i) total_rows += n_w[i];
    const int sms = sm_count > 0 ? sm_count : 148;
    long long want = (3ll * sms + nkb - 1) / nkb;              // slabs wanted over the group
    if (want < 1) want = 1;
    const long long unit = 16ll * GB_WARPS_PER_CTA;             // one step per warp at least
    long long rows = (total_rows + want - 1) / want;
    rows = (rows + unit - 1) / unit * unit;
    pl.rows_per_slab = (int)rows;
    int slabs = 0;
    for (int i = 0; i < count; ++i) {
        pl.first[i] = slabs;
        slabs += (int)((n_w[i] + rows - 1) / rows);
    }
    pl.slabs = slabs;
    pl.ldp = (k_w + 3) / 4 * 4;
    pl.ws_bytes = (size_t)slabs * (size_t)m * (size_t)pl.ldp * sizeof(float);
    return pl;
}

cudaError_t launch_gemv_bwd_group(const GemmGroupArgs& ga, cudaStream_t stream, const char** why) {
    const GemmArgs& a = ga.item[0];
    long long n_w[GEMM_MAX_GROUP];
    for (int i = 0; i < ga.count; ++i) n_w[i] = ga.item[i].n_w;
    const StreamBwdPlan pl = plan_stream_bwd(a.m, n_w, ga.count, a.k_w, a.sm_count);
    if (a.workspace == nullptr || a.workspace_bytes < pl.ws_bytes) {
        *why = "small-M backward: workspace too small";
        return cudaErrorInvalidValue;
    }
    GemvParams p = {};
    p.n_prob = ga.count;
    p.m = (int)a.m; p.k_w = (int)a.k_w;
    p.planes = static_cast<float*>(a.workspace);
    p.ldp = pl.ldp;
    p.rows_per_slab = pl.rows_per_slab;
    p.n_slabs = pl.slabs;
    const long long nkb = a.k_w / 64;
    static std::atomic<unsigned> cursor{0};
    p.ticket_base = nkb <= TICKET_SPAN
        ? (int)((cursor.fetch_add(1u, std::memory_order_relaxed) % TICKET_LAUNCHES) * TICKET_SPAN)
        : -1;
    for (int i = 0; i < ga.count; ++i) {
        fill_problem(p.prob[i], ga.item[i]);
        p.prob[i].first = pl.first[i];
    }
    for (int i = ga.count; i < GV_MAXP; ++i) p.prob[i] = p.prob[0];
    cudaError_t e = launch_pdl(nf4_gemv_bwd_kernel<GB_WARPS_PER_CTA>,
                               dim3((unsigned)(a.k_w / 64), (unsigned)pl.slabs), dim3(GB_WARPS_PER_CTA * 32),
                               0, stream, p);
    if (e != cudaSuccess) { *why = "small-M backward kernel launch"; return e; }
    if (p.ticket_base >= 0) return e;
    e = launch_splitk_reduce(p.planes, a.m, a.k_w, pl.ldp, pl.slabs, nullptr, a.out, a.ld_out,
                             a.sm_count, stream);
    if (e != cudaSuccess) *why = "small-M backward reduce launch";
    return e;
}

}  // namespace nf4
