// The quantiser objects by themselves (quantizer.py:93-306, kv_cache.py:45-116): plain rows in, the reference's flat
// planes out, and back.  Nothing goes through a block pool: a call is one kernel that reads its input once and writes
// its output once.
//
//   keys    rows -> codes, sign bits, norms (tensor cores, head_dim 128), planes -> rows
//   values  rows -> codes, scales, zero points, planes -> rows
//   scores  query against key planes
//
// The products run on mma.sync with fp16 limbs: a number scaled away from fp16's subnormals is the sum of two fp16 numbers
// to 2^-22, and three products of limbs, accumulated in fp32, give the fp32 product to about the rounding of its own sum
// (three bf16 limbs would need six).  A pair of warps owns 16 rows from load to packed output with its A operand in registers;
// the constant operands (two limbs of 128 x 128 each) stay in shared memory.  At these sizes - a tile per CTA - a kernel is
// its chain of phases, so four warps a scheduler cover one another, the loops stay small enough to be fetched, and every
// kernel starts under the launch ahead of it: its constants arrive while it waits.
//
// Measured (B200, 16000 rows of 128, fp32, 3-bit keys, 2-bit values, 4 queries, calls back to back; in brackets with a warp per
// 16 rows, eight query slots whatever was asked for, a thread per group of values and plain launches): quantise 20.2 us
// (31.7), dequantise 13.2 (14.6), scores 8.2 (12.0), values 6.9 (10.4) and 4.5 (6.2), everything in turn 50.1 (76.0); 480 rows
// 41.5 (62.9).
#include "tq_decode_common.cuh"

using namespace tqdec;

namespace {

// ------------------------------------------------------------------ values

// What every kernel of this file does first: whatever it reads or writes of the caller's belongs to the launch ahead until the
// wait; only then may the launch behind it begin, so that what it does before its own wait comes after everything ahead of here.
__device__ __forceinline__ void wait_for_launch_ahead() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Four lanes per group of 32 channels, eight consecutive channels each.  Arithmetic of kv_cache.py:64-90 with the rounding of
// the tensor's dtype after every operation; scale and zero point pass through fp16, the form they are stored in.
template <int DT, int VAL_BITS>
__global__ void __launch_bounds__(256) tq_rows_quantize_values_kernel(const void* v, int64_t n_groups, int groups_per_row, int64_t stride_row,
                                                                      uint8_t* data, void* scales, void* zeros) {
    using E = TqElem<DT>;
    wait_for_launch_ahead();
    const int64_t unit = (int64_t)blockIdx.x * 256 + threadIdx.x, i = unit >> 2;
    const int part = (int)(unit & 3);
    const bool live = i < n_groups;   // the four lanes of a group alike
    const int64_t row = i / groups_per_row;
    const int64_t at = row * stride_row + (i - row * groups_per_row) * 32 + part * 8;
    float x[8] = {};
    if (live) {
        if (DT == TQ_F32) {
            const float4* src = reinterpret_cast<const float4*>((const float*)v + at);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 q = src[j];
                x[4 * j] = q.x;
                x[4 * j + 1] = q.y;
                x[4 * j + 2] = q.z;
                x[4 * j + 3] = q.w;
            }
        } else {
            const uint4 q = *reinterpret_cast<const uint4*>((const uint16_t*)v + at);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (DT == TQ_BF16) {
                    x[2 * k] = __uint_as_float(w[k] << 16);
                    x[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
                } else {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
                    x[2 * k] = f.x;
                    x[2 * k + 1] = f.y;
                }
            }
        }
    }
    float vmin = x[0], vmax = x[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        vmin = fminf(vmin, x[j]);
        vmax = fmaxf(vmax, x[j]);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
        vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if (!live) return;
    constexpr float LEVELS = (float)((1 << VAL_BITS) - 1);
    float scale = E::round(__fdiv_rn(E::round(vmax - vmin), LEVELS));
    scale = fmaxf(scale, E::round(1e-10f));
    uint32_t out = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float r = rintf(E::round(__fdiv_rn(E::round(x[j] - vmin), scale)));
        out |= (uint32_t)fminf(fmaxf(r, 0.f), LEVELS) << (VAL_BITS * j);
    }
    if (VAL_BITS == 2) reinterpret_cast<uint16_t*>(data)[unit] = (uint16_t)out;
    else reinterpret_cast<uint32_t*>(data)[unit] = out;
    if (part == 0) {
        E::store(scales, i, __half2float(__float2half_rn(scale)));
        E::store(zeros, i, __half2float(__float2half_rn(vmin)));
    }
}

// code * scale + zero in fp32 (kv_cache.py:101-116); one thread per four channels
template <int VAL_BITS>
__global__ void __launch_bounds__(256) tq_rows_dequantize_values_kernel(const uint8_t* data, const void* scales,
                                                                        const void* zeros, int sdt, int64_t n_quads, float* out) {
    wait_for_launch_ahead();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n_quads) return;
    const uint32_t w = VAL_BITS == 2 ? data[i] : reinterpret_cast<const uint16_t*>(data)[i];
    const float sc = __half2float(__float2half_rn(tq_load_any(scales, i >> 3, sdt)));
    const float zr = __half2float(__float2half_rn(tq_load_any(zeros, i >> 3, sdt)));
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = (float)((w >> (VAL_BITS * k)) & ((1u << VAL_BITS) - 1u)) * sc + zr;
    reinterpret_cast<float4*>(out)[i] = make_float4(v[0], v[1], v[2], v[3]);
}

// ------------------------------------------------------------------ keys, head_dim 128

constexpr int RD = 128, R_GROUPS = 8, R_ROWS = 16 * R_GROUPS;   // row groups of a tile, 16 rows each
constexpr int R_THREADS = 2 * R_GROUPS * 32;       // a pair of warps per row group, half of the columns each
constexpr int R_MAT = RD * RD * 2;                 // one limb of a constant operand in shared memory
constexpr int KSTEPS = RD / 16;
constexpr int R_XCHG = R_GROUPS * KSTEPS * 2 * 32 * 16;   // A fragments that the warps of a pair hand each other

// the two warps of a row group
__device__ __forceinline__ void pair_sync(int group) { asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory"); }

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t pack_h(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// a pair of fp32 numbers as LIMBS packed fp16 pairs
template <int LIMBS>
__device__ __forceinline__ void split(float x, float y, uint32_t* l, int step) {
#pragma unroll
    for (int i = 0; i < LIMBS; ++i) {
        const __half2 v = __floats2half2_rn(x, y);
        l[i * step] = *reinterpret_cast<const uint32_t*>(&v);
        const float2 f = __half22float2(v);
        x -= f.x;
        y -= f.y;
    }
}

// (128 x 128) fp16, row-major in global memory -> shared memory, 16-byte chunks of a row swizzled by row % 8
__device__ __forceinline__ void load_operand(uint8_t* dst, const void* src, int tid, int nt) {
    for (int i = tid; i < RD * RD / 8; i += nt) {
        const int row = i >> 4, ch = i & 15;
        const uint32_t d = tq_smem_u32(dst + row * 256 + ((ch ^ (row & 7)) << 4));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(static_cast<const uint4*>(src) + i) : "memory");
    }
}
// B fragments of columns n0..n0+15, k-step ks: {n8 block 0: b0, b1, block 1: b0, b1}.
// Rows of the stored matrix are n (TRANS = false) or k (TRANS = true).
template <bool TRANS>
__device__ __forceinline__ void b_frag(uint32_t mat, int n0, int ks, int lane, uint32_t (&r)[4]) {
    // lane l addresses row l % 8 of block l / 8; blocks in the order (n8 0, k8 0), (n8 0, k8 1), (n8 1, k8 0), (n8 1, k8 1)
    const int blk = lane >> 3, i = lane & 7;
    const int row = TRANS ? ks * 16 + 8 * (blk & 1) + i : n0 + 8 * (blk >> 1) + i;
    const int ch = TRANS ? (n0 >> 3) + (blk >> 1) : 2 * ks + (blk & 1);
    ldsm4<TRANS>(mat + row * 256 + ((ch ^ (row & 7)) << 4), r);
}
// The same onto zero
__device__ __forceinline__ void mma_f16_z(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// acc[2][4] += A (LA limbs in registers) * B (two limbs), without lo * lo.
// The pipe drops what does not fit its accumulator instead of rounding, so the large products (hi * hi) must not pass through
// it together with the small ones, which have accumulators of their own.  STEPS: not with each other either - every k-step's
// sum is added up in fp32.  Error of a product against 64 bits, unit vectors: one chain for all 4.6e-7 of the result (5.6e-7
// with 3-bit codes), two chains 1.9e-7 (2.5e-7), STEPS 0.9e-7 (1.1e-7); the fp32 fused multiply-adds of the kernels on records
// 2.0e-7.  Of 384 million fp32 coordinates 319, 129 and 58 sign bits came out wrong, 259 in the fp32 store.  With a warp per
// 16 rows a pass over 16000 (quantise, score, dequantise) took 73 us with one chain, 67 with two for quantising and STEPS for
// dequantising, 75 with STEPS everywhere.
template <int LA, bool TRANS, bool STEPS>
__device__ __forceinline__ void product(float (&acc)[2][4], const uint32_t (*a)[KSTEPS][4], uint32_t mats, int n0, int lane) {
    float low[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
        uint32_t b[4], bl[4];
        b_frag<TRANS>(mats, n0, ks, lane, b);
        b_frag<TRANS>(mats + R_MAT, n0, ks, lane, bl);
#pragma unroll
        for (int n8 = 0; n8 < 2; ++n8) {
            if (STEPS) {
                float t[4];
                mma_f16_z(t, a[0][ks], b[2 * n8], b[2 * n8 + 1]);
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[n8][c] += t[c];
            } else {
                mma_f16(acc[n8], a[0][ks], b[2 * n8], b[2 * n8 + 1]);
            }
            if (LA == 2) mma_f16(low[n8], a[LA - 1][ks], b[2 * n8], b[2 * n8 + 1]);
            mma_f16(low[n8], a[0][ks], bl[2 * n8], bl[2 * n8 + 1]);
        }
    }
#pragma unroll
    for (int n8 = 0; n8 < 2; ++n8)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[n8][c] += low[n8][c];
}

constexpr float R_SCALE = 64.f;   // of every A operand and of Pi: unit vectors, centroids and residuals are far below 1

struct RowsParams {
    const void* x;
    int64_t n, stride_row;
    const void *pi[2], *other[2];   // limbs of 64 Pi and of M = S Pi^T (quantise) or S (dequantise), (128, 128) row-major
    const float* pi_t;
    TqCodebook cb;
    uint8_t* codes;
    uint8_t* signs;
    void* norms;
    void* rnorms;
    int norm_dt, rnorm_dt;
    float qjl_scale;
    int with_qjl;
    float* out;
};

template <int DT>
__device__ __forceinline__ void load2(const void* p, int64_t i, float& a, float& b) {
    if (DT == TQ_F32) {
        const float2 v = *reinterpret_cast<const float2*>((const float*)p + i);
        a = v.x;
        b = v.y;
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>((const __half*)p + i));
        a = f.x;
        b = f.y;
    }
}
template <int DT>
__device__ __forceinline__ void load4(const void* p, int64_t i, float* x) {
    load2<DT>(p, i, x[0], x[1]);
    load2<DT>(p, i + 2, x[2], x[3]);
}

// The limb products and the fp32 store kernel's chain of fused multiply-adds agree to a few 1e-7 (|u| = 1, rows of Pi have
// norm 1).  A coordinate that lies closer than this to a decision boundary - some 20 in a million - is computed again as
// that chain, so that the codes are the fp32 kernel's on both sides of a tie.  Where the chain decides differently, in one row of some
// 30 000, its number takes the product's place before anything follows from it (as a whole row by that chain, behind the rest of
// its tile, such a row made a call of 16000 rows take 28.9 us; now 20.2 with or without one).
constexpr float NEAR = 1e-6f;
// Off the usual path, from a cold instruction cache, where a line of eight instructions costs more than the arithmetic in
// it: loops stay rolled.
// One coordinate by the whole warp: lane l holds the terms l, 32 + l, ...; every lane returns the sum.
template <int DT>
__device__ __noinline__ float serial_product(const void* x, int64_t at, float den, const float* pi_t_col, int lane) {
    using E = TqElem<DT>;
    float u[RD / 32], w[RD / 32], y = 0.f;
#pragma unroll
    for (int i = 0; i < RD / 32; ++i) w[i] = __ldg(pi_t_col + (32 * i + lane) * RD);
#pragma unroll
    for (int i = 0; i < RD / 32; ++i) u[i] = E::round(__fdiv_rn(E::load(x, at + 32 * i + lane), den));
#pragma unroll
    for (int i = 0; i < RD / 32; ++i)
#pragma unroll 4
        for (int l = 0; l < 32; ++l) y = fmaf(__shfl_sync(0xffffffffu, u[i], l), __shfl_sync(0xffffffffu, w[i], l), y);
    return y;
}

// quantizer.py:129-149,231-257 for 16 rows per pair of warps: norm, x / |x| (rounded to the dtype like torch), Y = u Pi^T,
// bucket search, residual in rotated space r' = (Y - c) + E, E = (x / |x| - u) Pi^T, sign bits of r' M^T with M = S Pi^T.
// A warp works out half of the k-steps of its rows' A operands and half of the columns of both products; what the other needs
// goes through shared memory as whole fragments.  Four warps a scheduler instead of two cover one another's chains, and the
// loops over columns stay rolled: unrolled they were 100 KB of instructions that a call of one tile per CTA reads once.
template <int DT, int MSE_BITS>
__global__ void __launch_bounds__(R_THREADS, 1) tq_rows_quantize_keys_kernel(const __grid_constant__ RowsParams p, int vec /* rows of x are 16-byte aligned */) {
    using E = TqElem<DT>;
    constexpr int LU = DT == TQ_F32 ? 2 : 1;   // limbs that hold u; else the second place holds e = x / |x| - u
    constexpr int NB = (1 << MSE_BITS) - 1;
    constexpr int HALF = KSTEPS / 2;           // k-steps, and blocks of 16 columns, of one warp of the pair
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float s_ss[R_ROWS], s_n2[2][R_ROWS];
    const int tid = threadIdx.x, group = (tid >> 5) & (R_GROUPS - 1), mine = tid >> 8, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) load_operand(smem + i * R_MAT, p.pi[i], tid, R_THREADS);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 1
    for (int i = 0; i < 2; ++i) load_operand(smem + (2 + i) * R_MAT, p.other[i], tid, R_THREADS);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t sp = tq_smem_u32(smem), sm = sp + 2 * R_MAT;
    uint4* xchg = reinterpret_cast<uint4*>(smem + 4 * R_MAT) + group * (KSTEPS * 2 * 32) + lane;   // [k-step][limb][lane]
    constexpr int ES = DT == TQ_F32 ? 4 : 2, RB = RD * ES;
    static_assert(16 * RB <= KSTEPS * 2 * 32 * 16, "the rows of a pair fit the place of its fragments");
    // chunk c of row r there: eight rows' same chunk (or four rows' same two, of fp32) in different banks
    auto at_row = [&](int r, int c) -> uint8_t* {
        return smem + 4 * R_MAT + group * (KSTEPS * 2 * 32 * 16) + r * RB + ((c ^ (DT == TQ_F32 ? (r & 3) << 1 : r & 7)) << 4);
    };
    wait_for_launch_ahead();
    bool first = true;
#pragma unroll 1
    for (int64_t tile = blockIdx.x; tile * R_ROWS < p.n; tile += gridDim.x) {
        const int64_t base_row = tile * R_ROWS + group * 16, r0 = base_row + gid, r1 = r0 + 8;
        {   // the pair's rows, whole lines at a time, into the place of the fragments: chunks of 16 bytes, swizzled by row (each lane
            // fetching its own pairs of numbers from global memory, twice over with the norms, added 0.6 us to 28.9, of fp16 1.4 to 31.8)
            constexpr int CHUNKS = 16 * RB / 16 / 64;   // of one thread
            uint4 v[CHUNKS];
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                const int c = i * 64 + mine * 32 + lane;
                const int64_t row = base_row + c / (RB / 16);
                v[i] = make_uint4(0u, 0u, 0u, 0u);
                if (row < p.n) {
                    const char* src = static_cast<const char*>(p.x) + row * p.stride_row * ES + c % (RB / 16) * 16;
                    if (vec) {
                        v[i] = *reinterpret_cast<const uint4*>(src);
                    } else {
                        const uint2 lo = reinterpret_cast<const uint2*>(src)[0], hi = reinterpret_cast<const uint2*>(src)[1];
                        v[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) {
                const int c = i * 64 + mine * 32 + lane;
                *reinterpret_cast<uint4*>(at_row(c / (RB / 16), c % (RB / 16))) = v[i];
            }
        }
        pair_sync(group);
        float x[HALF][2][2][2];   // this warp's k-steps: [row][half][element]
#pragma unroll
        for (int ks = 0; ks < HALF; ++ks)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const int byte = ((mine * HALF + ks) * 16 + hf * 8 + 2 * tig) * ES;
                    load2<DT>(at_row(gid + 8 * r, byte >> 4) + (byte & 15), 0, x[ks][r][hf][0], x[ks][r][hf][1]);
                }
        {   // norms, in the fp32 store kernel's order: eight sums of 16 squares, added up in order.  Lane = (row % 4, sum), two rows a lane.
            const int ch = lane & 7;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row_l = 8 * mine + 4 * i + (lane >> 3);
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; j += 16 / ES)
#pragma unroll
                    for (int k = 0; k < 16 / ES; k += 4) load4<DT>(at_row(row_l, (ch * 16 + j) * ES >> 4), k, v + j + k);
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < 16; ++j) s = fmaf(v[j], v[j], s);
                float tot = 0.f;
#pragma unroll
                for (int c = 0; c < 8; ++c) tot += __shfl_sync(0xffffffffu, s, (lane & 24) + c);
                if (ch == 0) s_ss[group * 16 + row_l] = tot;
            }
        }
        pair_sync(group);
        float nd[2], den[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            nd[r] = E::round(__fsqrt_rn(s_ss[group * 16 + gid + 8 * r]));
            den[r] = E::round(nd[r] + 1e-10f);
        }
#pragma unroll
        for (int ks = 0; ks < HALF; ++ks) {
            uint32_t f[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const float q0 = __fdiv_rn(x[ks][r][hf][0], den[r]), q1 = __fdiv_rn(x[ks][r][hf][1], den[r]);
                    const float u0 = E::round(q0), u1 = E::round(q1);
                    split<LU>(u0 * R_SCALE, u1 * R_SCALE, &f[0][hf * 2 + r], 4);
                    if (DT != TQ_F32) f[1][hf * 2 + r] = pack_h((q0 - u0) * R_SCALE, (q1 - u1) * R_SCALE);
                }
#pragma unroll
            for (int l = 0; l < 2; ++l) xchg[((mine * HALF + ks) * 2 + l) * 32] = make_uint4(f[l][0], f[l][1], f[l][2], f[l][3]);
        }
        uint32_t a[2][KSTEPS][4];
        auto take = [&]() {   // all fragments of the pair's rows
            pair_sync(group);
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks)
#pragma unroll
                for (int l = 0; l < 2; ++l) {
                    const uint4 v = xchg[(ks * 2 + l) * 32];
                    a[l][ks][0] = v.x; a[l][ks][1] = v.y; a[l][ks][2] = v.z; a[l][ks][3] = v.w;
                }
            pair_sync(group);
        };
        take();
        if (first) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
        }
        // ---- codes, r' as limbs in the A layout of the second product ----
        uint32_t cw[2][MSE_BITS == 2 ? 1 : 2] = {};   // this warp's code words of the two rows, word j in lane j % 4
        float rn2[2] = {0.f, 0.f};
#pragma unroll 1
        for (int j = 0; j < HALF; ++j) {
            const int nb = mine * HALF + j;
            float acc[2][4] = {};
            product<LU, false, false>(acc, a, sp, nb * 16, lane);
            float er[2][4] = {};
            if (DT != TQ_F32) {
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {   // |q - u| <= 2^-12: Pi's first limb is enough
                    uint32_t b[4];
                    b_frag<false>(sp, nb * 16, ks, lane, b);
                    mma_f16(er[0], a[1][ks], b[0], b[1]);
                    mma_f16(er[1], a[1][ks], b[2], b[3]);
                }
            }
            uint32_t near = 0;   // of the lane's eight: those next to a boundary, whose side the fp32 store kernel's chain decides
#pragma unroll
            for (int n8 = 0; n8 < 2; ++n8)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float gap = 1.f;
#pragma unroll
                    for (int i = 0; i < NB; ++i) gap = fminf(gap, fabsf(acc[n8][c] * (1.f / (R_SCALE * R_SCALE)) - p.cb.boundaries[i]));
                    if (gap < NEAR) near |= 1u << (n8 * 4 + c);
                }
            if (r0 >= p.n || nd[0] == 0.f) near &= 0xccu;
            if (r1 >= p.n || nd[1] == 0.f) near &= 0x33u;
            if (__any_sync(0xffffffffu, near != 0)) {
#pragma unroll 1
                for (uint32_t who; (who = __ballot_sync(0xffffffffu, near != 0)) != 0;) {
                    const int from = __ffs(who) - 1;   // this lane's next coordinate, for the whole warp
                    const int bit = __shfl_sync(0xffffffffu, __ffs(near) - 1, from);
                    const int64_t row = base_row + (from >> 2) + (bit & 2 ? 8 : 0);
                    const float y = serial_product<DT>(p.x, row * p.stride_row, __shfl_sync(0xffffffffu, bit & 2 ? den[1] : den[0], from),
                                                       p.pi_t + nb * 16 + (bit >> 2) * 8 + 2 * (from & 3) + (bit & 1), lane);
                    if (lane == from) {
                        near &= near - 1;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {   // where it decides differently, it is what is coded
                            float& had = acc[i >> 2][i & 3];
                            int k = 0;
#pragma unroll
                            for (int b = 0; b < NB; ++b) k += (p.cb.boundaries[b] < y) - (p.cb.boundaries[b] < had * (1.f / (R_SCALE * R_SCALE)));
                            if (i == bit && k != 0) had = y * (R_SCALE * R_SCALE);
                        }
                    }
                }
            }
            uint32_t word[2] = {0u, 0u}, rl[2][4];
#pragma unroll
            for (int n8 = 0; n8 < 2; ++n8) {
                uint32_t code[4];
                float r[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float y = acc[n8][c] * (1.f / (R_SCALE * R_SCALE));
                    uint32_t k = 0;
                    float cv = p.cb.centroids[0];
#pragma unroll
                    for (int i = 0; i < NB; ++i)
                        if (p.cb.boundaries[i] < y) {
                            k = i + 1;
                            cv = p.cb.centroids[i + 1];
                        }
                    if (y != y) {   // searchsorted orders NaN after every number
                        k = NB;
                        cv = p.cb.centroids[NB];
                    }
                    code[c] = k;
                    r[c] = fmaf(er[n8][c], 1.f / (R_SCALE * R_SCALE), y - cv);
                    rn2[c >> 1] = fmaf(r[c], r[c], rn2[c >> 1]);
                }
                split<2>(r[0] * R_SCALE, r[1] * R_SCALE, &rl[0][n8 * 2], 4);       // row r0
                split<2>(r[2] * R_SCALE, r[3] * R_SCALE, &rl[0][n8 * 2 + 1], 4);   // row r1
#pragma unroll
                for (int r2 = 0; r2 < 2; ++r2) {
                    uint32_t w = MSE_BITS == 2 ? (code[2 * r2] | (code[2 * r2 + 1] << 2)) << (4 * tig) : (code[2 * r2] | (code[2 * r2 + 1] << 4)) << (8 * tig);
                    w |= __shfl_xor_sync(0xffffffffu, w, 1);
                    w |= __shfl_xor_sync(0xffffffffu, w, 2);
                    if (MSE_BITS == 2) {   // 16 bits of one word for each n8
                        word[r2] |= w << (16 * n8);
                        if (n8 && tig == j) cw[r2][0] = word[r2];
                    } else if (tig == ((2 * j + n8) & 3)) {
                        if (j < 2) cw[r2][0] = w;
                        else cw[r2][MSE_BITS == 2 ? 0 : 1] = w;
                    }
                }
            }
#pragma unroll
            for (int l = 0; l < 2; ++l) xchg[(nb * 2 + l) * 32] = make_uint4(rl[l][0], rl[l][1], rl[l][2], rl[l][3]);
        }
        if (first) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            first = false;
        }
        // ---- sign bits of r' M^T ----
        take();
        uint32_t sw[2][2] = {};
#pragma unroll 1
        for (int j = 0; j < HALF; ++j) {
            float acc[2][4] = {};
            product<2, false, false>(acc, a, sm, (mine * HALF + j) * 16, lane);
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2) {
                uint32_t w = 0;
#pragma unroll
                for (int n8 = 0; n8 < 2; ++n8)
                    w |= ((acc[n8][2 * r2] > 0.f ? 1u : 0u) | (acc[n8][2 * r2 + 1] > 0.f ? 2u : 0u)) << (2 * tig + 8 * n8);
                w <<= 16 * (j & 1);
                if (j < 2) sw[r2][0] |= w;
                else sw[r2][1] |= w;
            }
        }
        // ---- out ----
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            const int64_t row = r2 ? r1 : r0;
            float n2 = rn2[r2];
            n2 += __shfl_xor_sync(0xffffffffu, n2, 1);
            n2 += __shfl_xor_sync(0xffffffffu, n2, 2);
            if (tig == 0) s_n2[mine][group * 16 + gid + 8 * r2] = n2;
            uint32_t s[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t w = sw[r2][i];
                w |= __shfl_xor_sync(0xffffffffu, w, 1);
                w |= __shfl_xor_sync(0xffffffffu, w, 2);
                s[i] = nd[r2] == 0.f ? 0u : w;   // a zero key has a zero residual
            }
            if (row >= p.n) continue;
            constexpr int CB = MSE_BITS == 2 ? RD / 4 : RD / 2;
            if (tig == 0) *reinterpret_cast<uint2*>(p.signs + row * (RD / 8) + 8 * mine) = make_uint2(s[0], s[1]);
#pragma unroll
            for (int q = 0; q < CB / 32; ++q) *reinterpret_cast<uint32_t*>(p.codes + row * CB + mine * (CB / 2) + 16 * q + 4 * tig) = cw[r2][q];
        }
        pair_sync(group);   // both halves of the residual norms are written
        if (mine == 0 && tig == 3) {
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2) {
                const int64_t row = r2 ? r1 : r0;
                const float n2 = s_n2[0][group * 16 + gid + 8 * r2] + s_n2[1][group * 16 + gid + 8 * r2];
                if (row >= p.n) continue;
                tq_store_any(p.norms, row, __half2float(__float2half_rn(nd[r2])), p.norm_dt);
                tq_store_any(p.rnorms, row, nd[r2] == 0.f ? 0.f : __half2float(__float2half_rn(nd[r2] * __fsqrt_rn(n2))), p.rnorm_dt);
            }
        }
    }
}

// quantizer.py:151-165,259-272 for 16 rows per pair of warps, half of the columns each: (c[idx] Pi) * norm + qjl_scale * rnorm *
// (signs S).  The codes' product first; a thread leaves its sums in shared memory while the signs take over the operand's registers.
template <int MSE_BITS>
__global__ void __launch_bounds__(R_THREADS, 1) tq_rows_dequantize_keys_kernel(const RowsParams p) {
    constexpr int HALF = KSTEPS / 2;   // blocks of 16 columns of one warp
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, group = (tid >> 5) & (R_GROUPS - 1), mine = tid >> 8, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) load_operand(smem + i * R_MAT, p.pi[i], tid, R_THREADS);
    if (p.with_qjl)
#pragma unroll 1
        for (int i = 0; i < 2; ++i) load_operand(smem + (2 + i) * R_MAT, p.other[i], tid, R_THREADS);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t sp = tq_smem_u32(smem), ssg = sp + 2 * R_MAT;
    float4* held = reinterpret_cast<float4*>(smem + 4 * R_MAT) + tid;   // [block of columns][n8][thread]
    float* cen = reinterpret_cast<float*>(smem + 4 * R_MAT + HALF * 2 * R_THREADS * sizeof(float4));
    if (tid < (1 << MSE_BITS)) cen[tid] = p.cb.centroids[tid];
    wait_for_launch_ahead();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    constexpr int CB = MSE_BITS == 2 ? RD / 4 : RD / 2;
#pragma unroll 1
    for (int64_t tile = blockIdx.x; tile * R_ROWS < p.n; tile += gridDim.x) {
        const int64_t rows[2] = {tile * R_ROWS + group * 16 + gid, tile * R_ROWS + group * 16 + gid + 8};
        {
            uint32_t a[2][KSTEPS][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {
                    uint32_t cbits = 0, cbits2 = 0;   // 16 coordinates of the k-step: 2-bit codes in one word, nibbles in two
                    if (rows[r] < p.n) {
                        if (MSE_BITS == 2) {
                            cbits = reinterpret_cast<const uint32_t*>(p.codes + rows[r] * CB)[ks];
                        } else {
                            const uint2 v = reinterpret_cast<const uint2*>(p.codes + rows[r] * CB)[ks];
                            cbits = v.x;
                            cbits2 = v.y;
                        }
                    }
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int k = hf * 8 + 2 * tig;
                        float c0, c1;
                        if (MSE_BITS == 2) {
                            c0 = cen[(cbits >> (2 * k)) & 3u];
                            c1 = cen[(cbits >> (2 * k + 2)) & 3u];
                        } else {
                            const uint32_t w = hf ? cbits2 : cbits;
                            c0 = cen[(w >> (8 * tig)) & 7u];
                            c1 = cen[(w >> (8 * tig + 4)) & 7u];
                        }
                        split<2>(c0 * R_SCALE, c1 * R_SCALE, &a[0][ks][hf * 2 + r], KSTEPS * 4);
                    }
                }
#pragma unroll 1
            for (int j = 0; j < HALF; ++j) {
                float ak[2][4] = {};
                product<2, true, true>(ak, a, sp, (mine * HALF + j) * 16, lane);
#pragma unroll
                for (int n8 = 0; n8 < 2; ++n8) held[(j * 2 + n8) * R_THREADS] = make_float4(ak[n8][0], ak[n8][1], ak[n8][2], ak[n8][3]);
            }
        }
        uint32_t sg[1][KSTEPS][4];   // +1 / -1
        float norm[2], rn[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool live = rows[r] < p.n;
            norm[r] = live ? 1.f / (R_SCALE * R_SCALE) * __half2float(__float2half_rn(tq_load_any(p.norms, rows[r], p.norm_dt))) : 0.f;
            rn[r] = live && p.with_qjl ? p.qjl_scale * __half2float(__float2half_rn(tq_load_any(p.rnorms, rows[r], p.rnorm_dt))) : 0.f;
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
                const uint32_t bits = live && p.with_qjl ? reinterpret_cast<const uint16_t*>(p.signs + rows[r] * (RD / 8))[ks] : 0u;
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const uint32_t b = bits >> (hf * 8 + 2 * tig);
                    sg[0][ks][hf * 2 + r] = ((b & 1u) ? 0x3c00u : 0xbc00u) | ((b & 2u) ? 0x3c000000u : 0xbc000000u);
                }
            }
        }
#pragma unroll 1
        for (int j = 0; j < HALF; ++j) {
            const int n0 = (mine * HALF + j) * 16;
            float as[2][4] = {};
            if (p.with_qjl) product<1, true, true>(as, sg, ssg, n0, lane);
#pragma unroll
            for (int n8 = 0; n8 < 2; ++n8) {
                const float4 ak = held[(j * 2 + n8) * R_THREADS];
                float* out = p.out + n0 + n8 * 8 + 2 * tig;
                if (rows[0] < p.n) *reinterpret_cast<float2*>(out + rows[0] * RD) = make_float2(ak.x * norm[0] + as[n8][0] * rn[0], ak.y * norm[0] + as[n8][1] * rn[0]);
                if (rows[1] < p.n) *reinterpret_cast<float2*>(out + rows[1] * RD) = make_float2(ak.z * norm[1] + as[n8][2] * rn[1], ak.w * norm[1] + as[n8][3] * rn[1]);
            }
        }
    }
}

// The same on CUDA cores for head_dim 256: one CTA of 256 threads (a column each) takes 16 rows.
__global__ void __launch_bounds__(256) tq_rows_dequantize_keys256_kernel(const RowsParams p, const float* __restrict__ pi, const float* __restrict__ s, int mse_bits) {
    constexpr int D = 256;
    __shared__ __align__(16) float yh[D][20], sg[D][20];   // [coordinate][16 rows], padded
    wait_for_launch_ahead();
    const int j = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * 16;
    const int width = mse_bits == 2 ? 2 : 4, vpb = 8 / width, cb = D / vpb;
    for (int t = 0; t < 16; ++t) {
        float c = 0.f, q = 0.f;
        if (row0 + t < p.n) {
            const uint8_t byte = p.codes[(row0 + t) * cb + j / vpb];
            c = p.cb.centroids[(byte >> ((j % vpb) * width)) & ((1 << width) - 1)];
            if (p.with_qjl) q = ((p.signs[(row0 + t) * (D / 8) + (j >> 3)] >> (j & 7)) & 1) ? 1.f : -1.f;
        }
        yh[j][t] = c;
        sg[j][t] = q;
    }
    __syncthreads();
    float am[16], aq[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) am[t] = aq[t] = 0.f;
#pragma unroll 4
    for (int k = 0; k < D; ++k) {
        const float pv = __ldg(pi + (size_t)k * D + j), sv = p.with_qjl ? __ldg(s + (size_t)k * D + j) : 0.f;
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
            const float4 y = *reinterpret_cast<const float4*>(&yh[k][t]), g = *reinterpret_cast<const float4*>(&sg[k][t]);
            am[t] = fmaf(y.x, pv, am[t]);
            am[t + 1] = fmaf(y.y, pv, am[t + 1]);
            am[t + 2] = fmaf(y.z, pv, am[t + 2]);
            am[t + 3] = fmaf(y.w, pv, am[t + 3]);
            aq[t] = fmaf(g.x, sv, aq[t]);
            aq[t + 1] = fmaf(g.y, sv, aq[t + 1]);
            aq[t + 2] = fmaf(g.z, sv, aq[t + 2]);
            aq[t + 3] = fmaf(g.w, sv, aq[t + 3]);
        }
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const int64_t r = row0 + t;
        if (r >= p.n) break;
        float v = am[t] * __half2float(__float2half_rn(tq_load_any(p.norms, r, p.norm_dt)));
        if (p.with_qjl) v += aq[t] * (p.qjl_scale * __half2float(__float2half_rn(tq_load_any(p.rnorms, r, p.rnorm_dt))));
        p.out[r * D + j] = v;
    }
}

// ------------------------------------------------------------------ scores of key planes

// Unscaled logits of 64 tokens of one head (two threads per token) for GP queries; the queries are prepared (qprep).  A thread
// asks for its whole half row at once (16 bytes at a time where the planes are aligned: `vec`), and a CTA holds no more queries
// than it was asked for.
template <int D, int MSE_BITS, int GP>
__global__ void __launch_bounds__(128) tq_rows_scores_kernel(const RowsParams p, const float* qprep, int64_t n_k, int n_q, int vec, float* logits) {
    constexpr int NSW = HalfRow<D, MSE_BITS>::NSW, NCW = HalfRow<D, MSE_BITS>::NCW;
    __shared__ __align__(16) float qs[GP][2][D];
    __shared__ float sp[GP * 64], cent[TQ_MAX_CENTROIDS];
    const int tid = threadIdx.x, h = blockIdx.y, q0 = blockIdx.z * GP, nq = min(GP, n_q - q0);
    if (tid < TQ_MAX_CENTROIDS) cent[tid] = p.cb.centroids[tid];
    const int tk = tid & 63, half = tid >> 6;
    const int64_t t = (int64_t)blockIdx.x * 64 + tk, row = (int64_t)h * n_k + t;
    wait_for_launch_ahead();
    uint32_t cw[NCW], sw[NSW];
    float norm = 0.f, rn = 0.f;
    if (t < n_k) {
        const uint32_t* c = reinterpret_cast<const uint32_t*>(p.codes + row * (8 * NCW)) + half * NCW;
        const uint32_t* g = reinterpret_cast<const uint32_t*>(p.signs + row * (D / 8)) + half * NSW;
        if (vec) {
#pragma unroll
            for (int k = 0; k < NCW; k += 4) {
                const uint4 v = *reinterpret_cast<const uint4*>(c + k);
                cw[k] = v.x; cw[k + 1] = v.y; cw[k + 2] = v.z; cw[k + 3] = v.w;
            }
#pragma unroll
            for (int k = 0; k < NSW; k += 2) {
                const uint2 v = *reinterpret_cast<const uint2*>(g + k);
                sw[k] = v.x; sw[k + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < NCW; ++k) cw[k] = c[k];
#pragma unroll
            for (int k = 0; k < NSW; ++k) sw[k] = g[k];
        }
        norm = __half2float(__float2half_rn(tq_load_any(p.norms, row, p.norm_dt)));
        rn = __half2float(__float2half_rn(tq_load_any(p.rnorms, row, p.rnorm_dt))) * p.qjl_scale;
    }
    const float4* src = reinterpret_cast<const float4*>(qprep + ((int64_t)h * n_q + q0) * 2 * D);
    for (int i = tid; i < GP * 2 * D / 4; i += 128)
        reinterpret_cast<float4*>(qs)[i] = i < nq * 2 * D / 4 ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    float part[GP];
    if (t < n_k) {
        float am[GP], aq[GP];
        half_row_dots<D, MSE_BITS, GP>(cw, sw, qs, cent, half, am, aq);
#pragma unroll
        for (int g = 0; g < GP; ++g) part[g] = norm * am[g] + rn * aq[g];
        if (half)
#pragma unroll
            for (int g = 0; g < GP; ++g) sp[g * 64 + tk] = part[g];
    }
    __syncthreads();
    if (!half && t < n_k)
#pragma unroll
        for (int g = 0; g < GP; ++g)
            if (g < nq) logits[((int64_t)h * n_q + q0 + g) * n_k + t] = part[g] + sp[g * 64 + tk];
}

// A kernel of this file behind whatever was launched last: its constants are loaded under that launch.
template <class Kern, class... Args>
int launch_rows(Kern kern, dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    tq_note_launch(st, TQ_LAUNCH_WAITED);
    return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess ? TQ_OK : TQ_ERR_CUDA;
}

bool aligned(const void* p, size_t n) { return ((uintptr_t)p & (n - 1)) == 0; }

int fill(RowsParams& p, const tq_consts* c, bool quantise) {
    for (int i = 0; i < 2; ++i) {
        p.pi[i] = c->rows_pi[i];
        p.other[i] = quantise ? c->rows_m[i] : c->rows_s[i];
        if (c->cfg.head_dim == RD && (!p.pi[i] || !p.other[i] || !aligned(p.pi[i], 16) || !aligned(p.other[i], 16))) return TQ_ERR_UNSUPPORTED;
    }
    for (int i = 0; i < TQ_MAX_CENTROIDS; ++i) {
        p.cb.centroids[i] = c->centroids[i];
        p.cb.boundaries[i] = c->boundaries[i];
    }
    p.qjl_scale = c->qjl_scale;
    p.pi_t = c->pi_t;
    return TQ_OK;
}

unsigned rows_grid(int64_t n) {
    const int64_t tiles = (n + R_ROWS - 1) / R_ROWS;
    return (unsigned)(tiles < tq_sm_count() ? tiles : tq_sm_count());
}

}  // namespace

extern "C" int tq_rows_quantize_values(const void* v, tq_dtype dtype, int64_t n_rows, int32_t head_dim, int64_t stride_row, int32_t bits,
                                       uint8_t* data, void* scales, void* zeros, void* stream) {
    if (!v || !data || !scales || !zeros) return TQ_ERR_NULL;
    if (n_rows < 0 || head_dim <= 0 || head_dim % 32 || stride_row < head_dim) return TQ_ERR_SHAPE;
    if (bits != 2 && bits != 4) return TQ_ERR_UNSUPPORTED;
    if (!aligned(v, 16) || (stride_row * (int64_t)tq_dtype_size(dtype)) % 16 || !aligned(data, 16)) return TQ_ERR_ALIGN;
    if (n_rows == 0) return TQ_OK;
    const int gpr = head_dim / 32;
    const int64_t n = n_rows * gpr;
    const dim3 grid((unsigned)((4 * n + 255) / 256));
    cudaStream_t st = (cudaStream_t)stream;
#define TQ_QV(DT)                                                                                                     \
    return bits == 2 ? launch_rows(tq_rows_quantize_values_kernel<DT, 2>, grid, 256, 0, st, v, n, gpr, stride_row, data, scales, zeros) \
                     : launch_rows(tq_rows_quantize_values_kernel<DT, 4>, grid, 256, 0, st, v, n, gpr, stride_row, data, scales, zeros)
    if (dtype == TQ_F32) TQ_QV(TQ_F32);
    if (dtype == TQ_BF16) TQ_QV(TQ_BF16);
    if (dtype == TQ_F16) TQ_QV(TQ_F16);
#undef TQ_QV
    return TQ_ERR_UNSUPPORTED;
}

extern "C" int tq_rows_dequantize_values(const uint8_t* data, const void* scales, const void* zeros, tq_dtype scale_dtype, int64_t n_rows,
                                         int32_t head_dim, int32_t bits, float* out, void* stream) {
    if (!data || !scales || !zeros || !out) return TQ_ERR_NULL;
    if (n_rows < 0 || head_dim <= 0 || head_dim % 32) return TQ_ERR_SHAPE;
    if (bits != 2 && bits != 4) return TQ_ERR_UNSUPPORTED;
    if (!aligned(data, 4) || !aligned(out, 16)) return TQ_ERR_ALIGN;
    if (n_rows == 0) return TQ_OK;
    const int64_t quads = n_rows * head_dim / 4;
    const dim3 grid((unsigned)((quads + 255) / 256));
    cudaStream_t st = (cudaStream_t)stream;
    return bits == 2 ? launch_rows(tq_rows_dequantize_values_kernel<2>, grid, 256, 0, st, data, scales, zeros, (int)scale_dtype, quads, out)
                     : launch_rows(tq_rows_dequantize_values_kernel<4>, grid, 256, 0, st, data, scales, zeros, (int)scale_dtype, quads, out);
}

extern "C" int tq_rows_quantize_keys(const tq_consts* consts, const void* x, tq_dtype dtype, int64_t n_rows, int64_t stride_row, uint8_t* codes,
                                     uint8_t* signs, void* norms, tq_dtype norm_dtype, void* residual_norms, tq_dtype residual_dtype, void* stream) {
    if (!consts || !x || !codes || !signs || !norms || !residual_norms) return TQ_ERR_NULL;
    int rc = tq_check_config(&consts->cfg);
    if (rc != TQ_OK) return rc;
    if (consts->cfg.head_dim != RD || dtype == TQ_BF16 || !consts->pi_t) return TQ_ERR_UNSUPPORTED;
    if (n_rows < 0 || stride_row < RD) return TQ_ERR_SHAPE;
    if (!aligned(x, 8) || (stride_row * (int64_t)tq_dtype_size(dtype)) % 8 || !aligned(codes, 16) || !aligned(signs, 16)) return TQ_ERR_ALIGN;
    if (n_rows == 0) return TQ_OK;
    RowsParams p = {};
    if ((rc = fill(p, consts, true)) != TQ_OK) return rc;
    p.x = x;
    p.n = n_rows;
    p.stride_row = stride_row;
    p.codes = codes;
    p.signs = signs;
    p.norms = norms;
    p.rnorms = residual_norms;
    p.norm_dt = norm_dtype;
    p.rnorm_dt = residual_dtype;
    cudaStream_t st = (cudaStream_t)stream;
    const int vec = aligned(x, 16) && (stride_row * (int64_t)tq_dtype_size(dtype)) % 16 == 0;
    constexpr size_t smem = 4 * R_MAT + R_XCHG;
#define TQ_QK(DT, MB)                                                                            \
    do {                                                                                         \
        static TqSmemOptIn opt_in;                                                               \
        if (tq_opt_in_smem(tq_rows_quantize_keys_kernel<DT, MB>, smem, opt_in) != TQ_OK) return TQ_ERR_CUDA; \
        return launch_rows(tq_rows_quantize_keys_kernel<DT, MB>, dim3(rows_grid(n_rows)), R_THREADS, smem, st, p, vec); \
    } while (0)
    const int mb = consts->cfg.key_bits - 1;
    if (dtype == TQ_F32) { if (mb == 2) TQ_QK(TQ_F32, 2); else TQ_QK(TQ_F32, 3); }
    if (dtype == TQ_F16) { if (mb == 2) TQ_QK(TQ_F16, 2); else TQ_QK(TQ_F16, 3); }
#undef TQ_QK
    return TQ_ERR_UNSUPPORTED;
}

extern "C" int tq_rows_dequantize_keys(const tq_consts* consts, const uint8_t* codes, const uint8_t* signs, const void* norms, tq_dtype norm_dtype,
                                       const void* residual_norms, tq_dtype residual_dtype, int64_t n_rows, int32_t with_qjl, float* out, void* stream) {
    if (!consts || !codes || !norms || !out || (with_qjl && (!signs || !residual_norms))) return TQ_ERR_NULL;
    int rc = tq_check_config(&consts->cfg);
    if (rc != TQ_OK) return rc;
    if (!consts->pi || !consts->s) return TQ_ERR_NULL;
    if (n_rows < 0) return TQ_ERR_SHAPE;
    if (!aligned(codes, 8) || (signs && !aligned(signs, 4)) || !aligned(out, 8)) return TQ_ERR_ALIGN;
    if (n_rows == 0) return TQ_OK;
    RowsParams p = {};
    rc = fill(p, consts, false);
    if (rc != TQ_OK) return rc;
    p.n = n_rows;
    p.codes = const_cast<uint8_t*>(codes);
    p.signs = const_cast<uint8_t*>(signs);
    p.norms = const_cast<void*>(norms);
    p.rnorms = const_cast<void*>(residual_norms);
    p.norm_dt = norm_dtype;
    p.rnorm_dt = residual_dtype;
    p.with_qjl = with_qjl;
    p.out = out;
    cudaStream_t st = (cudaStream_t)stream;
    const int mb = consts->cfg.key_bits - 1;
    if (consts->cfg.head_dim != RD)
        return launch_rows(tq_rows_dequantize_keys256_kernel, dim3((unsigned)((n_rows + 15) / 16)), 256, 0, st, p, (const float*)consts->pi, (const float*)consts->s, mb);
    constexpr size_t smem = 4 * R_MAT + KSTEPS * R_THREADS * sizeof(float4) + 16 * sizeof(float);
    static TqSmemOptIn opt2, opt3;
    if (mb == 2) {
        if (tq_opt_in_smem(tq_rows_dequantize_keys_kernel<2>, smem, opt2) != TQ_OK) return TQ_ERR_CUDA;
        return launch_rows(tq_rows_dequantize_keys_kernel<2>, dim3(rows_grid(n_rows)), R_THREADS, smem, st, p);
    }
    if (tq_opt_in_smem(tq_rows_dequantize_keys_kernel<3>, smem, opt3) != TQ_OK) return TQ_ERR_CUDA;
    return launch_rows(tq_rows_dequantize_keys_kernel<3>, dim3(rows_grid(n_rows)), R_THREADS, smem, st, p);
}

extern "C" int tq_rows_scores(const tq_consts* consts, const uint8_t* codes, const uint8_t* signs, const void* norms, tq_dtype norm_dtype,
                              const void* residual_norms, tq_dtype residual_dtype, int32_t n_heads, int64_t n_keys, const void* query, tq_dtype q_dtype,
                              int32_t n_q, float* logits, void* workspace, size_t workspace_bytes, void* stream) {
    if (!consts || !codes || !signs || !norms || !residual_norms || !query || !logits || !workspace) return TQ_ERR_NULL;
    int rc = tq_check_config(&consts->cfg);
    if (rc != TQ_OK) return rc;
    if (!consts->pi_t || !consts->s_t) return TQ_ERR_NULL;
    if (n_heads <= 0 || n_keys < 0 || n_q <= 0) return TQ_ERR_SHAPE;
    if (n_heads > 65535 || n_q > 8 * 65535) return TQ_ERR_UNSUPPORTED;
    if (!aligned(codes, 4) || !aligned(signs, 4) || !aligned(workspace, 256)) return TQ_ERR_ALIGN;
    size_t need = 0;
    tq_scores_workspace_bytes(&consts->cfg, (int64_t)n_heads * n_q, &need);
    if (need > workspace_bytes) return TQ_ERR_WORKSPACE;
    if (n_keys == 0) return TQ_OK;
    RowsParams p = {};
    for (int i = 0; i < TQ_MAX_CENTROIDS; ++i) p.cb.centroids[i] = consts->centroids[i];
    p.qjl_scale = consts->qjl_scale;
    p.codes = const_cast<uint8_t*>(codes);
    p.signs = const_cast<uint8_t*>(signs);
    p.norms = const_cast<void*>(norms);
    p.rnorms = const_cast<void*>(residual_norms);
    p.norm_dt = norm_dtype;
    p.rnorm_dt = residual_dtype;
    float* qprep = reinterpret_cast<float*>((uint8_t*)workspace + TQ_WS_HEADER_BYTES);
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = tq_prepare_queries(consts, query, q_dtype, (int64_t)n_heads * n_q, qprep, st)) != TQ_OK) return rc;
    const int gp = n_q > 4 ? 8 : n_q > 2 ? 4 : n_q, vec = aligned(codes, 16) && aligned(signs, 8);
    const dim3 grid((unsigned)((n_keys + 63) / 64), (unsigned)n_heads, (unsigned)((n_q + gp - 1) / gp));
#define TQ_RS_(DD, MB, GP) return launch_rows(tq_rows_scores_kernel<DD, MB, GP>, grid, 128, 0, st, p, (const float*)qprep, n_keys, (int)n_q, vec, logits)
#define TQ_RS(DD, MB)                      \
    do {                                   \
        if (gp == 1) TQ_RS_(DD, MB, 1);    \
        if (gp == 2) TQ_RS_(DD, MB, 2);    \
        if (gp == 4) TQ_RS_(DD, MB, 4);    \
        TQ_RS_(DD, MB, 8);                 \
    } while (0)
    const int mb = consts->cfg.key_bits - 1;
    if (consts->cfg.head_dim == 128 && mb == 2) TQ_RS(128, 2);
    if (consts->cfg.head_dim == 128) TQ_RS(128, 3);
    if (mb == 2) TQ_RS(256, 2);
    TQ_RS(256, 3);
#undef TQ_RS
#undef TQ_RS_
}
