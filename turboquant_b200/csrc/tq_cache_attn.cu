// The two halves of attention of the single-object cache (kv_cache.py:225-320): logits of all tokens, compressed history
// and exact buffer alike, and the weighted sum of their values.  One launch each (the logits behind the query
// preparation); the history is never dequantised to memory and neither half is assembled from pieces afterwards.
//
// Both are small (a few hundred KB of records): what bounds them is the number of launches and the length of the
// dependent chain per CTA, so the tokens are cut fine enough for a wave of CTAs.
//
// Measured (B200, 8 heads, 4096 tokens, one query, fp16): 18.0 us a step of logits, softmax and output (logits 3.6, output 6.3,
// query preparation and softmax 3.3 each); 28.5 while a CTA worked for eight (logits) or four queries whatever it was asked for,
// and read its records word by word in chains (logits 9.6, output 10.2).
#include "tq_decode_common.cuh"

using namespace tqdec;

namespace {

constexpr int CA_TOK = 64;        // tokens per CTA (logits)
constexpr int AT_REC = 8;         // records per CTA (values): 128 tokens
constexpr int AT_NQ = 4;          // queries a CTA accumulates at a time
// Queries of one call: the partial sums of so many take as much memory as the dequantised history of the way that this kernel
// replaces (a split is 128 tokens), and its matrix product overtakes the kernel's passes over the records between 128 and 256
// (8 heads of 128, 4096 / 32768 tokens: 108 against 162 us and 750 against 904 at 128 queries, 195 against 164 and 1459 against
// 907 at 256; 4 heads of 256, 8192 tokens: 205 against 261, 387 against 265).
constexpr int AT_NQ_MAX = 128;
constexpr int AT_TICKETS = 4096;  // heads x groups of AT_NQ queries; at a fixed place, so that no call's scratch lands on them

struct CacheParams {
    const uint8_t* pool;
    int64_t num_blocks;
    int H;
    const int32_t* block_table;
    int64_t n_tokens;
    int n_q;
    const float* qprep;           // [H][n_q][2][D]
    const void* query;
    int q_dt;
    const void* buf;              // exact keys / values: element (h, t, :) at h * stride_head + t * stride_token
    int buf_dt;
    int64_t n_buf, stride_head, stride_token;
    float scale, qjl_scale;
    TqCodebook cb;
    float* out;
    const void* weights;
    int w_dt;
    float* partials;
    int32_t* tickets;
    int splits;
    int pool_late;                // a store ahead of the query preparation may still be writing records
    int32_t* status;
};

// eight 16-bit elements as fp32
__device__ __forceinline__ void widen8(const uint4& v, int dt, float (&x)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (dt == TQ_BF16) {
            x[2 * j] = __uint_as_float(w[j] << 16);
            x[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
            x[2 * j] = f.x;
            x[2 * j + 1] = f.y;
        }
    }
}
__device__ __forceinline__ void load8(const float* p, float (&x)[8]) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

// grid (history tiles + buffer tiles, heads, groups of GP queries); two threads per token, one per half of the dims.
// A CTA holds no more queries than it was asked for (GP = 1, 2, 4 or 8), and a thread asks for its whole half row in one go,
// in front of the wait for the query preparation where the pool is known to be at rest: what is left behind the wait is the
// prepared query's trip from L2 and a chain of 64 or 128 fused multiply-adds.
template <int D, int MSE_BITS, int GP>
__global__ void __launch_bounds__(128) tq_cache_scores_kernel(const CacheParams p, int key_bits, int val_bits) {
    constexpr int NSW = HalfRow<D, MSE_BITS>::NSW, NCW = HalfRow<D, MSE_BITS>::NCW;
    const TqLayout L = tq_make_layout(D, key_bits, val_bits);
    __shared__ __align__(16) float qs[GP][2][D];         // rotated and sketched query; of a buffer tile the query as it is
    __shared__ float sp[GP * CA_TOK], cent[TQ_MAX_CENTROIDS];
    const int tid = threadIdx.x, h = blockIdx.y, q0 = blockIdx.z * GP, nq = min(GP, p.n_q - q0);
    const int hist_tiles = (int)((p.n_tokens + CA_TOK - 1) / CA_TOK);
    const bool hist = (int)blockIdx.x < hist_tiles;
    const int tk = tid & (CA_TOK - 1), half = tid >> 6;
    const int64_t t = (int64_t)(hist ? blockIdx.x : blockIdx.x - hist_tiles) * CA_TOK + tk;
    const int64_t n = hist ? p.n_tokens : p.n_buf;
    if (tid < TQ_MAX_CENTROIDS) cent[tid] = p.cb.centroids[tid];
    if (p.pool_late) asm volatile("griddepcontrol.wait;" ::: "memory");   // a store may still be writing records
    uint32_t cw[NCW], sw[NSW];
    float norm = 0.f, rnorm = 0.f;
    if (hist && t < n) {
        int64_t phys = p.block_table[t >> 4];
        if (phys < 0 || phys >= p.num_blocks) {
            atomicCAS(p.status, 0, (int)TQ_ERR_RANGE);
            phys = 0;
        }
        const uint8_t* rec = p.pool + (phys * p.H + h) * (int64_t)L.block_bytes;
        const int tl = (int)(t & 15);
        const uint4* c4 = reinterpret_cast<const uint4*>(rec + L.off_kcodes + tl * L.kcode_row) + half * (NCW / 4);
#pragma unroll
        for (int k = 0; k < NCW / 4; ++k) {
            const uint4 v = c4[k];
            cw[4 * k] = v.x; cw[4 * k + 1] = v.y; cw[4 * k + 2] = v.z; cw[4 * k + 3] = v.w;
        }
        const uint2* s2 = reinterpret_cast<const uint2*>(rec + L.off_ksigns + tl * L.ksign_row) + half * (NSW / 2);
#pragma unroll
        for (int k = 0; k < NSW / 2; ++k) {
            const uint2 v = s2[k];
            sw[2 * k] = v.x; sw[2 * k + 1] = v.y;
        }
        norm = __half2float(reinterpret_cast<const __half*>(rec + L.off_knorm)[tl]);
        rnorm = __half2float(reinterpret_cast<const __half*>(rec + L.off_krnorm)[tl]) * p.qjl_scale;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the prepared query (and with it everything launched before)
    if (hist) {
        const float4* src = reinterpret_cast<const float4*>(p.qprep + ((int64_t)h * p.n_q + q0) * 2 * D);
        for (int i = tid; i < GP * 2 * D / 4; i += 128)
            reinterpret_cast<float4*>(qs)[i] = i < nq * 2 * D / 4 ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        for (int i = tid; i < GP * D; i += 128)
            qs[i / D][0][i % D] = i < nq * D ? tq_load_any(p.query, ((int64_t)h * p.n_q + q0) * D + i, p.q_dt) : 0.f;
    }
    float part[GP];
#pragma unroll
    for (int g = 0; g < GP; ++g) part[g] = 0.f;
    if (hist) {
        __syncthreads();
        if (t < n) {
            float am[GP], aq[GP];
            half_row_dots<D, MSE_BITS, GP>(cw, sw, qs, cent, half, am, aq);
#pragma unroll
            for (int g = 0; g < GP; ++g) part[g] = norm * am[g] + rnorm * aq[g];
        }
    } else {
        const int64_t row = (int64_t)h * p.stride_head + t * p.stride_token + half * (D / 2);
        uint4 raw[D / 16];   // the half row, for 16-bit types; on its way while the query is stored
        if (t < n && p.buf_dt != TQ_F32)
#pragma unroll
            for (int k = 0; k < D / 16; ++k) raw[k] = reinterpret_cast<const uint4*>((const uint16_t*)p.buf + row)[k];
        __syncthreads();
        if (t < n) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
                float x[8];
                if (p.buf_dt == TQ_F32) load8((const float*)p.buf + row + 8 * k, x);
                else widen8(raw[k], p.buf_dt, x);
#pragma unroll
                for (int g = 0; g < GP; ++g) {
                    const float4 a = *reinterpret_cast<const float4*>(&qs[g][0][half * (D / 2) + 8 * k]), b = *reinterpret_cast<const float4*>(&qs[g][0][half * (D / 2) + 8 * k + 4]);
                    part[g] = fmaf(a.x, x[0], part[g]); part[g] = fmaf(a.y, x[1], part[g]); part[g] = fmaf(a.z, x[2], part[g]); part[g] = fmaf(a.w, x[3], part[g]);
                    part[g] = fmaf(b.x, x[4], part[g]); part[g] = fmaf(b.y, x[5], part[g]); part[g] = fmaf(b.z, x[6], part[g]); part[g] = fmaf(b.w, x[7], part[g]);
                }
            }
        }
    }
    if (half)
#pragma unroll
        for (int g = 0; g < GP; ++g) sp[g * CA_TOK + tk] = part[g];
    __syncthreads();
    const int64_t row_len = p.n_tokens + p.n_buf;
    if (!half && t < n)
#pragma unroll
        for (int g = 0; g < GP; ++g)
            if (g < nq) p.out[((int64_t)h * p.n_q + q0 + g) * row_len + (hist ? 0 : p.n_tokens) + t] = (part[g] + sp[g * CA_TOK + tk]) * p.scale;
}

// grid (splits, heads, groups of AT_NQ queries), thread = (strand, channel).  A split is AT_REC records of the history or as
// many buffered tokens, which the strands share: strand s takes records s, s + STRANDS, ..., all of whose loads are under way
// at once.  The split that finishes last adds the partial sums up, every strand a range of them.  NQ: queries held, 1, 2 or 4.
constexpr int AT_THREADS = 512;
template <int D, int VAL_BITS, int NQ>
__global__ void __launch_bounds__(AT_THREADS) tq_cache_attend_kernel(const CacheParams p, int key_bits) {
    const TqLayout L = tq_make_layout(D, key_bits, VAL_BITS);
    constexpr int TOK = AT_REC * TQ_BLOCK_TOKENS, STRANDS = AT_THREADS / D, MINE = AT_REC / STRANDS;
    __shared__ __align__(16) float w[NQ][TOK];
    __shared__ float strand_sum[NQ][AT_THREADS];
    __shared__ int last;
    const int tid = threadIdx.x, d = tid % D, strand = tid / D, h = blockIdx.y, q0 = blockIdx.z * AT_NQ, nq = min(NQ, p.n_q - q0);
    const int hist_splits = (int)((p.n_tokens + TOK - 1) / TOK), x = blockIdx.x;
    const bool hist = x < hist_splits;
    const int64_t first = (int64_t)(hist ? x : x - hist_splits) * TOK;
    const int n_here = (int)min((int64_t)TOK, (hist ? p.n_tokens : p.n_buf) - first);
    const int64_t row_len = p.n_tokens + p.n_buf;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // weights and records belong to the launches ahead
    for (int i = tid; i < NQ * TOK; i += AT_THREADS) {
        const int q = i / TOK, t = i % TOK;
        w[q][t] = q < nq && t < n_here ? tq_load_any(p.weights, ((int64_t)h * p.n_q + q0 + q) * row_len + (hist ? 0 : p.n_tokens) + first + t, p.w_dt) : 0.f;
    }
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
    if (hist) {
        const int grp = d >> 5;
        const int nrec = (n_here + 15) / 16;
        // code bytes in the decode kernel's order: 32-bit word (tokens 4q + 2p, + 1) of this channel's byte column
        const int cbyte = VAL_BITS == 2 ? d >> 2 : d >> 1, sh = VAL_BITS == 2 ? 2 * (d & 3) : 4 * (d & 1);
        uint32_t cw[MINE][8];
        uint4 sc[MINE][2], zr[MINE][2];   // 16 tokens of this group, fp16
#pragma unroll
        for (int m = 0; m < MINE; ++m) {
            const int r = strand + m * STRANDS;
            if (r < nrec) {
                int64_t phys = p.block_table[(first >> 4) + r];
                if (phys < 0 || phys >= p.num_blocks) {
                    if (d == 0) atomicCAS(p.status, 0, (int)TQ_ERR_RANGE);
                    phys = 0;
                }
                const uint8_t* rec = p.pool + (phys * p.H + h) * (int64_t)L.block_bytes;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    cw[m][k] = *reinterpret_cast<const uint32_t*>(rec + L.off_vcodes + (tq_vcode_native(D, VAL_BITS, 2 * k, cbyte) & ~3));
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    sc[m][i] = reinterpret_cast<const uint4*>(rec + L.off_vscale + grp * 32)[i];
                    zr[m][i] = reinterpret_cast<const uint4*>(rec + L.off_vzero + grp * 32)[i];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < MINE; ++m) {
            const int r = strand + m * STRANDS;
            if (r < nrec) {
                const uint32_t s8[8] = {sc[m][0].x, sc[m][0].y, sc[m][0].z, sc[m][0].w, sc[m][1].x, sc[m][1].y, sc[m][1].z, sc[m][1].w};
                const uint32_t z8[8] = {zr[m][0].x, zr[m][0].y, zr[m][0].z, zr[m][0].w, zr[m][1].x, zr[m][1].y, zr[m][1].z, zr[m][1].w};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t c = cw[m][k] >> (8 * (tq_vcode_native(D, VAL_BITS, 2 * k, cbyte) & 3) + sh);
                    const float2 s2 = __half22float2(*reinterpret_cast<const __half2*>(&s8[k])), z2 = __half22float2(*reinterpret_cast<const __half2*>(&z8[k]));
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const int t = 16 * r + 2 * k + o;
                        const uint32_t code = (c >> (16 * o)) & ((1u << VAL_BITS) - 1u);
                        // slots past the last token may hold anything
                        const float v = t < n_here ? (float)code * (o ? s2.y : s2.x) + (o ? z2.y : z2.x) : 0.f;
#pragma unroll
                        for (int q = 0; q < NQ; ++q) acc[q] = fmaf(w[q][t], v, acc[q]);
                    }
                }
            }
        }
    } else {
        __syncthreads();
#pragma unroll 8
        for (int t = strand; t < n_here; t += STRANDS) {
            const float v = tq_load_any(p.buf, (int64_t)h * p.stride_head + (first + t) * p.stride_token + d, p.buf_dt);
#pragma unroll
            for (int q = 0; q < NQ; ++q) acc[q] = fmaf(w[q][t], v, acc[q]);
        }
    }
    // the strands' sums, one thread a channel and query
    auto gather = [&](float (&a)[NQ], float (&out)[NQ]) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) strand_sum[q][tid] = a[q];
        __syncthreads();
        if (strand == 0)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                out[q] = a[q];
#pragma unroll
                for (int s = 1; s < STRANDS; ++s) out[q] += strand_sum[q][s * D + d];
            }
    };
    float sum[NQ];
    gather(acc, sum);
    if (strand == 0) {
        float* mine = p.partials + (((int64_t)blockIdx.z * p.H + h) * p.splits + x) * (AT_NQ * D) + d;
#pragma unroll
        for (int q = 0; q < NQ; ++q) mine[q * D] = sum[q];
    }
    __syncthreads();
    if (tid == 0) {
        int t;
        asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(t) : "l"(p.tickets + (int64_t)blockIdx.z * p.H + h) : "memory");
        last = t == p.splits - 1;
        if (last) p.tickets[(int64_t)blockIdx.z * p.H + h] = 0;
    }
    __syncthreads();
    if (!last) return;
    const float* base = p.partials + ((int64_t)blockIdx.z * p.H + h) * p.splits * (AT_NQ * D) + d;
    const int lo = (int)((int64_t)strand * p.splits / STRANDS), hi = (int)((int64_t)(strand + 1) * p.splits / STRANDS);
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
#pragma unroll 8
    for (int s = lo; s < hi; ++s)
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] += __ldcg(base + (int64_t)s * (AT_NQ * D) + q * D);
    gather(acc, sum);
    if (strand == 0)
        for (int q = 0; q < nq; ++q) p.out[((int64_t)h * p.n_q + q0 + q) * D + d] = sum[q];
}

int64_t tiles(int64_t n, int per) { return (n + per - 1) / per; }

int common(CacheParams& p, const tq_consts* consts, const tq_pool* pool, const int32_t* block_table, int64_t n_tokens, int32_t n_q, const void* buf,
           tq_dtype buf_dtype, int64_t n_buf, int64_t stride_head, int64_t stride_token, void* workspace) {
    if (!consts || !pool || !pool->base || !block_table || !workspace || (n_buf > 0 && !buf)) return TQ_ERR_NULL;
    const int rc = tq_check_config(&consts->cfg);
    if (rc != TQ_OK) return rc;
    if (n_tokens <= 0 || n_q <= 0 || n_buf < 0 || pool->num_kv_heads <= 0) return TQ_ERR_SHAPE;
    if (n_q > 8 * 65535 || pool->num_kv_heads > 65535) return TQ_ERR_UNSUPPORTED;
    if (((uintptr_t)pool->base & 15) || ((uintptr_t)workspace & 255)) return TQ_ERR_ALIGN;
    const int64_t eb = (int64_t)tq_dtype_size(buf_dtype);
    if (n_buf > 0 && (((uintptr_t)buf | (uintptr_t)(stride_head * eb) | (uintptr_t)(stride_token * eb)) & 15)) return TQ_ERR_ALIGN;
    p.pool = (const uint8_t*)pool->base;
    p.num_blocks = pool->num_blocks;
    p.H = pool->num_kv_heads;
    p.block_table = block_table;
    p.n_tokens = n_tokens;
    p.n_q = n_q;
    p.buf = buf;
    p.buf_dt = buf_dtype;
    p.n_buf = n_buf;
    p.stride_head = stride_head;
    p.stride_token = stride_token;
    p.qjl_scale = consts->qjl_scale;
    for (int i = 0; i < TQ_MAX_CENTROIDS; ++i) p.cb.centroids[i] = consts->centroids[i];
    p.status = (int32_t*)workspace;
    return TQ_OK;
}

constexpr size_t SCRATCH_AT = TQ_WS_HEADER_BYTES + AT_TICKETS * sizeof(int32_t);

}  // namespace

extern "C" int tq_cache_scores_workspace_bytes(const tq_config* cfg, int32_t n_heads, int32_t n_q, size_t* out) {
    if (!cfg || !out) return TQ_ERR_NULL;
    const int rc = tq_check_config(cfg);
    if (rc != TQ_OK) return rc;
    if (n_heads <= 0 || n_q <= 0) return TQ_ERR_SHAPE;
    if (n_q > 8 * 65535 || n_heads > 65535) return TQ_ERR_UNSUPPORTED;
    *out = SCRATCH_AT + (size_t)n_heads * n_q * 2 * cfg->head_dim * sizeof(float);
    return TQ_OK;
}

extern "C" int tq_cache_attend_workspace_bytes(const tq_config* cfg, int32_t n_heads, int64_t n_tokens, int64_t n_buf, int32_t n_q, size_t* out) {
    if (!cfg || !out) return TQ_ERR_NULL;
    const int rc = tq_check_config(cfg);
    if (rc != TQ_OK) return rc;
    if (n_heads <= 0 || n_tokens < 0 || n_buf < 0 || n_q <= 0) return TQ_ERR_SHAPE;
    const int64_t zs = tiles(n_q, AT_NQ), splits = tiles(n_tokens, AT_REC * TQ_BLOCK_TOKENS) + tiles(n_buf, AT_REC * TQ_BLOCK_TOKENS);
    if (n_q > AT_NQ_MAX || n_heads > 65535 || zs * n_heads > AT_TICKETS) return TQ_ERR_UNSUPPORTED;
    *out = SCRATCH_AT + (size_t)(zs * n_heads * splits * AT_NQ * cfg->head_dim) * sizeof(float);
    return TQ_OK;
}

extern "C" int tq_cache_workspace_bytes(const tq_config* cfg, int32_t n_heads, int64_t n_tokens, int64_t n_buf, int32_t n_q, size_t* out) {
    size_t scores = 0, attend = 0;
    int rc = tq_cache_scores_workspace_bytes(cfg, n_heads, n_q, &scores);
    if (rc == TQ_OK) rc = tq_cache_attend_workspace_bytes(cfg, n_heads, n_tokens, n_buf, n_q, &attend);
    if (rc != TQ_OK && rc != TQ_ERR_UNSUPPORTED) return rc;
    if (scores == 0 && attend == 0) return rc;
    if (!out) return TQ_ERR_NULL;
    *out = scores > attend ? scores : attend;
    return TQ_OK;
}

extern "C" int tq_cache_scores(const tq_consts* consts, const tq_pool* pool, const int32_t* block_table, int64_t n_tokens, const void* query,
                               tq_dtype q_dtype, int32_t n_q, const void* buf_keys, tq_dtype buf_dtype, int64_t n_buf, int64_t stride_head,
                               int64_t stride_token, float scale, float* logits, void* workspace, size_t workspace_bytes, void* stream) {
    CacheParams p = {};
    int rc = common(p, consts, pool, block_table, n_tokens, n_q, buf_keys, buf_dtype, n_buf, stride_head, stride_token, workspace);
    if (rc != TQ_OK) return rc;
    if (!query || !logits || !consts->pi_t || !consts->s_t) return TQ_ERR_NULL;
    const int D = consts->cfg.head_dim;
    size_t need = 0;
    if ((rc = tq_cache_scores_workspace_bytes(&consts->cfg, p.H, n_q, &need)) != TQ_OK) return rc;
    if (need > workspace_bytes) return TQ_ERR_WORKSPACE;
    float* qprep = reinterpret_cast<float*>((uint8_t*)workspace + SCRATCH_AT);
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = tq_prepare_queries(consts, query, q_dtype, (int64_t)p.H * n_q, qprep, st)) != TQ_OK) return rc;
    p.qprep = qprep;
    p.query = query;
    p.q_dt = q_dtype;
    p.scale = scale;
    p.out = logits;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    p.pool_late = tq_pool_is_late(tq_last_launch(st));
    const int gp = n_q > 4 ? 8 : n_q > 2 ? 4 : n_q;
    cfg.gridDim = dim3((unsigned)(tiles(n_tokens, CA_TOK) + tiles(n_buf, CA_TOK)), (unsigned)p.H, (unsigned)tiles(n_q, gp));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    const int kb = consts->cfg.key_bits, vb = consts->cfg.value_bits;
    cudaError_t e = cudaSuccess;
#define TQ_CS(DD, MB)                                                                                     \
    do {                                                                                                  \
        if (gp == 1) e = cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<DD, MB, 1>, p, kb, vb);          \
        else if (gp == 2) e = cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<DD, MB, 2>, p, kb, vb);     \
        else if (gp == 4) e = cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<DD, MB, 4>, p, kb, vb);     \
        else e = cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<DD, MB, 8>, p, kb, vb);                  \
    } while (0)
    if (D == 128 && kb == 3) TQ_CS(128, 2);
    else if (D == 128) TQ_CS(128, 3);
    else if (kb == 3) TQ_CS(256, 2);
    else TQ_CS(256, 3);
#undef TQ_CS
    return e == cudaSuccess ? TQ_OK : TQ_ERR_CUDA;
}

extern "C" int tq_cache_attend(const tq_consts* consts, const tq_pool* pool, const int32_t* block_table, int64_t n_tokens, const void* weights,
                               tq_dtype w_dtype, int32_t n_q, const void* buf_values, tq_dtype buf_dtype, int64_t n_buf, int64_t stride_head,
                               int64_t stride_token, float* out, void* workspace, size_t workspace_bytes, void* stream) {
    CacheParams p = {};
    int rc = common(p, consts, pool, block_table, n_tokens, n_q, buf_values, buf_dtype, n_buf, stride_head, stride_token, workspace);
    if (rc != TQ_OK) return rc;
    if (!weights || !out) return TQ_ERR_NULL;
    const int D = consts->cfg.head_dim;
    size_t need = 0;
    if ((rc = tq_cache_attend_workspace_bytes(&consts->cfg, p.H, n_tokens, n_buf, n_q, &need)) != TQ_OK) return rc;
    if (need > workspace_bytes) return TQ_ERR_WORKSPACE;
    const int64_t zs = tiles(n_q, AT_NQ);
    p.weights = weights;
    p.w_dt = w_dtype;
    p.out = out;
    p.splits = (int)(tiles(n_tokens, AT_REC * TQ_BLOCK_TOKENS) + tiles(n_buf, AT_REC * TQ_BLOCK_TOKENS));
    p.tickets = reinterpret_cast<int32_t*>((uint8_t*)workspace + TQ_WS_HEADER_BYTES);
    p.partials = reinterpret_cast<float*>((uint8_t*)workspace + SCRATCH_AT);
    cudaStream_t st = (cudaStream_t)stream;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // it waits before its first read, and lets nobody start early
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)p.splits, (unsigned)p.H, (unsigned)zs);
    cfg.blockDim = dim3(AT_THREADS);
    cfg.stream = st;
    tq_note_launch(st, TQ_LAUNCH_WAITED);
    const int kb = consts->cfg.key_bits, vb = consts->cfg.value_bits;
    cudaError_t e = cudaSuccess;
#define TQ_CA(DD, VB)                                                                             \
    do {                                                                                          \
        if (n_q == 1) e = cudaLaunchKernelEx(&cfg, tq_cache_attend_kernel<DD, VB, 1>, p, kb);     \
        else if (n_q == 2) e = cudaLaunchKernelEx(&cfg, tq_cache_attend_kernel<DD, VB, 2>, p, kb); \
        else e = cudaLaunchKernelEx(&cfg, tq_cache_attend_kernel<DD, VB, 4>, p, kb);              \
    } while (0)
    if (D == 128 && vb == 2) TQ_CA(128, 2);
    else if (D == 128) TQ_CA(128, 4);
    else if (vb == 2) TQ_CA(256, 2);
    else TQ_CA(256, 4);
#undef TQ_CA
    return e == cudaSuccess ? TQ_OK : TQ_ERR_CUDA;
}
