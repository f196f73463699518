// The two halves of attention of the single-object cache (kv_cache.py:225-320): logits of all tokens, compressed history
// and exact buffer alike, and the weighted sum of their values.  One launch each (the logits behind the query
// preparation); the history is never dequantised to memory and neither half is assembled from pieces afterwards.
//
// Both are small (a few hundred KB of records): what bounds them is the number of launches and the length of the
// dependent chain per CTA, so the tokens are cut fine enough for a wave of CTAs.
//
// Measured (B200, 8 heads, 4096 tokens, one query): 171 us a step of logits, softmax and output -> 29, of which 27 on the
// device (logits 9.5, output 10.5).
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
    int32_t* status;
};

// eight consecutive elements (16-byte aligned for 16-bit types) as fp32
__device__ __forceinline__ void load8(const void* p, int64_t i, int dt, float (&x)[8]) {
    if (dt == TQ_F32) {
        const float4 a = *reinterpret_cast<const float4*>((const float*)p + i), b = *reinterpret_cast<const float4*>((const float*)p + i + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        return;
    }
    const uint4 v = *reinterpret_cast<const uint4*>((const uint16_t*)p + i);
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

// grid (history tiles + buffer tiles, heads, groups of eight queries); two threads per token, one per half of the dims
template <int D, int MSE_BITS>
__global__ void __launch_bounds__(128) tq_cache_scores_kernel(const CacheParams p, int key_bits, int val_bits) {
    constexpr int GP = 8;
    const TqLayout L = tq_make_layout(D, key_bits, val_bits);
    __shared__ __align__(16) float qr[D * GP], qs[D * GP], sp[2 * GP * CA_TOK], cent[TQ_MAX_CENTROIDS];
    const int tid = threadIdx.x, h = blockIdx.y, q0 = blockIdx.z * GP, nq = min(GP, p.n_q - q0);
    const int hist_tiles = (int)((p.n_tokens + CA_TOK - 1) / CA_TOK);
    const bool hist = (int)blockIdx.x < hist_tiles;
    if (tid < TQ_MAX_CENTROIDS) cent[tid] = p.cb.centroids[tid];
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the prepared query (and with it everything launched before)
    for (int i = tid; i < D * GP; i += 128) {
        const int j = i / GP, g = i % GP;
        float a = 0.f, c = 0.f;
        if (g < nq) {
            const int64_t v = (int64_t)h * p.n_q + q0 + g;
            a = hist ? p.qprep[v * 2 * D + j] : tq_load_any(p.query, v * D + j, p.q_dt);
            if (hist) c = p.qprep[(v * 2 + 1) * D + j];
        }
        qr[i] = a;
        qs[i] = c;
    }
    __syncthreads();
    const int tk = tid & (CA_TOK - 1), half = tid >> 6;
    const int64_t t = hist ? (int64_t)blockIdx.x * CA_TOK + tk : (int64_t)(blockIdx.x - hist_tiles) * CA_TOK + tk;
    float part[GP];
#pragma unroll
    for (int g = 0; g < GP; ++g) part[g] = 0.f;
    if (hist && t < p.n_tokens) {
        int64_t phys = p.block_table[t >> 4];
        if (phys < 0 || phys >= p.num_blocks) {
            atomicCAS(p.status, 0, (int)TQ_ERR_RANGE);
            phys = 0;
        }
        token_half_scores<D, MSE_BITS, GP>(p.pool + (phys * p.H + h) * (int64_t)L.block_bytes, L, (int)(t & 15), half, qr, qs, cent, p.qjl_scale, part);
    } else if (!hist && t < p.n_buf) {
        const int64_t row = (int64_t)h * p.stride_head + t * p.stride_token + half * (D / 2);
#pragma unroll 2
        for (int j = 0; j < D / 2; j += 8) {
            float x[8];
            load8(p.buf, row + j, p.buf_dt, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float* q = qr + (half * (D / 2) + j + i) * GP;
#pragma unroll
                for (int g = 0; g < GP; ++g) part[g] = fmaf(q[g], x[i], part[g]);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < GP; ++g) sp[(half * GP + g) * CA_TOK + tk] = part[g];
    __syncthreads();
    const int64_t row_len = p.n_tokens + p.n_buf;
    for (int i = tid; i < nq * CA_TOK; i += 128) {
        const int g = i / CA_TOK, tt = i % CA_TOK;
        const int64_t at = (int64_t)(hist ? blockIdx.x : blockIdx.x - hist_tiles) * CA_TOK + tt;
        if (at < (hist ? p.n_tokens : p.n_buf))
            p.out[((int64_t)h * p.n_q + q0 + g) * row_len + (hist ? 0 : p.n_tokens) + at] = (sp[g * CA_TOK + tt] + sp[(GP + g) * CA_TOK + tt]) * p.scale;
    }
}

// grid (splits, heads, groups of AT_NQ queries), thread = channel.  A split is AT_REC records of the history or as many
// buffered tokens; the split that finishes last adds the partial sums up, in order.
template <int D, int VAL_BITS>
__global__ void __launch_bounds__(D) tq_cache_attend_kernel(const CacheParams p, int key_bits) {
    const TqLayout L = tq_make_layout(D, key_bits, VAL_BITS);
    constexpr int TOK = AT_REC * TQ_BLOCK_TOKENS;
    __shared__ __align__(16) float w[AT_NQ][TOK];
    __shared__ int last;
    const int d = threadIdx.x, h = blockIdx.y, q0 = blockIdx.z * AT_NQ, nq = min(AT_NQ, p.n_q - q0);
    const int hist_splits = (int)((p.n_tokens + TOK - 1) / TOK), x = blockIdx.x;
    const bool hist = x < hist_splits;
    const int64_t first = (int64_t)(hist ? x : x - hist_splits) * TOK;
    const int n_here = (int)min((int64_t)TOK, (hist ? p.n_tokens : p.n_buf) - first);
    const int64_t row_len = p.n_tokens + p.n_buf;
    for (int i = d; i < AT_NQ * TOK; i += D) {
        const int q = i / TOK, t = i % TOK;
        w[q][t] = q < nq && t < n_here ? tq_load_any(p.weights, ((int64_t)h * p.n_q + q0 + q) * row_len + (hist ? 0 : p.n_tokens) + first + t, p.w_dt) : 0.f;
    }
    __syncthreads();
    float acc[AT_NQ];
#pragma unroll
    for (int q = 0; q < AT_NQ; ++q) acc[q] = 0.f;
    if (hist) {
        const int grp = d >> 5;
        const int nrec = (n_here + 15) / 16;
#pragma unroll 2
        for (int r = 0; r < nrec; ++r) {
            int64_t phys = p.block_table[(first >> 4) + r];
            if (phys < 0 || phys >= p.num_blocks) {
                if (d == 0) atomicCAS(p.status, 0, (int)TQ_ERR_RANGE);
                phys = 0;
            }
            const uint8_t* rec = p.pool + (phys * p.H + h) * (int64_t)L.block_bytes;
            // code bytes in the decode kernel's order: 32-bit word (tokens 4q + 2p, + 1) of this channel's byte column
            const int cbyte = VAL_BITS == 2 ? d >> 2 : d >> 1, sh = VAL_BITS == 2 ? 2 * (d & 3) : 4 * (d & 1);
            uint32_t cw[4][2];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int pp = 0; pp < 2; ++pp) {
                    const int off = tq_vcode_native(D, VAL_BITS, 4 * q + 2 * pp, cbyte);
                    cw[q][pp] = *reinterpret_cast<const uint32_t*>(rec + L.off_vcodes + (off & ~3)) >> (8 * (off & 3) + sh);
                }
            uint32_t sc[8], zr[8];   // 16 tokens of this group, fp16
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint4 a = reinterpret_cast<const uint4*>(rec + L.off_vscale + grp * 32)[i], b = reinterpret_cast<const uint4*>(rec + L.off_vzero + grp * 32)[i];
                sc[4 * i] = a.x; sc[4 * i + 1] = a.y; sc[4 * i + 2] = a.z; sc[4 * i + 3] = a.w;
                zr[4 * i] = b.x; zr[4 * i + 1] = b.y; zr[4 * i + 2] = b.z; zr[4 * i + 3] = b.w;
            }
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const uint32_t code = (cw[t >> 2][(t >> 1) & 1] >> (16 * (t & 1))) & ((1u << VAL_BITS) - 1u);
                const float2 s2 = __half22float2(*reinterpret_cast<const __half2*>(&sc[t >> 1])), z2 = __half22float2(*reinterpret_cast<const __half2*>(&zr[t >> 1]));
                // slots past the last token may hold anything
                const float v = 16 * r + t < n_here ? (float)code * ((t & 1) ? s2.y : s2.x) + ((t & 1) ? z2.y : z2.x) : 0.f;
#pragma unroll
                for (int q = 0; q < AT_NQ; ++q) acc[q] = fmaf(w[q][16 * r + t], v, acc[q]);
            }
        }
    } else {
#pragma unroll 8
        for (int t = 0; t < n_here; ++t) {
            const float v = tq_load_any(p.buf, (int64_t)h * p.stride_head + (first + t) * p.stride_token + d, p.buf_dt);
#pragma unroll
            for (int q = 0; q < AT_NQ; ++q) acc[q] = fmaf(w[q][t], v, acc[q]);
        }
    }
    float* mine = p.partials + (((int64_t)blockIdx.z * p.H + h) * p.splits + x) * (AT_NQ * D) + d;
#pragma unroll
    for (int q = 0; q < AT_NQ; ++q) mine[q * D] = acc[q];
    __syncthreads();
    if (d == 0) {
        int t;
        asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(t) : "l"(p.tickets + (int64_t)blockIdx.z * p.H + h) : "memory");
        last = t == p.splits - 1;
        if (last) p.tickets[(int64_t)blockIdx.z * p.H + h] = 0;
    }
    __syncthreads();
    if (!last) return;
    const float* base = p.partials + ((int64_t)blockIdx.z * p.H + h) * p.splits * (AT_NQ * D) + d;
    float sum[AT_NQ];
#pragma unroll
    for (int q = 0; q < AT_NQ; ++q) sum[q] = 0.f;
#pragma unroll 8
    for (int s = 0; s < p.splits; ++s)
#pragma unroll
        for (int q = 0; q < AT_NQ; ++q) sum[q] += __ldcg(base + (int64_t)s * (AT_NQ * D) + q * D);
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
    cfg.gridDim = dim3((unsigned)(tiles(n_tokens, CA_TOK) + tiles(n_buf, CA_TOK)), (unsigned)p.H, (unsigned)tiles(n_q, 8));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    const int kb = consts->cfg.key_bits, vb = consts->cfg.value_bits;
    cudaError_t e;
    if (D == 128) e = kb == 3 ? cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<128, 2>, p, kb, vb) : cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<128, 3>, p, kb, vb);
    else e = kb == 3 ? cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<256, 2>, p, kb, vb) : cudaLaunchKernelEx(&cfg, tq_cache_scores_kernel<256, 3>, p, kb, vb);
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
    const dim3 grid((unsigned)p.splits, (unsigned)p.H, (unsigned)zs);
    cudaStream_t st = (cudaStream_t)stream;
    tq_note_launch(st, TQ_LAUNCH_UNKNOWN);
    const int kb = consts->cfg.key_bits, vb = consts->cfg.value_bits;
    if (D == 128) {
        if (vb == 2) tq_cache_attend_kernel<128, 2><<<grid, 128, 0, st>>>(p, kb);
        else tq_cache_attend_kernel<128, 4><<<grid, 128, 0, st>>>(p, kb);
    } else {
        if (vb == 2) tq_cache_attend_kernel<256, 2><<<grid, 256, 0, st>>>(p, kb);
        else tq_cache_attend_kernel<256, 4><<<grid, 256, 0, st>>>(p, kb);
    }
    return cudaGetLastError() == cudaSuccess ? TQ_OK : TQ_ERR_CUDA;
}
