// The true 32-bit path's attention over the paged cache (32-bit queries, keys and values, heads of up to 128 elements):
// k_attn_generic's arithmetic, operation for operation, on tiles that several rows share.
//
// k_attn_generic gives every (row, query head) a warp that reads all its keys and values by itself, a lane a key: 32
// neighbouring lanes then read 32 different 128-byte lines per element. Here a block takes the rows of neighbouring tokens
// and of the query heads that read one key/value head (AR_ROWS of them, four a warp), brings each run of 32 positions
// into shared memory once, 16 bytes a copy and one run ahead, and every warp computes its four rows from there: a lane
// holds a position for the scores (q . k in order of the elements) and four neighbouring dimensions for P V (positions in
// order). Runs start at multiples of 32 of the absolute position, sums and running maxima go by runs, and a position that a
// row does not see is left out, as there, so a row's bits are the same however the step's tokens are cut. What bounds it is
// the chain of a row's runs (latency), no unit of the GPU: two prompts of 313 and 201 tokens (8 heads of 128 on 2 key/value
// heads) keep 41 % of the issue slots and 23 % of the FMA pipe busy, a warp waiting for its own last result; 52 us a layer
// instead of 445 in k_attn_generic. Together with the tiles of gemm_f32.cu a step of these prompts through four layers of
// width 1024 takes 2.94 ms instead of 5.89.
#include "common.cuh"

#define AR_WARPS 4
#define AR_R 4                          // rows a warp
#define AR_ROWS (AR_WARPS * AR_R)
#define AR_HD 128

__device__ __forceinline__ void ar_cp16(uint32_t dst, const void* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(AR_WARPS * 32) k_attn_rows(const float* KB_STEP_DATA q, int ldq, float* __restrict__ out,
        int ldo, const int* __restrict__ pos, const int* __restrict__ seq, const int* __restrict__ slot, int Tn, int nkv,
        int group, int gh, int tb, int hd, float scale, int window, int keep_first, KbCacheView cv, int* status,
        const float* __restrict__ sink, const float* KB_STEP_DATA gate, int ldg, int chunk, float cap, int vd) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_pos[AR_ROWS], s_seq[AR_ROWS];
    kb_pdl_launch();
    const int ldk = hd + 4;
    float* ks = sm;                                  // [2][32][hd + 4]
    float* vs = ks + 2 * 32 * ldk;                   // [2][32][vd]
    float* qs = vs + 2 * 32 * vd;                    // [AR_ROWS][hd]
    float* ps = qs + AR_ROWS * hd;                   // [AR_WARPS][32][AR_R]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hk = blockIdx.y % nkv, h0 = (blockIdx.y / nkv) * gh;          // heads h0 .. of the group
    const int nh_here = min(gh, group - h0);
    const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * tb, nt = min(tb, Tn - t0);     // (the longest rows first)
    bool first = false;                              // of its sequence's tokens in the tile
    if (tid < nt) {
        const int p = pos[t0 + tid], s = seq[t0 + tid];
        s_pos[tid] = p;
        s_seq[tid] = s;
        first = p >= 0 && (tid == 0 || pos[t0 + tid - 1] < 0 || seq[t0 + tid - 1] != s);
    }
    if (gridDim.z > 1 && __syncthreads_count(first) <= (int)blockIdx.z) return;
    kb_pdl_wait();
    const int n_rows = nt * nh_here;
    for (int e = tid * 4; e < n_rows * hd; e += AR_WARPS * 32 * 4) {
        const int r = e / hd, d = e % hd;
        const float4 v = *(const float4*)(q + (size_t)(t0 + r / nh_here) * ldq +
                                          (size_t)(hk * group + h0 + r % nh_here) * hd + d);
        *(float4*)(qs + e) = make_float4(__fmul_rn(v.x, scale), __fmul_rn(v.y, scale), __fmul_rn(v.z, scale),
                                         __fmul_rn(v.w, scale));
    }
    __syncthreads();
    const uint32_t ks_u = (uint32_t)__cvta_generic_to_shared(ks), vs_u = (uint32_t)__cvta_generic_to_shared(vs);
    float* pw = ps + warp * 32 * AR_R;

    // the tile's tokens, one sequence after the other (padding rows belong to none), every gridDim.z-th sequence here
    int part = 0;
    for (int i0 = 0; i0 < nt;) {
        int i1 = i0 + 1;
        if (s_pos[i0] < 0) {
            i0 = i1;
            continue;
        }
        int lo_min = kb_span_lo(s_pos[i0], window, chunk), p_max = s_pos[i0];
        while (i1 < nt && s_pos[i1] >= 0 && s_seq[i1] == s_seq[i0]) {
            lo_min = min(lo_min, kb_span_lo(s_pos[i1], window, chunk));
            p_max = max(p_max, s_pos[i1]);
            i1++;
        }
        if (part++ % (int)gridDim.z != (int)blockIdx.z) {        // (another block's)
            i0 = i1;
            continue;
        }
        const int* trow = cv.table + (size_t)slot[s_seq[i0]] * cv.table_stride;
        const int c_lo = lo_min & ~31, c_keep = min((keep_first + 31) & ~31, c_lo);
        // (a page holds two whole runs: a run's positions lie in one page)
        auto page_of = [&](int c) {
            const int page = trow[c / KB_PAGE];
            return page < cv.n_pages ? page : -1;
        };
        auto fetch = [&](int c, int page, int buf) { // the run of positions c .. c + 31 (none past the last row's)
            const int pieces_k = hd / 4, pieces_v = vd / 4;
            const float* kr = (const float*)cv.pool + (page < 0 ? 0 : kb_kv_offset(cv, page, 0, hk, c % KB_PAGE));
            const float* vr = (const float*)cv.pool + (page < 0 ? 0 : kb_kv_offset(cv, page, 1, hk, c % KB_PAGE));
            for (int e = tid; e < 32 * pieces_k; e += AR_WARPS * 32) {
                const int r = e / pieces_k, d = (e % pieces_k) * 4;
                const bool on = page >= 0 && c + r <= p_max;
                ar_cp16(ks_u + ((buf * 32 + r) * ldk + d) * 4, on ? kr + (size_t)r * hd + d : cv.pool, on);
            }
            for (int e = tid; e < 32 * pieces_v; e += AR_WARPS * 32) {
                const int r = e / pieces_v, d = (e % pieces_v) * 4;
                const bool on = page >= 0 && c + r <= p_max;
                ar_cp16(vs_u + ((buf * 32 + r) * vd + d) * 4, on ? vr + (size_t)r * hd + d : cv.pool, on);
            }
        };
        float m[AR_R], l[AR_R], o[AR_R][4];
        int p_q[AR_R], lo[AR_R], rq[AR_R];           // position, first position, row of qs
#pragma unroll
        for (int r = 0; r < AR_R; r++) {
            const int row = warp * AR_R + r, i = row / nh_here;
            const bool on = row < n_rows && i >= i0 && i < i1;
            p_q[r] = on ? s_pos[i] : -1;
            lo[r] = on ? kb_span_lo(s_pos[i], window, chunk) : 0;
            rq[r] = on ? row : 0;
            m[r] = -1e30f;
            l[r] = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; c++) o[r][c] = 0.0f;
        }
        int c0 = c_keep > 0 ? 0 : c_lo, buf = 0;
        int page = page_of(c0);
        fetch(c0, page, 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (; c0 <= p_max; buf ^= 1) {
            const int cn = c0 + 32 == c_keep ? c_lo : c0 + 32;
            const int page_n = cn <= p_max ? page_of(cn) : -1;
            if (cn <= p_max) fetch(cn, page_n, buf ^ 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            const int p = c0 + lane;
            bool ok[AR_R], any = false;
            uint32_t mask[AR_R];
#pragma unroll
            for (int r = 0; r < AR_R; r++) {
                const bool live = (p >= lo[r] || p < keep_first) && p <= p_q[r];
                if (live && page < 0) atomicOr(status, KB_ST_BAD_PAGE);
                ok[r] = live && page >= 0;
                mask[r] = __ballot_sync(0xffffffffu, ok[r]);
                any = any || mask[r] != 0;
            }
            if (any) {
                float a[AR_R] = {0.0f, 0.0f, 0.0f, 0.0f};
                const float* kl = ks + (buf * 32 + lane) * ldk;
#pragma unroll 4
                for (int d = 0; d < hd; d += 4) {
                    const float4 k4 = *(const float4*)(kl + d);
#pragma unroll
                    for (int r = 0; r < AR_R; r++) {
                        const float4 q4 = *(const float4*)(qs + rq[r] * hd + d);
                        a[r] = fmaf(q4.x, k4.x, a[r]);
                        a[r] = fmaf(q4.y, k4.y, a[r]);
                        a[r] = fmaf(q4.z, k4.z, a[r]);
                        a[r] = fmaf(q4.w, k4.w, a[r]);
                    }
                }
                float pr[AR_R];
#pragma unroll
                for (int r = 0; r < AR_R; r++) {
                    pr[r] = 0.0f;
                    if (mask[r] == 0) continue;      // (uniform) nothing of this run is seen: the row stays as it is
                    const float sc = cap > 0.0f ? cap * tanhf(a[r] / cap) : a[r];
                    const float mx = kb_warp_max(ok[r] ? sc : -1e30f);
                    const float mn = fmaxf(m[r], mx);
                    const float f = expf(m[r] - mn);
                    pr[r] = ok[r] ? expf(sc - mn) : 0.0f;
                    l[r] = l[r] * f + kb_warp_sum(pr[r]);
                    m[r] = mn;
#pragma unroll
                    for (int c = 0; c < 4; c++) o[r][c] *= f;
                }
                *(float4*)(pw + lane * AR_R) = make_float4(pr[0], pr[1], pr[2], pr[3]);
                __syncwarp();
                if (lane * 4 < vd) {
                    const float* vl = vs + buf * 32 * vd + lane * 4;
                    if ((mask[0] & mask[1] & mask[2] & mask[3]) == 0xffffffffu) {
#pragma unroll 8
                        for (int j = 0; j < 32; j++) {
                            const float4 v4 = *(const float4*)(vl + j * vd), p4 = *(const float4*)(pw + j * AR_R);
                            const float pj[AR_R] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int r = 0; r < AR_R; r++) {
                                o[r][0] = fmaf(pj[r], v4.x, o[r][0]);
                                o[r][1] = fmaf(pj[r], v4.y, o[r][1]);
                                o[r][2] = fmaf(pj[r], v4.z, o[r][2]);
                                o[r][3] = fmaf(pj[r], v4.w, o[r][3]);
                            }
                        }
                    } else {
                        for (int j = 0; j < 32; j++) {
                            const float4 v4 = *(const float4*)(vl + j * vd), p4 = *(const float4*)(pw + j * AR_R);
                            const float pj[AR_R] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int r = 0; r < AR_R; r++)
                                if ((mask[r] >> j) & 1u) {
                                    o[r][0] = fmaf(pj[r], v4.x, o[r][0]);
                                    o[r][1] = fmaf(pj[r], v4.y, o[r][1]);
                                    o[r][2] = fmaf(pj[r], v4.z, o[r][2]);
                                    o[r][3] = fmaf(pj[r], v4.w, o[r][3]);
                                }
                        }
                    }
                }
            }
            __syncthreads();                         // the buffer is free for the run after the next
            c0 = cn;
            page = page_n;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int r = 0; r < AR_R; r++) {
            if (p_q[r] < 0) continue;
            const int row = warp * AR_R + r, t = t0 + row / nh_here, h = hk * group + h0 + row % nh_here;
            if (sink != nullptr) {
                const float sk = sink[h];
                const float mn = fmaxf(m[r], sk);
                const float f = expf(m[r] - mn);
                l[r] = l[r] * f + expf(sk - mn);
#pragma unroll
                for (int c = 0; c < 4; c++) o[r][c] *= f;
            }
            if (lane * 4 < vd) {
                float v[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    v[c] = o[r][c] / l[r];
                    if (gate != nullptr)
                        v[c] = v[c] * (1.0f / (1.0f + expf(-gate[(size_t)t * ldg + (size_t)h * vd + lane * 4 + c])));
                }
                *(float4*)(out + (size_t)t * ldo + (size_t)h * vd + lane * 4) = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
        i0 = i1;
    }
}

// whether k_attn_rows takes the shape: everything it moves 16 bytes at a time is aligned for it
bool kb_attn_rows_takes(const void* q, int ldq, const void* out, int ldo, const void* pool, int hd, int vd) {
    return hd <= AR_HD && hd % 4 == 0 && vd % 4 == 0 && ldq % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)q & 15) == 0 &&
           ((uintptr_t)out & 15) == 0 && ((uintptr_t)pool & 15) == 0;
}

// Sequences (at most n_seq) that share a tile run through it one after the other, each with the chain of its own positions, so
// a tile is not made longer than a sequence's rows on average (single tokens: a tile each), and the sequences of a tile are
// dealt out over gridDim.z blocks, as many as a grid of 4096 blocks has room for and at least two; blocks that find nothing
// leave. 16 decoded tokens of 16 heads on their own key/value heads, context 1000: one block a tile of 16 sequences 1179 us,
// a tile each 99 (k_attn_generic 785); 200 new tokens beside 15 single tokens at 4000: 2527 and 460 (3235).
int kb_attn_rows(const float* q, int ldq, float* out, int ldo, const int* pos, const int* seq, const int* slot, int T, int n_seq,
                 int nkv, int group, int hd, float scale, int window, int keep_first, const KbCacheView& cv, int* status,
                 const float* sink, const float* gate, int ldg, int chunk, float cap, int vd, cudaStream_t st) {
    const int B = n_seq < 1 ? 1 : n_seq < T ? n_seq : T;
    const int gh = group < AR_ROWS ? group : AR_ROWS, most = AR_ROWS / gh, mean = (T + B - 1) / B, tb = mean < most ? mean : most;
    const int tiles = (T + tb - 1) / tb, y = nkv * ((group + gh - 1) / gh);
    const long long room = 4096 / ((long long)tiles * y);
    int z = tb < B ? tb : B;
    if (z > (room < 2 ? 2 : room)) z = room < 2 ? 2 : (int)room;
    const size_t smem = (size_t)(2 * 32 * (hd + 4) + 2 * 32 * vd + AR_ROWS * hd + AR_WARPS * 32 * AR_R) * 4;
    static char once_tag;
    if (kb_first_use(&once_tag)) {
        const int bytes = (2 * 32 * (AR_HD + 4) + 2 * 32 * AR_HD + AR_ROWS * AR_HD + AR_WARPS * 32 * AR_R) * 4;
        cudaError_t e = cudaFuncSetAttribute(k_attn_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
    }
    kb_launch(k_attn_rows, dim3(tiles, y, z), AR_WARPS * 32, smem, st, q, ldq, out, ldo, pos,
              seq, slot, T, nkv, group, gh, tb, hd, scale, window, keep_first, cv, status, sink, gate, ldg, chunk, cap, vd);
    KB_LAUNCH_RET();
}
