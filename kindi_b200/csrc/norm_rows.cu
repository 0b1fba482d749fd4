// Residual add and norm (RMS or layer norm) of prompt-sized steps on the bfloat16 path: WPR warps a row, the row's share of
// every warp in registers, the planes PB at a time.
//
// v = x + sum of the planes in order (with a scale per column, ls: x + ls * that sum), written back to x; then
// y = v / rms(v) * w, or (v - mean) / std(v) * w + b. A row's sums are taken by a fixed number of threads in a fixed order.
// What bounds it is the memory: with one plane a row of E elements is 14 E bytes (2048 rows of 2560: 73 MB, much of it in the
// L2). One warp a row with the whole row in registers (the form before, from 1792 rows on) leaves 16 warps on an SM, and four
// warps a row holding three planes at once 16 as well: a block's loads, sums and stores then follow one another with little
// beside them. Few registers and 32 warps on an SM let rows overlap. With
// one plane, RMS norm: 2048 rows of 2560 12.2 -> 8.2 us, 8171 of 5120 155 -> 106 us (5.5 TB/s), 1536 of 2048 7.7 -> 6.2; layer norm
// of 2048 rows of 2560 22.2 -> 11.0, of 4096 32.7 -> 24.3, of 2048 with four planes 25.8 -> 22.0 us (between ordinary kernels).
#include "common.cuh"

// The order of a row's sums. Routers pick experts by what follows a layer norm, and a sum in another order picks others at
// close calls, so a layer norm keeps the order of the form it stands in for: up to 2048 columns one warp a row (NR_LN_LANES:
// lane by lane over the row's pieces of 128 elements in order, then over the lanes), beyond it the block of 512 threads a row
// of k_add_layernorm (NR_LN_BLOCK: a thread's pieces lie 2048 elements apart, then over the lanes of its warp, then over 16
// warps in order). RMS norm (NR_RMS): every warp's own sum, added in the warps' order.
enum { NR_RMS, NR_LN_LANES, NR_LN_BLOCK };
#define NR_BLOCK_WARPS 16               // of k_add_layernorm

// G4: the gains lie on boundaries of four (their loads are then asked for early, before the sums)
template <typename TW, int WPR, int NC, int PB, int KIND, int MINB, bool G4>
__global__ void __launch_bounds__(256, MINB) k_norm_rows(float* KB_STEP_DATA x, const float* KB_STEP_DATA delta, int n_delta,
        size_t delta_stride, const TW* __restrict__ w, const TW* __restrict__ bias, float eps, bf16* __restrict__ y, int T, int E,
        const TW* __restrict__ ls) {
    constexpr bool LN = KIND != NR_RMS;
    constexpr int ROWS = 8 / WPR, STEP = KIND == NR_LN_BLOCK ? WPR * 128 : 128;      // elements between a thread's pieces
    constexpr int VW = NR_BLOCK_WARPS / WPR;                                         // warps of the block form a warp stands for
    __shared__ float red[2][ROWS][KIND == NR_LN_BLOCK ? NR_BLOCK_WARPS : WPR];
    __shared__ float pieces[KIND == NR_LN_LANES ? 2 : 1][KIND == NR_LN_LANES ? ROWS : 1][KIND == NR_LN_LANES ? WPR * NC : 1][32];
    kb_pdl_launch();
    kb_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = warp % WPR, own = warp / WPR;
    const int t = blockIdx.x * ROWS + own;
    const bool live = t < T;
    float* xr = x + (size_t)(live ? t : 0) * E;
    const float* dr = delta + (size_t)(live ? t : 0) * E;
    const bool scaled = !LN && ls != nullptr && n_delta > 0;
    const int i0 = ((KIND == NR_LN_BLOCK ? part : part * NC) * 32 + lane) * 4;      // this thread's elements: i0 + STEP c .. + 3
    float4 v[NC];
#pragma unroll
    for (int c = 0; c < NC; c++)
        v[c] = live && i0 + STEP * c < E && !scaled ? *(const float4*)(xr + i0 + STEP * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < n_delta; s0 += PB) {
        float4 d[PB][NC];
#pragma unroll
        for (int k = 0; k < PB; k++)
#pragma unroll
            for (int c = 0; c < NC; c++)
                d[k][c] = live && s0 + k < n_delta && i0 + STEP * c < E
                              ? *(const float4*)(dr + (size_t)(s0 + k) * delta_stride + i0 + STEP * c)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < PB; k++)
            if (s0 + k < n_delta) {
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    v[c].x += d[k][c].x;
                    v[c].y += d[k][c].y;
                    v[c].z += d[k][c].z;
                    v[c].w += d[k][c].w;
                }
            }
    }
    if (scaled && live) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int i = i0 + STEP * c;
            if (i < E) {
                const float4 xv = *(const float4*)(xr + i);
                v[c].x = __fadd_rn(xv.x, __fmul_rn(v[c].x, kb_to_f<TW>(ls[i])));
                v[c].y = __fadd_rn(xv.y, __fmul_rn(v[c].y, kb_to_f<TW>(ls[i + 1])));
                v[c].z = __fadd_rn(xv.z, __fmul_rn(v[c].z, kb_to_f<TW>(ls[i + 2])));
                v[c].w = __fadd_rn(xv.w, __fmul_rn(v[c].w, kb_to_f<TW>(ls[i + 3])));
            }
        }
    }
    if (n_delta > 0 && live) {
#pragma unroll
        for (int c = 0; c < NC; c++)
            if (i0 + STEP * c < E) *(float4*)(xr + i0 + STEP * c) = v[c];
    }
    auto row_sum = [&](const float (&piece)[NC], int slot) {
        float tot = 0.0f;
        if (KIND == NR_LN_LANES) {
            float* mine = pieces[slot][own][0];
#pragma unroll
            for (int c = 0; c < NC; c++) mine[(part * NC + c) * 32 + lane] = piece[c];
            __syncthreads();
#pragma unroll
            for (int c = 0; c < WPR * NC; c++) tot += mine[c * 32 + lane];
            return kb_warp_sum(tot);
        }
        if (KIND == NR_LN_BLOCK) {
            float s[VW];
#pragma unroll
            for (int k = 0; k < VW; k++) s[k] = 0.0f;
#pragma unroll
            for (int c = 0; c < NC; c++) s[c % VW] += piece[c];
#pragma unroll
            for (int k = 0; k < VW; k++) {
                s[k] = kb_warp_sum(s[k]);
                if (lane == 0) red[slot][own][part + WPR * k] = s[k];
            }
            __syncthreads();
            tot = red[slot][own][0];
#pragma unroll
            for (int k = 1; k < NR_BLOCK_WARPS; k++) tot += red[slot][own][k];
            return tot;
        }
        float s = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; c++) s += piece[c];
        s = kb_warp_sum(s);
        if (lane == 0) red[slot][own][part] = s;
        __syncthreads();
        tot = red[slot][own][0];
#pragma unroll
        for (int k = 1; k < WPR; k++) tot += red[slot][own][k];
        return tot;
    };
    float piece[NC];
    float mean = 0.0f;
    if (LN) {
#pragma unroll
        for (int c = 0; c < NC; c++) piece[c] = (v[c].x + v[c].y) + (v[c].z + v[c].w);
        mean = row_sum(piece, 0) / (float)E;
    }
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const float a = v[c].x - mean, b = v[c].y - mean, cc = v[c].z - mean, d = v[c].w - mean;
        piece[c] = i0 + STEP * c < E ? (a * a + b * b) + (cc * cc + d * d) : 0.0f;
        v[c] = make_float4(a, b, cc, d);
    }
    const float q = row_sum(piece, 1) / (float)E + eps;
    if (!live) return;
    const float inv = LN ? 1.0f / sqrtf(q) : rsqrtf(q);
    bf16* yr = y + (size_t)t * E;
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const int i = i0 + STEP * c;
        if (i >= E) continue;
        float g[4], o[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
        if (!G4) {
#pragma unroll
            for (int k = 0; k < 4; k++) g[k] = kb_to_f<TW>(w[i + k]);
        } else if (sizeof(TW) == 2) {
            const uint2 r = *(const uint2*)(w + i);
            const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&r.x), b = __bfloat1622float2(*(const __nv_bfloat162*)&r.y);
            g[0] = a.x; g[1] = a.y; g[2] = b.x; g[3] = b.y;
        } else {
            const float4 r = *(const float4*)(w + i);
            g[0] = r.x; g[1] = r.y; g[2] = r.z; g[3] = r.w;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            o[k] = __fmul_rn(__fmul_rn(inv, o[k]), g[k]);
            if (LN) o[k] = __fadd_rn(o[k], kb_to_f<TW>(bias[i + k]));
        }
        __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
        *(uint2*)(yr + i) = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
    }
}

template <typename TW, bool LN, bool G4>
static int norm_rows_of(float* x, const float* delta, int n_delta, size_t stride, const TW* w, const TW* bias, float eps, bf16* y, int T,
                     int E, const TW* ls, cudaStream_t st) {
#define NR_GO(WPR, NC, PB, MINB)                                                                                       \
    return (int)kb_launch(k_norm_rows<TW, WPR, NC, PB, !LN ? NR_RMS : WPR * NC <= 16 ? NR_LN_LANES : NR_LN_BLOCK, MINB, G4>, \
                          (T + 8 / WPR - 1) / (8 / WPR), 256, 0, st, x, delta, n_delta, stride, w, bias, eps, y, T, E, ls)
    if (n_delta <= 1) {
        if (E <= 1024) NR_GO(4, 2, 1, 6);
        if (E <= 2048) NR_GO(4, 4, 1, 4);
        if (E <= 3072) NR_GO(4, 6, 1, 4);
        if (E <= 4096) NR_GO(8, 4, 1, 4);
        NR_GO(8, 6, 1, 4);
    }
    if (E <= 1024) NR_GO(4, 2, 4, 4);
    if (E <= 2048) NR_GO(4, 4, 2, 4);
    if (E <= 3072) NR_GO(4, 6, 2, 2);
    if (E <= 4096) NR_GO(8, 4, 2, 4);
    NR_GO(8, 6, 2, 2);
#undef NR_GO
}

template <typename TW, bool LN>
static int norm_rows(float* x, const float* delta, int n_delta, size_t stride, const TW* w, const TW* bias, float eps, bf16* y, int T,
                     int E, const TW* ls, cudaStream_t st) {
    return ((uintptr_t)w & (sizeof(TW) * 4 - 1)) == 0 ? norm_rows_of<TW, LN, true>(x, delta, n_delta, stride, w, bias, eps, y, T, E, ls, st)
                                                      : norm_rows_of<TW, LN, false>(x, delta, n_delta, stride, w, bias, eps, y, T, E, ls, st);
}

// whether k_norm_rows takes the operands (E up to 6144; x, planes and stride in 16-byte pieces, y in 4 elements)
bool kb_norm_rows_takes(const void* x, const void* delta, int n_delta, long long stride, const void* y, int E) {
    return E % 4 == 0 && E <= 6144 && ((uintptr_t)x & 15) == 0 && (n_delta == 0 || (((uintptr_t)delta & 15) == 0 && stride % 4 == 0)) &&
           ((uintptr_t)y & 7) == 0;
}

int kb_norm_rows(float* x, const float* delta, int n_delta, size_t stride, const void* w, const void* bias, int wdtype, float eps,
                 void* y, int T, int E, const void* ls, bool layer_norm, cudaStream_t st) {
    if (wdtype == KB_F32)
        return layer_norm ? norm_rows<float, true>(x, delta, n_delta, stride, (const float*)w, (const float*)bias, eps, (bf16*)y, T, E, nullptr, st)
                          : norm_rows<float, false>(x, delta, n_delta, stride, (const float*)w, nullptr, eps, (bf16*)y, T, E, (const float*)ls, st);
    return layer_norm ? norm_rows<bf16, true>(x, delta, n_delta, stride, (const bf16*)w, (const bf16*)bias, eps, (bf16*)y, T, E, nullptr, st)
                      : norm_rows<bf16, false>(x, delta, n_delta, stride, (const bf16*)w, nullptr, eps, (bf16*)y, T, E, (const bf16*)ls, st);
}
