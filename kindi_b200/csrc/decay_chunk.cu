// Linear attention with a decay per head over long prompts (key sizes up to 128): a sequence's runs ("chunks") of C tokens
// side by side, as matrix products over tiles of 64 tokens. All arithmetic is 32-bit. Per head with decay w,
//     S_t = w S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t,   q, k, v through silu,
// so with S the state before a chunk and t, s counted inside it:
//     o_t = w^(t+1) S^T q_t + sum_(s <= t) w^(t-s) (q_t . k_s) v_s,       S_end = w^n S + sum_s w^(n-1-s) k_s v_s^T.
//   k_decay_add     what every chunk adds to the state (all chunks side by side; the weight sits on k)
//   k_decay_states  the states before the chunks, in order, and the sequence's new state
//   k_decay_out     the outputs of 64 tokens of a chunk for 64 columns of the state: the state's part, then the chunk's own
//                   keys up to the tokens, tile by tile
// No factor is ever divided out: every power of w has an exponent of at least zero.
// What bounds it are the 32-bit multiply-adds and the phases between them (36 to 42 % of the FMA pipe, shared memory 66 to 69 %).
// The form in its place held a column of the state per thread and made three multiply-adds per state element and token with 12
// warps on an SM: 278 us for 1777 tokens of 16 heads of 128 x 128.
// Here a thread makes 4 x 4 (4 x 8) outputs from 16-byte reads of shared memory, and a token costs two multiply-adds per
// state element and 64 per element of its key and value: 133 us.
#include "common.cuh"
#include "mma_sync.cuh"

#define DQ_T 64                 // tokens of a tile
#define DQ_E 64                 // columns of the state of a block
#define DQ_LV (DQ_T + 4)        // floats between rows of transposed values and of scores (and D + 4: rows of keys): the
                                // eight rows a quarter-warp reads fall into different banks

template <typename TIN>
__device__ __forceinline__ float dq_rd(const TIN* src, int n_planes, size_t plane_stride, size_t i) {
    float v = kb_to_f<TIN>(src[i]);
    for (int s = 1; s < n_planes; s++) v += kb_to_f<TIN>(src[(size_t)s * plane_stride + i]);
    return v;
}
__device__ __forceinline__ float dq_silu(float z) { return __fdividef(z, 1.0f + __expf(-z)); }

// rows r0 .. r0 + n - 1 of 64, columns col .. col + w - 1 of W (zeros elsewhere), through silu; put(row, column, value of
// eight neighbouring columns). vec: rows (and planes) on 16-byte boundaries, w a multiple of 8 (32-bit planes element by
// element: 8192 tokens of 16 heads of 128 x 256 3.92 ms, token by token 3.06, 16 bytes a load 1.46)
template <typename TIN, int W, bool ROW_LANES, typename F>
__device__ __forceinline__ void dq_stage(const TIN* in, int n_planes, size_t plane_stride, int ld_in, int r0, int n, size_t col,
                                         int w, bool vec, F put) {
    constexpr int PIECES = DQ_T * W / 8, PER = (PIECES + 255) / 256;
    constexpr bool HALF = sizeof(TIN) == 2;
    uint4 raw[HALF ? PER : 1];
#pragma unroll
    for (int u = 0; HALF && u < PER; u++) {
        const int e = threadIdx.x + 256 * u, t = ROW_LANES ? e % DQ_T : e / (W / 8), j = (ROW_LANES ? e / DQ_T : e % (W / 8)) * 8;
        raw[u] = make_uint4(0u, 0u, 0u, 0u);
        if (vec && e < PIECES && t < n && j < w) raw[u] = *(const uint4*)((const bf16*)in + (size_t)(r0 + t) * ld_in + col + j);
    }
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int e = threadIdx.x + 256 * u, t = ROW_LANES ? e % DQ_T : e / (W / 8), j = (ROW_LANES ? e / DQ_T : e % (W / 8)) * 8;
        if (e >= PIECES) continue;
        float v[8];
        if (vec && !HALF) {
            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
            if (t < n && j < w) {
                const float* src = (const float*)in + (size_t)(r0 + t) * ld_in + col + j;
                lo = *(const float4*)src;
                hi = *(const float4*)(src + 4);
                for (int s = 1; s < n_planes; s++) {
                    const float4 a = *(const float4*)(src + (size_t)s * plane_stride), b = *(const float4*)(src + (size_t)s * plane_stride + 4);
                    lo = make_float4(lo.x + a.x, lo.y + a.y, lo.z + a.z, lo.w + a.w);
                    hi = make_float4(hi.x + b.x, hi.y + b.y, hi.z + b.z, hi.w + b.w);
                }
            }
            v[0] = dq_silu(lo.x); v[1] = dq_silu(lo.y); v[2] = dq_silu(lo.z); v[3] = dq_silu(lo.w);
            v[4] = dq_silu(hi.x); v[5] = dq_silu(hi.y); v[6] = dq_silu(hi.z); v[7] = dq_silu(hi.w);
        } else if (vec) {
            const __nv_bfloat162* h = (const __nv_bfloat162*)&raw[HALF ? u : 0];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float2 f = __bfloat1622float2(h[c]);
                v[2 * c] = dq_silu(f.x);
                v[2 * c + 1] = dq_silu(f.y);
            }
        } else {
            const TIN* src = in + (size_t)(r0 + t) * ld_in;
#pragma unroll
            for (int c = 0; c < 8; c++)
                v[c] = t < n && j + c < w ? dq_silu(dq_rd<TIN>(src, n_planes, plane_stride, col + j + c)) : 0.0f;
        }
        put(t, j, v);
    }
}

template <bool V> struct DqBool { static constexpr bool value = V; };
struct DqRows {
    int n_planes;
    size_t plane_stride;
    int ld_in, H, d, dv, C, nc_max;
    bool vec_k, vec_v;
};

// P[b, h, chunk][e][j] = sum_s w^(n-1-s) v_s[e] k_s[j]. Grid (B H, blocks of 64 e, chunks)
template <typename TIN, int D>
__global__ void __launch_bounds__(256, 3) k_decay_add(const TIN* KB_STEP_DATA in, const DqRows a, const float* __restrict__ decay,
        const int* __restrict__ q_start, float* __restrict__ P) {
    constexpr int JN = D / 16;
    extern __shared__ __align__(16) float sma[];
    float (*ks)[D] = (float (*)[D])sma;               // [64 t][D]
    float (*vs)[DQ_E] = (float (*)[DQ_E])(sma + DQ_T * D);
    float* lp = sma + DQ_T * (D + DQ_E);              // powers of the decay, 0 .. C
    kb_pdl_launch();
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, c = blockIdx.z, e0 = blockIdx.y * DQ_E;
    const int ra = q_start[b] + c * a.C, n = min(a.C, q_start[b + 1] - ra);
    if (n <= 0) return;
    const float lw = decay[h];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const size_t ok = (size_t)a.H * a.d + (size_t)h * a.d, ov = (size_t)2 * a.H * a.d + (size_t)h * a.dv + e0;
    for (int i = tid; i <= a.C; i += 256) lp[i] = powf(lw, (float)i);
    __syncthreads();
    kb_pdl_wait();
    float acc[4][JN];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < JN; j++) acc[i][j] = 0.0f;
    for (int t0 = 0; t0 < n; t0 += DQ_T) {
        const int m = min(DQ_T, n - t0);
        dq_stage<TIN, D, false>(in, a.n_planes, a.plane_stride, a.ld_in, ra + t0, m, ok, a.d, a.vec_k, [&](int t, int j, const float* v) {
            const float f = t < m ? lp[n - 1 - t0 - t] : 0.0f;
            *(float4*)&ks[t][j] = make_float4(f * v[0], f * v[1], f * v[2], f * v[3]);
            *(float4*)&ks[t][j + 4] = make_float4(f * v[4], f * v[5], f * v[6], f * v[7]);
        });
        dq_stage<TIN, DQ_E, false>(in, a.n_planes, a.plane_stride, a.ld_in, ra + t0, m, ov, a.dv - e0, a.vec_v, [&](int t, int j, const float* v) {
            *(float4*)&vs[t][j] = make_float4(v[0], v[1], v[2], v[3]);
            *(float4*)&vs[t][j + 4] = make_float4(v[4], v[5], v[6], v[7]);
        });
        __syncthreads();
#pragma unroll 4
        for (int t = 0; t < DQ_T; t++) {
            const float4 v4 = *(const float4*)&vs[t][ty * 4];
            const float vv[4] = {v4.x, v4.y, v4.z, v4.w};
            float kk[JN];
#pragma unroll
            for (int g = 0; g < JN / 4; g++) *(float4*)(kk + 4 * g) = *(const float4*)&ks[t][tx * 4 + 64 * g];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < JN; j++) acc[i][j] = fmaf(vv[i], kk[j], acc[i][j]);
        }
        __syncthreads();
    }
    float* dst = P + (((size_t)blockIdx.x * a.nc_max + c) * a.dv + e0) * a.d;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int e = ty * 4 + i;
        if (e0 + e >= a.dv) continue;
#pragma unroll
        for (int g = 0; g < JN / 4; g++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int j = tx * 4 + 64 * g + x;
                if (j < a.d) dst[(size_t)e * a.d + j] = acc[i][4 * g + x];
            }
    }
}

// P[c] (what chunk c adds) becomes the state BEFORE chunk c, element by element, and the slot's state the one after the last
__global__ void __launch_bounds__(256) k_decay_states(int H, int d, int dv, const float* __restrict__ decay,
        const int* __restrict__ q_start, const int* __restrict__ slot, float* KB_STEP_DATA P, float* KB_STEP_DATA state, int C,
        int nc_max) {
    kb_pdl_launch();
    const int b = blockIdx.x / H, h = blockIdx.x % H;
    const int rows = q_start[b + 1] - q_start[b], nc = (rows + C - 1) / C;
    if (nc <= 0) return;
    const float lw = decay[h], wc = powf(lw, (float)C), w_last = powf(lw, (float)(rows - (nc - 1) * C));
    const size_t n = (size_t)dv * d;
    float* own_p = P + (size_t)blockIdx.x * nc_max * n;
    float* srow = state + ((size_t)slot[b] * H + h) * n;
    kb_pdl_wait();
    for (size_t x = (size_t)blockIdx.y * 256 + threadIdx.x; x < n; x += (size_t)gridDim.y * 256) {
        float S = srow[x];
        // (eight chunks' parts are fetched before the first is used: the loads do not wait for one another)
        for (int c0 = 0; c0 < nc; c0 += 8) {
            float own[8];
#pragma unroll
            for (int u = 0; u < 8; u++) own[u] = c0 + u < nc ? own_p[(size_t)(c0 + u) * n + x] : 0.0f;
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (c0 + u < nc) {
                    own_p[(size_t)(c0 + u) * n + x] = S;
                    S = fmaf(c0 + u == nc - 1 ? w_last : wc, S, own[u]);
                }
        }
        srow[x] = S;
    }
}

// Outputs of tile blockIdx.z of a sequence (chunks of C tokens, ceil(C / 64) tiles each), columns e0 .. e0 + 63 of a head
template <typename TIN, int D>
__global__ void __launch_bounds__(256, 2) k_decay_out(const TIN* KB_STEP_DATA in, const DqRows a, const float* __restrict__ decay,
        const int* __restrict__ q_start, const float* KB_STEP_DATA P, float* __restrict__ out, int ldo) {
    constexpr int LK = D + 4;
    extern __shared__ __align__(16) float smd[];
    float* qs = smd;                                  // [64][D + 4]
    float* ks = qs + DQ_T * LK;                       // [64][D + 4]: the state's columns, then tiles of keys
    float* sc = ks + DQ_T * LK;                       // [64 t][64 s + 4]
    float* vt = sc + DQ_T * DQ_LV;                    // [64 e][64 s + 4]
    float* lp = vt + DQ_E * DQ_LV;                    // powers of the decay: 0 .. tokens of a chunk's tiles
    kb_pdl_launch();
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, e0 = blockIdx.y * DQ_E;
    const int per = (a.C + DQ_T - 1) / DQ_T, c = blockIdx.z / per, u = blockIdx.z % per;
    const int rc = q_start[b] + c * a.C, nc_rows = min(a.C, q_start[b + 1] - rc);      // the chunk's rows
    const int n = min(DQ_T, nc_rows - u * DQ_T);                                         // the tile's
    if (n <= 0) return;
    const float lw = decay[h];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const size_t oq = (size_t)h * a.d, ok = (size_t)a.H * a.d + oq, ov = (size_t)2 * a.H * a.d + (size_t)h * a.dv + e0;
    for (int i = tid; i <= per * DQ_T; i += 256) lp[i] = powf(lw, (float)i);
    kb_pdl_wait();
    // in flight beside the queries: the state's columns, and the first tile's keys and values as they came, in the places of
    // the scores and of the transposed values, which are needed only later
    const float* S = P + (((size_t)blockIdx.x * a.nc_max + c) * a.dv + e0) * a.d;
    const bool s_vec = a.d % 4 == 0 && ((uintptr_t)P & 15) == 0, raw = sizeof(TIN) == 2 && a.vec_k && a.vec_v;
    const uint32_t ks_u = (uint32_t)__cvta_generic_to_shared(ks), sc_u = (uint32_t)__cvta_generic_to_shared(sc);
    const uint32_t vt_u = (uint32_t)__cvta_generic_to_shared(vt);
    const int n0 = min(DQ_T, nc_rows);                // rows of the chunk's first tile
    if (s_vec) {
        for (int i = tid; i < DQ_E * (D / 4); i += 256) {
            const int e = i / (D / 4), j = (i % (D / 4)) * 4;
            const bool on = e0 + e < a.dv && j < a.d;
            cp_async16(ks_u + (e * LK + j) * 4, on ? S + (size_t)e * a.d + j : P, on);
        }
    }
    if (raw) {
        for (int i = tid; i < DQ_T * (D / 8); i += 256) {
            const int t = i / (D / 8), j = (i % (D / 8)) * 8;
            const bool on = t < n0 && j < a.d;
            cp_async16(sc_u + i * 16, on ? in + (size_t)(rc + t) * a.ld_in + ok + j : in, on);
        }
        for (int i = tid; i < DQ_T * (DQ_E / 8); i += 256) {
            const int t = i % DQ_T, j = (i / DQ_T) * 8;      // (neighbouring lanes: neighbouring tokens, see below)
            const bool on = t < n0 && e0 + j < a.dv;
            cp_async16(vt_u + i * 16, on ? in + (size_t)(rc + t) * a.ld_in + ov + j : in, on);
        }
    }
    dq_stage<TIN, D, false>(in, a.n_planes, a.plane_stride, a.ld_in, rc + u * DQ_T, n, oq, a.d, a.vec_k, [&](int t, int j, const float* v) {
        *(float4*)(qs + t * LK + j) = make_float4(v[0], v[1], v[2], v[3]);
        *(float4*)(qs + t * LK + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
    });
    if (!s_vec) {
        for (int i = tid; i < DQ_E * D; i += 256) {
            const int e = i / D, j = i % D;
            ks[e * LK + j] = e0 + e < a.dv && j < a.d ? S[(size_t)e * a.d + j] : 0.0f;
        }
    }
    cp_async_wait_all();
    __syncthreads();
    float o[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) o[i][j] = 0.0f;
    // 4 x 4 sums over D of rows ty + 16 i of qs and tx + 16 j of ks (`low`: only the pairs with j <= i)
    auto dots = [&](float (&r)[4][4], auto low) {
#pragma unroll 4
        for (int k = 0; k < D; k += 4) {
            float4 q4[4], k4[4];
#pragma unroll
            for (int i = 0; i < 4; i++) q4[i] = *(const float4*)(qs + (ty + 16 * i) * LK + k);
#pragma unroll
            for (int j = 0; j < 4; j++) k4[j] = *(const float4*)(ks + (tx + 16 * j) * LK + k);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (!decltype(low)::value || j <= i) {
                        r[i][j] = fmaf(q4[i].x, k4[j].x, r[i][j]);
                        r[i][j] = fmaf(q4[i].y, k4[j].y, r[i][j]);
                        r[i][j] = fmaf(q4[i].z, k4[j].z, r[i][j]);
                        r[i][j] = fmaf(q4[i].w, k4[j].w, r[i][j]);
                    }
        }
    };
    dots(o, DqBool<false>());
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float f = lp[u * DQ_T + ty + 16 * i + 1];
#pragma unroll
        for (int j = 0; j < 4; j++) o[i][j] *= f;
    }
    for (int us = 0; us <= u; us++) {
        const bool diag = us == u;
        const int ns = min(DQ_T, nc_rows - us * DQ_T);
        float probe = 0.0f;                           // stays zero while this thread's values are finite
        if (us == 0 && raw) {
            uint4 rk[DQ_T * D / 8 / 256], rv[DQ_T * DQ_E / 8 / 256];
#pragma unroll
            for (int x = 0; x < DQ_T * D / 8 / 256; x++) rk[x] = ((const uint4*)sc)[tid + 256 * x];
#pragma unroll
            for (int x = 0; x < DQ_T * DQ_E / 8 / 256; x++) rv[x] = ((const uint4*)vt)[tid + 256 * x];
            __syncthreads();                          // everybody has read the state and the raw rows
#pragma unroll
            for (int x = 0; x < DQ_T * D / 8 / 256; x++) {
                const int i = tid + 256 * x, t = i / (D / 8), j = (i % (D / 8)) * 8;
                const __nv_bfloat162* h2 = (const __nv_bfloat162*)&rk[x];
                float v[8];
#pragma unroll
                for (int y = 0; y < 4; y++) {
                    const float2 f = __bfloat1622float2(h2[y]);
                    v[2 * y] = dq_silu(f.x);
                    v[2 * y + 1] = dq_silu(f.y);
                }
                *(float4*)(ks + t * LK + j) = make_float4(v[0], v[1], v[2], v[3]);
                *(float4*)(ks + t * LK + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
            }
#pragma unroll
            for (int x = 0; x < DQ_T * DQ_E / 8 / 256; x++) {
                const int i = tid + 256 * x, t = i % DQ_T, j = (i / DQ_T) * 8;
                const __nv_bfloat162* h2 = (const __nv_bfloat162*)&rv[x];
#pragma unroll
                for (int y = 0; y < 4; y++) {
                    const float2 f = __bfloat1622float2(h2[y]);
                    const float v0 = dq_silu(f.x), v1 = dq_silu(f.y);
                    vt[(j + 2 * y) * DQ_LV + t] = v0;
                    vt[(j + 2 * y + 1) * DQ_LV + t] = v1;
                    probe = fmaf(v0, 0.0f, fmaf(v1, 0.0f, probe));
                }
            }
        } else {
            __syncthreads();                              // the state, or the tile before, has been read
            dq_stage<TIN, D, false>(in, a.n_planes, a.plane_stride, a.ld_in, rc + us * DQ_T, ns, ok, a.d, a.vec_k,
                                    [&](int t, int j, const float* v) {
                                        *(float4*)(ks + t * LK + j) = make_float4(v[0], v[1], v[2], v[3]);
                                        *(float4*)(ks + t * LK + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
                                    });
            // (neighbouring lanes take neighbouring tokens, so that the transposed stores fall into different banks)
            dq_stage<TIN, DQ_E, true>(in, a.n_planes, a.plane_stride, a.ld_in, rc + us * DQ_T, ns, ov, a.dv - e0, a.vec_v,
                                      [&](int t, int j, const float* v) {
#pragma unroll
                                          for (int x = 0; x < 8; x++) {
                                              vt[(j + x) * DQ_LV + t] = v[x];
                                              probe = fmaf(v[x], 0.0f, probe);
                                          }
                                      });
        }
        const bool odd = __syncthreads_or(!(probe == 0.0f));
        float s4[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s4[i][j] = 0.0f;
        if (diag) dots(s4, DqBool<true>());
        else dots(s4, DqBool<false>());
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int t = ty + 16 * i, s = tx + 16 * j, gap = (u - us) * DQ_T + t - s;
                sc[t * DQ_LV + s] = gap >= 0 ? s4[i][j] * lp[gap] : 0.0f;
            }
        __syncthreads();
        if (diag && odd) {
            // A value that is no number or infinite: 0 x infinity would carry it into tokens before it (the scores above the
            // diagonal are zeros), so every later token is left out. The same sums in the same order. (Leaving them out always
            // made the three kernels 3.5 % slower over 162 shapes, this check 0 %.)
#pragma unroll 1
            for (int s = 0; s < DQ_T; s++) {
                float v1[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v1[j] = vt[(tx + 16 * j) * DQ_LV + s];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float p = sc[(ty + 16 * i) * DQ_LV + s];
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (s <= ty + 16 * i) o[i][j] = fmaf(p, v1[j], o[i][j]);
                }
            }
            continue;
        }
#pragma unroll
        for (int sb = 0; sb < 4; sb++)
#pragma unroll
            for (int s = sb * 16; s < sb * 16 + 16; s += 4) {
                float4 v4[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v4[j] = *(const float4*)(vt + (tx + 16 * j) * DQ_LV + s);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (diag && i < sb) continue;     // (scores above the diagonal)
                    const float4 p = *(const float4*)(sc + (ty + 16 * i) * DQ_LV + s);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        o[i][j] = fmaf(p.x, v4[j].x, o[i][j]);
                        o[i][j] = fmaf(p.y, v4[j].y, o[i][j]);
                        o[i][j] = fmaf(p.z, v4[j].z, o[i][j]);
                        o[i][j] = fmaf(p.w, v4[j].w, o[i][j]);
                    }
                }
            }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = ty + 16 * i;
        if (t >= n) continue;
        float* orow = out + (size_t)(rc + u * DQ_T + t) * ldo + (size_t)h * a.dv + e0;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (e0 + tx + 16 * j < a.dv) orow[tx + 16 * j] = o[i][j];
    }
}

template <typename TIN, int D>
static int launch_decay(const TIN* in, const DqRows& a, int B, const float* decay, const int* q_start, const int* slot,
                        float* state, float* P, float* out, int ldo, cudaStream_t st) {
    const int eb = (a.dv + DQ_E - 1) / DQ_E, per = (a.C + DQ_T - 1) / DQ_T;
    const size_t smem_add = (size_t)(DQ_T * (D + DQ_E) + a.C + 1) * sizeof(float);
    const size_t smem = (size_t)(2 * DQ_T * (D + 4) + 2 * DQ_T * DQ_LV + per * DQ_T + 1) * sizeof(float);
    cudaError_t e;
    static char once_tag;
    if (kb_first_use(&once_tag)) {
        e = cudaFuncSetAttribute(k_decay_add<TIN, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_decay_out<TIN, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
    }
    kb_launch(k_decay_add<TIN, D>, dim3(B * a.H, eb, a.nc_max), 256, smem_add, st, in, a, decay, q_start, P);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    const int sb = (a.dv * a.d + 255) / 256;
    kb_launch(k_decay_states, dim3(B * a.H, sb < 64 ? sb : 64), 256, 0, st, a.H, a.d, a.dv, decay, q_start, slot, P, state, a.C,
              a.nc_max);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    kb_launch(k_decay_out<TIN, D>, dim3(B * a.H, eb, a.nc_max * per), 256, smem, st, in, a, decay, q_start, (const float*)P, out,
              ldo);
    KB_LAUNCH_RET();
}

// whether the tiles take chunks of C tokens, at most nc_max of them a sequence: grids and shared memory (the powers of the decay)
bool kb_decay_tiles_takes(int d, int C, int nc_max) {
    const long long per = (C + DQ_T - 1) / DQ_T, D = d <= 64 ? 64 : 128;
    return d <= 128 && nc_max * per <= 65535 && (DQ_T * (D + DQ_E) + C + 1) * 4 <= 227 * 1024 &&
           (2 * DQ_T * (D + 4) + 2 * DQ_T * DQ_LV + per * DQ_T + 1) * 4 <= 227 * 1024;
}

// P: float [B][H][nc_max][dv][d]
int kb_decay_tiles(const void* in, int in_dtype, int n_planes, size_t plane_stride, int ld_in, int B, int H, int d, int dv,
                   const float* decay, const int* q_start, const int* slot, float* state, float* P, float* out, int ldo, int C,
                   int nc_max, cudaStream_t st) {
    DqRows a{n_planes, plane_stride, ld_in, H, d, dv, C, nc_max, false, false};
    if (!kb_decay_tiles_takes(d, C, nc_max)) return (int)cudaErrorInvalidValue;
    const int piece = in_dtype == KB_BF16 ? 8 : 4;    // elements of 16 bytes
    if ((in_dtype == KB_F32 || n_planes == 1) && ld_in % piece == 0 && plane_stride % piece == 0 && ((uintptr_t)in & 15) == 0 && d % 8 == 0) {
        a.vec_k = true;
        a.vec_v = dv % 8 == 0;
    }
    if (in_dtype == KB_F32)
        return d <= 64 ? launch_decay<float, 64>((const float*)in, a, B, decay, q_start, slot, state, P, out, ldo, st)
                       : launch_decay<float, 128>((const float*)in, a, B, decay, q_start, slot, state, P, out, ldo, st);
    return d <= 64 ? launch_decay<bf16, 64>((const bf16*)in, a, B, decay, q_start, slot, state, P, out, ldo, st)
                   : launch_decay<bf16, 128>((const bf16*)in, a, B, decay, q_start, slot, state, P, out, ldo, st);
}
