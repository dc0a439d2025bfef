/*
 * The packed denoise with a temporal history, in two kernels (the
 * reference's denoise_nlm pass; CPU definition lib/ref/ref_denoise.c:168-336).
 *
 * k_dn_temporal   the temporal recursive average of every sample, once: the
 *   stabilised value T and the variance left V, as FP32 planes with an apron
 *   of the search's and patch's radius all around, and the next state. A
 *   tile that formed them itself would form its apron's as well, twice the
 *   samples of its output at over a hundred instructions each.
 * k_dn_history    the non-local means of one tile of the four planes, whose
 *   T and V arrive as two TMA tile copies, ready for the search.
 *
 * Bounds: k_dn_temporal instruction issue (136 instructions a sample, three
 * correctly rounded roots and an exponential among them; 72 % of the issue
 * slots, 3.4 TB/s); k_dn_history the FMA pipe, as the spatial search.
 *
 * The apron holds the value of the position its own 3x3 window mirrors to,
 * window by window, so that a sum of squares there adds in the mirrored
 * order; the tiles need no borders.
 */
#pragma once

#include "denoise_tile.cuh"

namespace craw_dn {

constexpr int HR = S + P;            /* the apron */

/* The planes' layout: w x h floats a plane, four planes of T, then of V.
 * Whole 32 x 16 tiles and the apron; rows of a multiple of 32 bytes. */
struct HistPlanes {
    int w, h;
    size_t n;                        /* floats a plane */
    __host__ __device__ HistPlanes(int pw, int ph)
        : w((pw + 31) / 32 * 32 + 2 * HR), h((ph + 15) / 16 * 16 + 2 * HR), n((size_t)w * h)
    {
    }
};

/* ------------------------------------------------------ temporal average */

/* A walking warp: mosaic rows of one parity, two planes; a lane owns two
 * columns of each (four mosaic columns), keeps the last plane rows' squared
 * differences in registers and takes its neighbours' by shuffle. Output
 * lanes 1 .. 30. */
constexpr int TW_N = 30, TW_WARPS = 4, TW_NT = 32 * TW_WARPS, TW_CTAS = 8;

struct TemporalGrid {
    int nx, seg, rows;               /* strips across; plane rows a segment; plane rows in all */
};

CRAW_DEV void temporal_walk(const CRAWKDenoise &k, const CRAWKDenoiseIO &io, float *tv, const TemporalGrid &g, int wid,
                            uint32_t *err)
{
    const int lane = threadIdx.x & 31, py = wid & 1, sx = (wid >> 1) % g.nx, sy = (wid >> 1) / g.nx;
    if (sy * g.seg >= g.rows)
        return;
    const HistPlanes P(k.pw, k.ph);
    /* Plane columns c, c + 1 and rows r0 .. r0 + n - 1, of the padded planes
     * (0 is the apron's first). */
    const int c = 2 * (sx * TW_N - 1 + lane), r0 = sy * g.seg, n = min(g.seg, g.rows - r0);
    const bool mine = lane >= 1 && lane <= TW_N && c < k.pw + 2 * HR;
    const int m0 = craw_mirror(c - HR, k.pw), m1 = craw_mirror(c + 1 - HR, k.pw);
    const float black[2] = { py ? k.black[2] : k.black[0], py ? k.black[3] : k.black[1] };
    const float irng[2] = { py ? k.inv_range[2] : k.inv_range[0], py ? k.inv_range[3] : k.inv_range[1] };

    struct Raw {
        uint32_t raw[2];
        float2 lvl[2];
        uint32_t var[2];
    };
    auto fetch = [&](int r) {
        Raw t;
        const int y = 2 * craw_mirror(r - HR, k.ph) + py;
        const char *src = (const char *)io.src + (size_t)y * io.src_pitch;
        const char *lvl = (const char *)io.lvl_prev + (size_t)y * io.lvl_pitch;
        const char *var = (const char *)io.var_prev + (size_t)y * io.var_pitch;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int m = i ? m1 : m0;
            t.raw[i] = 0u;
            t.lvl[i] = make_float2(0.0f, 0.0f);
            t.var[i] = 0u;
            if (craw_in_bounds(m >= 0 && m < k.pw && y >= 0 && y < 2 * k.ph, err)) {
                t.raw[i] = __ldg(reinterpret_cast<const uint32_t *>(src) + m);
                t.lvl[i] = __ldg(reinterpret_cast<const float2 *>(lvl) + m);
                t.var[i] = __ldg(reinterpret_cast<const uint16_t *>(var) + m);
            }
        }
        return t;
    };
    /* A row's stabilised values (this frame's, the last level's) and its
     * 3-wide row sums of squared differences (the same nine terms a window
     * as the reference's sum, as rows of three and then three rows). Sample
     * i: column c + i / 2 of the plane of column parity i & 1. */
    auto take = [&](const Raw &t, float cur[4], float prev[4], float hs[4]) {
        float sq[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t raw = i & 1 ? t.raw[i >> 1] >> 16 : t.raw[i >> 1] & 0xffffu;
            cur[i] = gat_fwd(k, ((float)raw * (1.0f / 65535.0f) - black[i & 1]) * irng[i & 1]);
            prev[i] = gat_fwd(k, i & 1 ? t.lvl[i >> 1].y : t.lvl[i >> 1].x);
            const float e = prev[i] - cur[i];
            sq[i] = __fmul_rn(e, e);
        }
        const float l0 = __shfl_up_sync(0xffffffffu, sq[2], 1), l1 = __shfl_up_sync(0xffffffffu, sq[3], 1);
        const float q0 = __shfl_down_sync(0xffffffffu, sq[0], 1), q1 = __shfl_down_sync(0xffffffffu, sq[1], 1);
        hs[0] = __fadd_rn(__fadd_rn(l0, sq[0]), sq[2]);
        hs[1] = __fadd_rn(__fadd_rn(l1, sq[1]), sq[3]);
        hs[2] = __fadd_rn(__fadd_rn(sq[0], sq[2]), q0);
        hs[3] = __fadd_rn(__fadd_rn(sq[1], sq[3]), q1);
    };

    float cur[4], prev[4], h0[4], h1[4];
    uint32_t var;
    Raw raw;
    {
        const Raw a = fetch(r0 - 1), b = fetch(r0);
        raw = fetch(r0 + 1);
        take(a, cur, prev, h0);
        take(b, cur, prev, h1);
        var = b.var[0] | b.var[1] << 16;
    }
#pragma unroll 1
    for (int r = r0; r < r0 + n; r++) {
        float c2[4], p2[4], h2[4], t[4], v[4];
        const uint32_t var2 = raw.var[0] | raw.var[1] << 16;
        take(raw, c2, p2, h2);
        raw = fetch(r + 2);
        /* Row r. */
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float d2 = __fadd_rn(__fadd_rn(h0[i], h1[i]), h2[i]);
            float x = d2 * (1.0f / 9.0f) * k.t_inv_h2 - 2.0f;
            float a = k.t_alpha * expf(-fmaxf(x, 0.0f));
            float sp = (float)((var >> (8 * i)) & 0xffu) * (1.0f / 255.0f);
            float vv = __fadd_rn(__fmul_rn(1.0f - a, 1.0f - a), __fmul_rn(a * a, sp * sp));
            t[i] = __fadd_rn(__fmul_rn(cur[i], 1.0f - a), __fmul_rn(prev[i], a));
            v[i] = fmaxf(vv, kVarMin);
        }
        if (mine) {
            float *at = tv + (size_t)(2 * py) * P.n + (size_t)r * P.w + c;
            if (craw_in_bounds(r >= 0 && r < P.h && c >= 0 && c + 1 < P.w, err)) {
                *reinterpret_cast<float2 *>(at) = make_float2(t[0], t[2]);
                *reinterpret_cast<float2 *>(at + P.n) = make_float2(t[1], t[3]);
                *reinterpret_cast<float2 *>(at + 4 * P.n) = make_float2(v[0], v[2]);
                *reinterpret_cast<float2 *>(at + 5 * P.n) = make_float2(v[1], v[3]);
            }
            const int qx = c - HR, qy = r - HR;
            if (qy >= 0 && qy < k.ph) {
                float *lr = (float *)((char *)io.lvl_next + (size_t)(2 * qy + py) * io.lvl_pitch);
                uint8_t *vr = io.var_next + (size_t)(2 * qy + py) * io.var_pitch;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (qx + j < 0 || qx + j >= k.pw ||
                        !craw_in_bounds((size_t)(qx + j + 1) * 8 <= io.lvl_pitch &&
                                        (size_t)(qx + j + 1) * 2 <= io.var_pitch, err))
                        continue;
                    reinterpret_cast<float2 *>(lr)[qx + j] = make_float2(gat_inv(k, t[2 * j]), gat_inv(k, t[2 * j + 1]));
                    uint32_t code = 0;
#pragma unroll
                    for (int i = 0; i < 2; i++)
                        code |= (uint32_t)(uint8_t)rintf(sqrtf(fminf(fmaxf(v[2 * j + i], 0.0f), 1.0f)) * 255.0f)
                                << (8 * i);
                    reinterpret_cast<uint16_t *>(vr)[qx + j] = (uint16_t)code;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            cur[i] = c2[i];
            prev[i] = p2[i];
            h0[i] = h1[i];
            h1[i] = h2[i];
        }
        var = var2;
    }
}

/* ------------------------------------------------------ non-local means */

struct HistCfg {
    static constexpr int M = 8, WP = 1;                  /* a thread's rows, warps a plane */
    static constexpr int OX = 32, OY = 2 * M * WP;       /* plane samples per tile */
    static constexpr int TX = OX + 2 * HR, TY = OY + 2 * HR, TS = TX, TN = TY * TS;
    static constexpr int NT = 4 * WP * 32;
    static constexpr uint32_t BYTES = 4 * TN * sizeof(float);   /* of T, and of V */
    static constexpr int RW_W = 2 * OX, RW_H = 2 * OY;
    /* T (then the tile's output), V, T's copy shifted left by one sample,
     * log2(e) over the centres' variance; and room to align it all to 128
     * bytes: 54 KB, four CTAs an SM. */
    static constexpr int LV_OFF = 12 * TN;
    static constexpr int smem_floats = LV_OFF + 4 * OX * OY + 32;
    static_assert(BYTES % 128 == 0 && TS * sizeof(float) % 16 == 0, "tile copies");
    static_assert(OX == 32 && OY == 16, "the planes are padded to these tiles");
};

CRAW_DEV void history_tile(const CRAWKDenoise &k, const CRAWKDenoiseIO &io, const float *tv, bool tma,
                           const CUtensorMap *tmap_t, const CUtensorMap *tmap_v, int bx, int by, float *smem,
                           uint32_t *err)
{
    using C = HistCfg;
    constexpr int M = C::M, WP = C::WP, TN = C::TN, TS = C::TS, NT = C::NT;
    float *T = smem, *V = smem + 4 * TN, *To = smem + 8 * TN;
    const int tid = threadIdx.x, tx0 = bx * C::OX, ty0 = by * C::OY;
    const int W = 2 * k.pw, H = 2 * k.ph, mx0 = 2 * tx0, my0 = 2 * ty0;
    __shared__ __align__(8) uint64_t bar;
    if (tma) {
        craw_tma::bar_init(&bar);
        if (tid == 0)
            craw_tma::load_3d2(T, tmap_t, V, tmap_v, tx0, ty0, 0, &bar, 2 * C::BYTES);
    }
    if (tma) {
        if (!__syncthreads_and(craw_tma::wait(&bar, 0))) {
            /* Never expected: record it, give the copies one more bound to
             * land before the CTA leaves, and skip the tile. */
            if (tid == 0 && err)
                atomicOr(err, CRAW_K_ERR_TMA_WAIT);
            (void)craw_tma::wait(&bar, 0);
            return;
        }
    } else {
        const HistPlanes P(k.pw, k.ph);
        for (int i = tid; i < 8 * TN / 4; i += NT) {
            const int a = i / TN, e = 4 * (i % TN);        /* T or V; the element of its four planes */
            const int pl = e / TN, y = e % TN / TS, x = e % TS;
            if (craw_in_bounds(a < 2 && pl < 4 && ty0 + y < P.h && tx0 + x + 3 < P.w, err))
                reinterpret_cast<float4 *>(T)[i] = *reinterpret_cast<const float4 *>(
                    tv + (size_t)(4 * a + pl) * P.n + (size_t)(ty0 + y) * P.w + tx0 + x);
        }
        __syncthreads();
    }
    for (int i = tid; i < 4 * TN - 1; i += NT)
        To[i] = T[i + 1];
    const int warp = tid >> 5, lane = tid & 31;
    const int pl = warp / WP, band = warp % WP;
    const int ox0 = (lane & 15) * 2, oy0 = ((band << 1) | (lane >> 4)) * M;
    float *lvc = smem + C::LV_OFF + (pl * C::OY + oy0) * C::OX + ox0;   /* the thread's own */
#pragma unroll
    for (int m = 0; m < M; m++) {
        const f2x v = f2_ld(V + pl * TN + (oy0 + HR + m) * TS + ox0 + HR);
        *reinterpret_cast<float2 *>(lvc + m * C::OX) =
            make_float2(__fdiv_rn(kLog2e, f2_lo(v)), __fdiv_rn(kLog2e, f2_hi(v)));
    }
    __syncthreads();

    SearchRows<HR, TS, true, 8 * TN, 4 * TN, C::OX> st;
    st.init(k.inv_h2);
#pragma unroll 1
    for (int dy = -S; dy <= S; dy++)
        st.step_dy(T + pl * TN + oy0 * TS + ox0, lvc, dy);

    /* The codes, over T once every warp has searched it. */
    const int px = pl & 1, py = pl >> 1;
    const float blk = pick4(k.black, pl), irng = pick4(k.inv_range, pl), rng = pick4(k.range, pl);
    uint16_t *out16 = reinterpret_cast<uint16_t *>(T);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int my = my0 + 2 * (oy0 + m) + py, mx = mx0 + 2 * (ox0 + j) + px;
            uint16_t raw0 = 0;
            if (my < H && mx < W && craw_in_bounds(my >= 0 && mx >= 0, err))
                raw0 = __ldg((const uint16_t *)((const char *)io.src + (size_t)my * io.src_pitch) + mx);
            const float res = j ? __fdiv_rn(f2_hi(st.acc[m]), f2_hi(st.wsum[m]))
                                : __fdiv_rn(f2_lo(st.acc[m]), f2_lo(st.wsum[m]));
            out16[(2 * (oy0 + m) + py) * C::RW_W + 2 * (ox0 + j) + px] =
                (uint16_t)rintf(encode(k, gat_inv(k, res), raw0, blk, irng, rng));
        }
    __syncthreads();
    constexpr int CH = C::RW_W / 8;
    const bool a16 = !(((uintptr_t)io.dst | io.dst_pitch) & 15);
    for (int i = tid; i < C::RW_H * CH; i += NT) {
        const int yy = i / CH, my = my0 + yy, mx = mx0 + (i % CH) * 8;
        if (my >= H || mx >= W || !craw_in_bounds(my >= 0 && mx >= 0 && yy < C::RW_H, err))
            continue;
        uint16_t *dr = (uint16_t *)((char *)io.dst + (size_t)my * io.dst_pitch) + mx;
        if (a16 && mx + 8 <= W) {
            *reinterpret_cast<uint4 *>(dr) = reinterpret_cast<const uint4 *>(out16)[i];
        } else {
            for (int e = 0; e < 8 && mx + e < W; e++)
                dr[e] = out16[8 * i + e];
        }
    }
}

} // namespace craw_dn
