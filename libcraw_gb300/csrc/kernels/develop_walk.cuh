/*
 * The develop stage by walking warps: a warp owns a strip of quad columns,
 * one column a lane, and walks down a segment of it one quad row (two
 * pixel rows) a step. What a column needs of its neighbours comes by warp
 * shuffles and what it needs of earlier rows stays in registers, so a step
 * has no barrier, no shared-memory ring and no index arithmetic beyond its
 * row pointers. The epilogue (intermediate, colour stage, stores, AWB
 * statistic) takes the quad's four pixels from the lane's registers.
 *
 * A strip has NQ output columns on lanes A .. A + NQ - 1; the lanes outside
 * them are the strip's apron and compute values that only their inner
 * neighbours read.
 *
 * Bound: instruction issue. The RCD takes 555 warp instructions a step of
 * 24 quads (110 M at 5760x3240, 74 % of the issue slots busy, 128 us), where
 * a column-a-thread kernel that passed its rows through shared-memory rings
 * between two barriers a step took 156 M (173 us) and 64x16 tiles 204 M
 * (233 us with the gamut compression, 140 us here): a third to a half of
 * their instructions were ring and tile addressing and the tiles' aprons.
 * Two steps a round of the loop halve the moves from one step's registers
 * to the next's; four (100 M instructions) wait longer on the spills and
 * loads than they save.
 */
#pragma once

#include <string.h>

#include "develop_tile.cuh"

namespace craw_dev {

/* The frame's part the strips cover, in quads: columns qx0 .. qx0 + nqx,
 * rows qy0 .. qy0 + nqy, in segments of `seg` rows a warp, `nx` strips
 * across. qx0, qy0 and a strip's output columns are multiples of 4, and seg
 * of what walk_unit() says, so that strips and segments start on 8x8 AWB
 * blocks (4x4 blocks of the chroma path) where a frame has them. */
struct WalkGrid {
    int qx0, nqx, qy0, nqy, seg, nx;
};

constexpr int WALK_WARPS = 4, WALK_NT = 32 * WALK_WARPS;   /* warps (strips) a CTA */

/* The quad rows that a segment is a multiple of: whole AWB blocks, or whole
 * blocks of the chroma path. */
inline int walk_unit(const CRAWKDevelopIO &io, int least)
{
    return io.awb.hist ? 4 : (io.quarter ? 2 : least);
}

/* Segments of one wave of `ctas` CTAs an SM: as tall as that allows (a
 * segment reads, and for the RCD computes, its first rows' surroundings
 * again), a multiple of `unit` quad rows; g.nx strips are set. Returns the
 * CTAs. */
inline unsigned walk_segments(WalkGrid &g, int sms, int ctas, int unit)
{
    const int room = sms * ctas * WALK_WARPS / g.nx;
    const int nseg = room > 1 ? room : 1;
    g.seg = unit * (((g.nqy + unit - 1) / unit + nseg - 1) / nseg);
    const int warps = g.nx * ((g.nqy + g.seg - 1) / g.seg);
    return (unsigned)((warps + WALK_WARPS - 1) / WALK_WARPS);
}

CRAW_DEV float walk_left(float v)    /* the left neighbour's v */
{
    return __shfl_up_sync(0xffffffffu, v, 1);
}
CRAW_DEV float walk_right(float v)
{
    return __shfl_down_sync(0xffffffffu, v, 1);
}

/* A row's sample pair, a step before it is used: volatile, so that the load
 * stays where it is written; not by the read-only path, since the kernel
 * that writes the row may still run when this one starts. */
CRAW_DEV uint32_t walk_ld(const char *p)
{
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

/* Bytes of a pixel of an RGB image of layout f. */
CRAW_DEV int walk_bytes(int f)
{
    return f == CRAW_K_OUT_RGB32F ? 12 : (f == CRAW_K_OUT_RGBA16F ? 8 : 16);
}

/* Eight floats to a 32-byte aligned address in one store. */
CRAW_DEV void walk_store8(float *p, float a, float b, float c, float d, float e, float f, float g, float h)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d), "f"(e), "f"(f), "f"(g), "f"(h) : "memory");
}

/* The colour stage of four pixels of a lane (craw_color; RGC: with the
 * gamut compression, without it, or -1: by its flag), the gamut compression
 * a channel at a time for all four, where any lane's pixel needs it:
 * branch-free, so the four chains interleave. The test for it needs no
 * division: a distance clearly below its threshold, beyond any rounding of
 * the compression's own reciprocal, leaves the channel alone. (A pixel at a
 * time with a branch a channel: 5760x3240 AP1 284 us a frame, against 197
 * this way and 174 without the compression.) The whole warp calls this;
 * `mine`: the lane's pixels count. */
template <int RGC>
CRAW_DEV void walk_colour(const CRAWKColor &c, bool mine, float o[4][3])
{
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float in[3] = { o[i][0], o[i][1], o[i][2] };
#pragma unroll
        for (int r = 0; r < 3; r++)
            o[i][r] = c.m[r][0] * in[0] + c.m[r][1] * in[1] + c.m[r][2] * in[2];
    }
    if (RGC < 0 ? (c.flags & CRAW_K_COLOR_RGC) != 0 : RGC) {
        float ach[4];
        bool need[3] = { false, false, false };
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ach[i] = fmaxf(o[i][0], fmaxf(o[i][1], o[i][2]));
            const float mag = fabsf(ach[i]) * (1.0f - 1e-6f);
#pragma unroll
            for (int r = 0; r < 3; r++)
                need[r] |= !(ach[i] - o[i][r] < c.gc_thr[r] * mag);
        }
        if (__any_sync(0xffffffffu, mine && (need[0] || need[1] || need[2]))) {
            float inv[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                inv[i] = craw_rcp(fabsf(ach[i]));
#pragma unroll
            for (int r = 0; r < 3; r++) {
                if (!__any_sync(0xffffffffu, mine && need[r]))
                    continue;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float y = craw_gamut_channel(c, r, ach[i], fabsf(ach[i]), inv[i], o[i][r]);
                    o[i][r] = ach[i] == 0.0f ? o[i][r] : y;
                }
            }
        }
    }
    if (c.flags & CRAW_K_COLOR_CLAMP) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int r = 0; r < 3; r++)
                o[i][r] = fmaxf(o[i][r], 0.0f);
    }
}

/* Shared memory of one warp: the camera RGB of the AWB block row in
 * progress (eight pixel rows, planar a row: 4 floats of padding after 32
 * spread the blocks a fold reads over the banks), and the sums of the
 * blocks that wait for their statistic. */
template <int NQ>
struct WalkSmem {
    static constexpr int PW = 2 * NQ, PITCH = PW + 4 * ((PW - 1) / 32);
    static constexpr int NB = NQ / 4, HOLD = 32 / NB;      /* blocks a row; block rows held */
    alignas(16) float a[8][3][PITCH];
    float sum[HOLD * NB][3];
    float cnt[HOLD * NB];
    CRAW_DEV static int col(int x) { return x + 4 * (x >> 5); }
};

/* The epilogue of one warp: takes the camera RGB of the four pixels of each
 * lane's quad, a quad row at a time. FMT (a CRAW_K_OUT_* layout), RGC (the
 * gamut compression: with it, without, or -1 by its flag): fixed per kernel, so that a step's code stays small
 * enough for the instruction cache; MORE: any layout, FP16 storage, the
 * kept intermediate and the chroma path's block means, by tests. */
template <int NQ, int A, int FMT, int RGC, bool MORE>
struct WalkOut {
    using S = WalkSmem<NQ>;
    const CRAWKDevelop &k;
    const CRAWKDevelopIO &io;
    S &s;
    int lane, nout;          /* the strip's output columns (a multiple of 4 but at the frame's right edge) */
    int qx, qy;              /* the strip's first output quad, the segment's first quad row */
    bool mine;               /* the lane has an output column */
    int held;                /* AWB blocks waiting for their statistic */
    char *dst, *inter;       /* the row pair to store next: the strip's first pixel */
    float qs[3];             /* chroma: this lane's 4x4 block sums */

    CRAW_DEV WalkOut(const CRAWKDevelop &k_, const CRAWKDevelopIO &io_, S &s_, int nout_, int qx_, int qy_)
        : k(k_), io(io_), s(s_), lane(threadIdx.x & 31), nout(nout_), qx(qx_), qy(qy_), held(0)
    {
        mine = lane >= A && lane < A + nout;
        dst = (char *)io.dst + (size_t)(2 * qy) * io.dst_pitch + (size_t)(2 * qx) * walk_bytes(fmt());
        inter = (char *)io.inter + (size_t)(2 * qy) * io.inter_pitch +
                (size_t)(2 * qx) * (k.fp16 ? 8 : 16);
        qs[0] = qs[1] = qs[2] = 0.0f;
    }
    CRAW_DEV int fmt() const { return MORE ? io.dst_fmt : FMT; }

    CRAW_DEV void colour(const float v[2][2][3], float o[2][2][3]) const
    {
        float q[4][3];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                q[i][c] = v[i >> 1][i & 1][c];
        walk_colour<RGC>(k.color, mine, q);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                o[i >> 1][i & 1][c] = q[i][c];
    }

    /* A row pair of an RGB image of layout `f` from `at` (the strip's first
     * pixel of it), two pixels a lane and row: v[row][pixel][channel]. */
    CRAW_DEV void store(char *at, size_t pitch, int f, int r, const float v[2][2][3])
    {
        const bool ok = craw_in_bounds(qx >= 0 && 2 * (qx + nout) <= k.width && 2 * (qy + r) >= 0 &&
                                       2 * (qy + r) + 1 < k.height, io.err);
        if (f == CRAW_K_OUT_RGB32F) {
            if (mine && ok) {
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    float2 *p = reinterpret_cast<float2 *>(at + b * pitch) + 3 * (lane - A);
                    p[0] = make_float2(v[b][0][0], v[b][0][1]);
                    p[1] = make_float2(v[b][0][2], v[b][1][0]);
                    p[2] = make_float2(v[b][1][1], v[b][1][2]);
                }
            }
        } else if (mine && ok) {
            at += (lane - A) * (f == CRAW_K_OUT_RGBA16F ? 16 : 32);
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const float *p = v[b][0], *q = v[b][1];
                char *d = at + b * pitch;
                if (f == CRAW_K_OUT_RGBA16F) {
                    const __half2 h0 = __floats2half2_rn(p[0], p[1]), h1 = __floats2half2_rn(p[2], 1.0f);
                    const __half2 h2 = __floats2half2_rn(q[0], q[1]), h3 = __floats2half2_rn(q[2], 1.0f);
                    uint4 u;
                    u.x = *reinterpret_cast<const uint32_t *>(&h0);
                    u.y = *reinterpret_cast<const uint32_t *>(&h1);
                    u.z = *reinterpret_cast<const uint32_t *>(&h2);
                    u.w = *reinterpret_cast<const uint32_t *>(&h3);
                    *reinterpret_cast<uint4 *>(d) = u;
                } else if (!((uintptr_t)d & 31)) {
                    walk_store8(reinterpret_cast<float *>(d), p[0], p[1], p[2], 1.0f, q[0], q[1], q[2], 1.0f);
                } else {
                    reinterpret_cast<float4 *>(d)[0] = make_float4(p[0], p[1], p[2], 1.0f);
                    reinterpret_cast<float4 *>(d)[1] = make_float4(q[0], q[1], q[2], 1.0f);
                }
            }
        }
    }

    /* 4x4 block means of (R - G, B - G, G), added row by row over the
     * pixels inside the frame (reference lib/ref/ref_chroma.c:49-74): the
     * left lane of a block's two adds its two pixels of a row to the
     * block's sums, the right lane its two after them. */
    CRAW_DEV void quarter(int r, bool last, const float v[2][2][3])
    {
        const bool right = (lane - A) & 1, in = mine;
        if (!((qy + r) & 1))
            qs[0] = qs[1] = qs[2] = 0.0f;
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float d[2];
#pragma unroll
                for (int p = 0; p < 2; p++)
                    d[p] = c == 2 ? v[b][p][1] : __fsub_rn(v[b][p][2 * c], v[b][p][1]);
                float t = __fadd_rn(__fadd_rn(qs[c], d[0]), d[1]);
                const float u = __fadd_rn(__fadd_rn(walk_left(t), d[0]), d[1]);
                if (right && in)
                    t = u;
                const float back = walk_right(t);
                /* The left lane goes on from the right one's sum where the
                 * frame has that column. */
                qs[c] = !right && lane + 1 < A + nout ? back : t;
            }
        if (!(((qy + r) & 1) || last) || right || !in)
            return;
        const int bx = (qx + lane - A) >> 1, by = (qy + r) >> 1;
        const int nx = min(4, k.width - 4 * bx), ny = min(4, k.height - 4 * by);
        const float n = (float)(nx * ny);
        if (craw_in_bounds(bx >= 0 && bx < (k.width + 3) / 4 && by >= 0 && by < (k.height + 3) / 4, io.err))
            craw_store_rgba(io.quarter, io.quarter_pitch, bx, by, k.fp16, __fdiv_rn(qs[0], n), __fdiv_rn(qs[1], n),
                            __fdiv_rn(qs[2], n));
    }

    /* The AWB block sums of the eight (at the frame's bottom fewer) rows
     * staged so far, row by row (reference lib/awb.c:239-253): lane
     * c NB + b sums channel c of block b. The statistic of a block is over
     * a hundred instructions, so blocks are held until a warp's worth has
     * gathered (or the segment ends). */
    CRAW_DEV void awb_rows(int r, int rows, bool last)
    {
        __syncwarp();
        const int b = lane % S::NB, c = lane / S::NB;
        const int w = min(8, 2 * nout - 8 * b);
        const bool sums = c < 3 && w > 0;
        if (sums) {
            float t = 0.0f;
            if (w == 8) {
#pragma unroll 2
                for (int j = 0; j < rows; j++) {
                    const float *p = &s.a[j][c][S::col(8 * b)];
                    const float4 q0 = *reinterpret_cast<const float4 *>(p), q1 = *reinterpret_cast<const float4 *>(p + 4);
                    t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, q0.x), q0.y), q0.z), q0.w);
                    t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, q1.x), q1.y), q1.z), q1.w);
                }
            } else {
                for (int j = 0; j < rows; j++)
                    for (int i = 0; i < w; i++)
                        t = __fadd_rn(t, s.a[j][c][S::col(8 * b) + i]);
            }
            s.sum[held + b][c] = t;
            if (c == 0)
                s.cnt[held + b] = (float)(w * rows);
        }
        held += (2 * nout + 7) / 8;
        __syncwarp();
        if (!last && held + S::NB <= S::HOLD * S::NB)
            return;
        uint64_t rec = 0;
        if (lane < held) {
            const float n = s.cnt[lane];
            rec = craw_awb_block(__fdiv_rn(s.sum[lane][0], n), __fdiv_rn(s.sum[lane][1], n),
                                 __fdiv_rn(s.sum[lane][2], n), k.awb_wb, io.awb.deferred, io.awb.nb_deferred,
                                 craw_awb_blocks(k.width, k.height));
        }
        __syncwarp();
        craw_awb_add(io.awb.hist, rec);
        held = 0;
        __syncwarp();
    }

    /* Quad row r of the segment (`last`: its last), v[row][pixel][channel]
     * the camera RGB of the lane's quad. The whole warp calls this, for the
     * rows of the segment in order. */
    CRAW_DEV void quad_row(int r, bool last, float v[2][2][3])
    {
        if constexpr (MORE) {
            if (k.fp16) {
#pragma unroll
                for (int b = 0; b < 2; b++)
#pragma unroll
                    for (int p = 0; p < 2; p++)
#pragma unroll
                        for (int c = 0; c < 3; c++)
                            v[b][p][c] = craw_round_half(v[b][p][c]);
            }
            if (io.inter) {
                store(inter, io.inter_pitch, k.fp16 ? CRAW_K_OUT_RGBA16F : CRAW_K_OUT_RGBA32F, r, v);
                inter += 2 * io.inter_pitch;
            }
            if (io.quarter) {
                quarter(r, last, v);
                return;
            }
        }
        if (io.awb.hist && mine) {
            float *a = &s.a[2 * (r & 3)][0][S::col(2 * (lane - A))];
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    *reinterpret_cast<float2 *>(a + (3 * b + c) * S::PITCH) = make_float2(v[b][0][c], v[b][1][c]);
        }
        if (!MORE || io.dst) {
            float o[2][2][3];
            colour(v, o);
            store(dst, io.dst_pitch, fmt(), r, o);
            dst += 2 * io.dst_pitch;
        }
        if (io.awb.hist && ((r & 3) == 3 || last))
            awb_rows(r, 2 * (r & 3) + 2, last);
    }
};

/* One raw row pair of samples (one row of a quad) prepped; row parity `py`. */
CRAW_DEV float2 walk_prep(const CRAWKDevelop &k, const CRAWKDevelopIO &io, uint32_t raw, int py)
{
    if (io.src_f16)   /* rebuilt highlights: fp16, already prepped */
        return __half22float2(*reinterpret_cast<const __half2 *>(&raw));
    return make_float2(craw_prep(k, (uint16_t)(raw & 0xffff), 2 * py),
                       craw_prep(k, (uint16_t)(raw >> 16), 2 * py + 1));
}

/* ----------------------------------------------------------------- RCD */

/* The RCD of the frame's interior (reference lib/ref/ref_debayer.c:204-395)
 * by walking warps, evaluated by the rq_* helpers as the tiles evaluate it,
 * so both give the same bits. Step s forms
 *   D, L of quad row s       (the four discriminations of the quad's
 *                            pixels, the low pass at R and B),
 *   W, G of row s - 1        (the weights from the 3x3 sums of D kept down
 *                            the column, green at R and B) and the colour
 *                            differences KR = R - G, KB = B - G there,
 *   C of row s - 2           (the missing colour at R and B) and its
 *                            differences JR = B - G at R, JB = R - G at B,
 *   the pixels of row s - 3.
 * Every neighbour's term is one of the differences, so each is formed once
 * and crosses the lanes once. Interior strips only: every sample read that
 * a result depends on, down to six pixels outside the strip's output, lies
 * inside the frame; reads past the frame's edge are clamped to it and only
 * feed values nothing reads. */
constexpr int RW_NQ = 24, RW_A = 4;

/* A part of a w x h frame as strips, without segments: the interior (0),
 * whose 64x16 tiles have their aprons inside the frame, and the border above,
 * below, left and right of it (1 to 4; of a frame without an interior, all in
 * 1). nqx or nqy is 0 where a part is empty. */
__host__ CRAW_DEV WalkGrid rcd_part(int width, int height, int i)
{
    const int w2 = width / 2, h2 = height / 2, c_hi = (width - QTW - 6) / QTW, r_hi = (height - QTH - 6) / QTH;
    const bool in = c_hi >= 1 && r_hi >= 1;
    const int x0 = in ? QTW / 2 : w2, x1 = in ? (c_hi + 1) * (QTW / 2) : w2;
    const int y0 = in ? QTH / 2 : h2, y1 = in ? (r_hi + 1) * (QTH / 2) : h2;
    WalkGrid g;
    g.qx0 = i == 0 ? x0 : (i == 4 ? x1 : 0);
    g.nqx = (i == 0 ? x1 : (i == 3 ? x0 : w2)) - g.qx0;
    g.qy0 = i == 1 ? 0 : (i == 2 ? y1 : y0);
    g.nqy = (i == 1 ? y0 : (i == 2 ? h2 : y1)) - g.qy0;
    g.nx = (g.nqx + RW_NQ - 1) / RW_NQ;
    g.seg = 4;
    return g;
}

/* Cuts a part into segments of at most `most` quad rows (a multiple of
 * `unit`, as they are), all alike; returns its warps. */
__host__ CRAW_DEV int walk_cut(WalkGrid &g, int most, int unit = 4)
{
    if (g.nqx <= 0 || g.nqy <= 0)
        return 0;
    const int n = (g.nqy + most - 1) / most;
    g.seg = unit * (((g.nqy + unit - 1) / unit + n - 1) / n);
    return g.nx * ((g.nqy + g.seg - 1) / g.seg);
}

/* The weights, and the colours at a green site, with the roundings of the
 * per-pixel tiles (RcdTile), where the two forms differ. */
CRAW_DEV float rp_wv(float4 s)
{
    const float hs = __fmul_rn(s.y, 1.0f / 9.0f);
    return __fmul_rn(hs, rq_rcp(__fadd_rn(__fmaf_rn(s.x, 1.0f / 9.0f, hs), RCD_EPS)));
}
CRAW_DEV float rp_wp(float4 s)
{
    const float qs = __fmul_rn(s.w, 1.0f / 9.0f);
    return __fmul_rn(qs, rq_rcp(__fadd_rn(__fmaf_rn(s.z, 1.0f / 9.0f, qs), RCD_EPS)));
}
CRAW_DEV void rp_green_site(float wt, float g00, float dh0, float dh1, float ev0, float ev1, float dv0,
                            float dv1, float eh0, float eh1, float &ch, float &cv)
{
    ch = __fmaf_rn(__fsub_rn(1.0f, wt), rq_half_sum(g00, dh0, dh1), __fmul_rn(wt, rq_half_sum(g00, ev0, ev1)));
    cv = rq_blend(wt, rq_half_sum(g00, dv0, dv1), rq_half_sum(g00, eh0, eh1));
}
CRAW_DEV float4 walk_left4(float4 v)
{
    return make_float4(walk_left(v.x), walk_left(v.y), walk_left(v.z), walk_left(v.w));
}
CRAW_DEV float4 walk_right4(float4 v)
{
    return make_float4(walk_right(v.x), walk_right(v.y), walk_right(v.z), walk_right(v.w));
}
/* s + a + b + c in that order. */
CRAW_DEV float4 rp_add3(float4 s, float4 a, float4 b, float4 c)
{
    return rq_add4(rq_add4(rq_add4(s, a), b), c);
}

struct RcdWalk {
    float v[6][6];                    /* pixel rows 2s-2 .. 2s+3, columns X-2 .. X+3 (X: the lane's R) */
    float q2[4], q3[4];               /* the quads of rows s-2, s-3: R, Gr, Gb, B */
    float2 l1, l2;                    /* L of rows s-1, s-2 */
    float4 h[3][2];                   /* 3-wide row sums of D, pixel rows 2s-3 .. 2s-1, two pixels */
    float2 wg2, wg3;                  /* weights at (Gr, Gb), rows s-2, s-3 */
    float2 wp2;                       /* diagonal weights at (R, B), row s-2 */
    float2 g2, g3;                    /* green at (R, B), rows s-2, s-3 */
    float kr2, kr3, krr2, krr3;       /* KR of rows s-2, s-3; the right neighbour's */
    float kb2, kb3, kb4, kbl2, kbl3;  /* KB of rows s-2 .. s-4; the left neighbour's */
    float jr3, jrr3, jb3, jb4, jbl3;  /* JR of row s-3, the right's; JB of rows s-3, s-4, the left's */
    float2 c3;                        /* C of row s-3 */

    /* The two new pixel rows, 2s+2 and 2s+3. */
    CRAW_DEV void rows(float2 a, float2 b)
    {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float2 t = i ? b : a;
            v[4 + i][0] = walk_left(t.x);
            v[4 + i][1] = walk_left(t.y);
            v[4 + i][2] = t.x;
            v[4 + i][3] = t.y;
            v[4 + i][4] = walk_right(t.x);
            v[4 + i][5] = walk_right(t.y);
        }
    }

    /* One step; o: the pixels of row s - 3. */
    CRAW_DEV void step(float o[2][2][3])
    {
        /* D, L of row s. */
        float2 l0;
        float lo[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int y = 2 + e, x = 2 + e;
            lo[e] = rq_lowpass(v[y][x], v[y - 1][x], v[y + 1][x], v[y][x - 1], v[y][x + 1], v[y - 1][x - 1],
                               v[y - 1][x + 1], v[y + 1][x - 1], v[y + 1][x + 1]);
        }
        l0 = make_float2(lo[0], lo[1]);
        float4 hn[2][2];
#pragma unroll
        for (int b = 0; b < 2; b++) {
            float4 d[2];
#pragma unroll
            for (int a = 0; a < 2; a++) {
                auto win = [&](int r, int c) { return v[b + r][a + c]; };
                d[a] = rq_disc4(win);
            }
            const float4 mid = rq_add4(d[0], d[1]);
            const float4 dl = make_float4(walk_left(d[1].x), walk_left(d[1].y), walk_left(d[1].z), walk_left(d[1].w));
            const float4 dr = make_float4(walk_right(d[0].x), walk_right(d[0].y), walk_right(d[0].z),
                                          walk_right(d[0].w));
            hn[b][0] = rq_add4(dl, mid);
            hn[b][1] = rq_add4(mid, dr);
        }
        /* W, G of row s - 1: the 3x3 sums of its first pixel row are h[0..2],
         * of its second h[1], h[2], hn[0]. */
        float4 sum[2][2];
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const float4 mid = rq_add4(h[1][a], h[2][a]);
            sum[0][a] = rq_add4(h[0][a], mid);
            sum[1][a] = rq_add4(hn[0][a], mid);
        }
        const float2 wp1 = make_float2(rq_wp(sum[0][0]), rq_wp(sum[1][1]));
        const float2 wg1 = make_float2(rq_wv(sum[0][1]), rq_wv(sum[1][0]));
        const float2 ll = make_float2(walk_left(l1.x), walk_left(l1.y));
        const float2 lr = make_float2(walk_right(l1.x), walk_right(l1.y));
        const float2 g1 = make_float2(
            rq_green(rq_wv(sum[0][0]), l1.x, q2[2], l2.x, v[1][2], l0.x, v[0][1], ll.x, v[0][3], lr.x),
            rq_green(rq_wv(sum[1][1]), l1.y, v[0][3], l2.y, v[2][3], l0.y, v[1][2], ll.y, v[1][4], lr.y));
        const float kr1 = __fsub_rn(v[0][2], g1.x), kb1 = __fsub_rn(v[1][3], g1.y);
        const float krr1 = walk_right(kr1), kbl1 = walk_left(kb1);
        /* C of row s - 2. */
        const float2 c2 = make_float2(rq_cross(wp2.x, g2.x, kbl2, kb3, kbl3, kb2),
                                      rq_cross(wp2.y, g2.y, kr1, krr2, kr2, krr1));
        const float jr2 = __fsub_rn(c2.x, g2.x), jb2 = __fsub_rn(c2.y, g2.y);
        const float jrr2 = walk_right(jr2), jbl2 = walk_left(jb2);
        /* The pixels of row s - 3. */
        o[0][0][0] = q3[0]; o[0][0][1] = g3.x;  o[0][0][2] = c3.x;
        o[0][1][1] = q3[1];
        rq_green_site(wg3.x, q3[1], kr3, krr3, jb4, jb3, kb4, kb3, jr3, jrr3, o[0][1][0], o[0][1][2]);
        o[1][0][1] = q3[2];
        rq_green_site(wg3.y, q3[2], kbl3, kb3, jr3, jr2, kr3, kr2, jbl3, jb3, o[1][0][2], o[1][0][0]);
        o[1][1][0] = c3.y;  o[1][1][1] = g3.y;  o[1][1][2] = q3[3];
        /* A row on. */
#pragma unroll
        for (int i = 0; i < 4; i++)
            q3[i] = q2[i];
        q2[0] = v[0][2]; q2[1] = v[0][3]; q2[2] = v[1][2]; q2[3] = v[1][3];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 6; c++)
                v[r][c] = v[r + 2][c];
        l2 = l1; l1 = l0;
#pragma unroll
        for (int a = 0; a < 2; a++) {
            h[0][a] = h[2][a];
            h[1][a] = hn[0][a];
            h[2][a] = hn[1][a];
        }
        wg3 = wg2; wg2 = wg1;
        wp2 = wp1;
        g3 = g2; g2 = g1;
        kr3 = kr2; kr2 = kr1; krr3 = krr2; krr2 = krr1;
        kb4 = kb3; kb3 = kb2; kb2 = kb1; kbl3 = kbl2; kbl2 = kbl1;
        jb4 = jb3; jb3 = jb2; jbl3 = jbl2; jr3 = jr2; jrr3 = jrr2;
        c3 = c2;
    }
};

/* The same on the frame's border, the ring of 64x16 tiles that touch it, in
 * the per-pixel tiles' arithmetic (the rp_* helpers where it differs; the 3x3 sums of D one
 * term after another). Outside the frame every array of the RCD holds the
 * value of the position that mirrors there, so:
 *   a column outside is one that the lane at the edge, or its neighbour,
 *   has (left: column -1 is 1, -2 is 2; right: w is w - 2, w + 1 is w - 3);
 *   the quad row above the first gives the first's second row (and its low
 *   pass two rows up is the one two rows down); the quad row below the last
 *   gives the last's first row.
 *
 * Bound: the chain of a step (1.4 us with a warp or two a scheduler). The
 * border by 32x16 tiles of a pixel a thread (920 instructions a pixel, a third
 * of them addresses and mirrored positions) took 26 us after the interior of
 * a 5760x3240 frame and 13 after a 1920x1080 one's; its warps take 21 and 15
 * by themselves, and where they share the interior's wave next to nothing.
 * In the interior's own launch they cost its code registers: 745 against
 * 706 us a 5760x3240 frame. */
struct RingWalk {
    float v[6][6];                    /* as RcdWalk's */
    float q2[4], q3[4];
    float2 l1, l2;
    float4 t[2], rr[2];               /* row 2s-1: the 3x3 sums' first six terms; its own three */
    float4 d0[4];                     /* D of pixel row 2s-2: the left column's, the quad's two, the right's */
    float wv0, wp0, wg0;              /* weights of pixel row 2s-2: at R vertical and diagonal, at Gr */
    float2 wg2, wg3, wp2, g2, g3;
    float kr2, kr3, krr2, krr3;
    float kb2, kb3, kb4, kbl2, kbl3;
    float jr3, jrr3, jb3, jb4, jbl3;
    float2 c3;

    CRAW_DEV void rows(float2 a, float2 b, bool first, bool last)
    {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float2 x = i ? b : a;
            const float lx = walk_left(x.x), ly = walk_left(x.y), rx = walk_right(x.x), ry = walk_right(x.y);
            v[4 + i][0] = first ? rx : lx;
            v[4 + i][1] = first ? x.y : ly;
            v[4 + i][2] = x.x;
            v[4 + i][3] = x.y;
            v[4 + i][4] = last ? x.x : rx;
            v[4 + i][5] = last ? ly : ry;
        }
    }

    /* Step s, `row` its quad row in the frame of h2; first, last: the lane's
     * column is the frame's first, last. o: the pixels of row - 3. */
    CRAW_DEV void step(int row, int h2, bool first, bool last, float o[2][2][3])
    {
        /* D, L of `row`. */
        float lo[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int y = 2 + e, x = 2 + e;
            lo[e] = rq_lowpass(v[y][x], v[y - 1][x], v[y + 1][x], v[y][x - 1], v[y][x + 1], v[y - 1][x - 1],
                               v[y - 1][x + 1], v[y + 1][x - 1], v[y + 1][x + 1]);
        }
        float2 l0 = make_float2(lo[0], lo[1]);
        float4 d[2][4];
#pragma unroll
        for (int b = 0; b < 2; b++) {
#pragma unroll
            for (int a = 0; a < 2; a++) {
                auto win = [&](int r, int c) { return v[b + r][a + c]; };
                d[b][1 + a] = rq_disc4(win);
            }
            const float4 l = walk_left4(d[b][2]), r = walk_right4(d[b][1]);
            d[b][0] = first ? d[b][2] : l;
            d[b][3] = last ? d[b][1] : r;
        }
        if (row == h2) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                d[0][c] = d0[c];
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
            d0[c] = d[0][c];
        float4 r3[2][2], sb[2], sa[2];
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int a = 0; a < 2; a++)
                r3[b][a] = rq_add4(rq_add4(d[b][a], d[b][a + 1]), d[b][a + 2]);
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const float4 up = row == 0 ? r3[1][a] : rr[a];
            sb[a] = rp_add3(t[a], d[0][a], d[0][a + 1], d[0][a + 2]);          /* pixel row 2s - 1 */
            sa[a] = rp_add3(rp_add3(up, d[0][a], d[0][a + 1], d[0][a + 2]), d[1][a], d[1][a + 1], d[1][a + 2]);
            t[a] = rp_add3(r3[0][a], d[1][a], d[1][a + 1], d[1][a + 2]);
            rr[a] = r3[1][a];
        }
        /* W, G of row - 1. */
        const float2 wp1 = make_float2(wp0, rp_wp(sb[1])), wg1 = make_float2(wg0, rp_wv(sb[0]));
        const float wv1 = wv0;
        wv0 = rp_wv(sa[0]);
        wp0 = rp_wp(sa[0]);
        wg0 = rp_wv(sa[1]);
        const float2 la = row == 1 ? make_float2(l0.x, l1.y) : l2;
        const float2 lb = row == h2 ? make_float2(l1.x, l2.y) : l0;
        const float2 le = make_float2(walk_left(l1.x), walk_left(l1.y));
        const float2 ri = make_float2(walk_right(l1.x), walk_right(l1.y));
        const float2 ll = first ? make_float2(ri.x, l1.y) : le, lr = last ? make_float2(l1.x, le.y) : ri;
        const float2 g1 = make_float2(
            rq_green(wv1, l1.x, q2[2], la.x, v[1][2], lb.x, v[0][1], ll.x, v[0][3], lr.x),
            rq_green(rp_wv(sb[1]), l1.y, v[0][3], la.y, v[2][3], lb.y, v[1][2], ll.y, v[1][4], lr.y));
        const float kr1 = __fsub_rn(v[0][2], g1.x), kb1 = __fsub_rn(v[1][3], g1.y);
        const float krn = walk_right(kr1), kbn = walk_left(kb1);
        const float krr1 = last ? kr1 : krn, kbl1 = first ? kb1 : kbn;
        /* C of row - 2. */
        const bool t2 = row == 2, b2 = row == h2 + 1;
        const float2 c2 = make_float2(
            rq_cross(wp2.x, g2.x, kbl2, t2 ? kb2 : kb3, t2 ? kbl2 : kbl3, kb2),
            rq_cross(wp2.y, g2.y, b2 ? kr2 : kr1, krr2, kr2, b2 ? krr2 : krr1));
        const float jr2 = __fsub_rn(c2.x, g2.x), jb2 = __fsub_rn(c2.y, g2.y);
        const float jrn = walk_right(jr2), jbn = walk_left(jb2);
        const float jrr2 = last ? jr2 : jrn, jbl2 = first ? jb2 : jbn;
        /* The pixels of row - 3. */
        const bool t3 = row == 3, b3 = row == h2 + 2;
        o[0][0][0] = q3[0]; o[0][0][1] = g3.x;  o[0][0][2] = c3.x;
        o[0][1][1] = q3[1];
        rp_green_site(wg3.x, q3[1], kr3, krr3, t3 ? jb3 : jb4, jb3, t3 ? kb3 : kb4, kb3, jr3, jrr3, o[0][1][0],
                      o[0][1][2]);
        o[1][0][1] = q3[2];
        rp_green_site(wg3.y, q3[2], kbl3, kb3, jr3, b3 ? jr3 : jr2, kr3, b3 ? kr3 : kr2, jbl3, jb3, o[1][0][2],
                      o[1][0][0]);
        o[1][1][0] = c3.y;  o[1][1][1] = g3.y;  o[1][1][2] = q3[3];
        /* A row on. */
#pragma unroll
        for (int i = 0; i < 4; i++)
            q3[i] = q2[i];
        q2[0] = v[0][2]; q2[1] = v[0][3]; q2[2] = v[1][2]; q2[3] = v[1][3];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 6; c++)
                v[r][c] = v[r + 2][c];
        l2 = l1; l1 = l0;
        wg3 = wg2; wg2 = wg1;
        wp2 = wp1;
        g3 = g2; g2 = g1;
        kr3 = kr2; kr2 = kr1; krr3 = krr2; krr2 = krr1;
        kb4 = kb3; kb3 = kb2; kb2 = kb1; kbl3 = kbl2; kbl2 = kbl1;
        jb4 = jb3; jb3 = jb2; jbl3 = jbl2; jr3 = jr2; jrr3 = jrr2;
        c3 = c2;
    }
};

/* The strip of warp `wid` of one of the border's parts. */
template <int FMT, int RGC, bool MORE>
CRAW_DEV void ring_walk(const CRAWKDevelop &k, const CRAWKDevelopIO &io, const WalkGrid &g, int wid,
                        WalkSmem<RW_NQ> &smem)
{
    const int sx = wid % g.nx, sy = wid / g.nx;
    const int nrows = min(g.seg, g.nqy - sy * g.seg);
    WalkOut<RW_NQ, RW_A, FMT, RGC, MORE> out(k, io, smem, min(RW_NQ, g.nqx - sx * RW_NQ), g.qx0 + sx * RW_NQ,
                                             g.qy0 + sy * g.seg);
    const int w2 = k.width / 2, h2 = k.height / 2, col = out.qx - RW_A + out.lane;
    const int q = max(0, min(col, w2 - 1)), y0 = 2 * out.qy;
    const bool first = col == 0, last = col == w2 - 1;
    const char *src = (const char *)io.src + 4 * (size_t)q;
    auto fetch = [&](int yr) {
        /* The rows that mirror two rows beyond the frame; farther out, any
         * row (nothing reads what comes of it). */
        const int m = abs(y0 + yr), y = max(0, min(m < k.height ? m : 2 * k.height - 2 - m, k.height - 1));
        if (!craw_in_bounds(q >= 0 && 2 * q + 1 < k.width && y >= 0, io.err))
            return 0u;
        return walk_ld(src + (size_t)y * io.src_pitch);
    };
    RingWalk t;
    memset(&t, 0, sizeof(t));
    uint32_t init[4], raw[2];
#pragma unroll
    for (int i = 0; i < 4; i++)
        init[i] = fetch(-6 + i);
#pragma unroll
    for (int i = 0; i < 2; i++)
        raw[i] = fetch(-2 + i);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        t.rows(walk_prep(k, io, init[2 * i], 0), walk_prep(k, io, init[2 * i + 1], 1), first, last);
#pragma unroll
        for (int c = 0; c < 6; c++) {
            t.v[2 * i][c] = t.v[4][c];
            t.v[2 * i + 1][c] = t.v[5][c];
        }
    }
#pragma unroll 1
    for (int s = -2; s <= nrows + 2; s++) {
        uint32_t next[2];
#pragma unroll
        for (int i = 0; i < 2; i++)
            next[i] = fetch(2 * s + 4 + i);
        float o[2][2][3];
        t.rows(walk_prep(k, io, raw[0], 0), walk_prep(k, io, raw[1], 1), first, last);
        t.step(out.qy + s, h2, first, last, o);
        const int r = s - 3;
        if (r >= 0 && r < nrows)
            out.quad_row(r, r == nrows - 1, o);
        raw[0] = next[0];
        raw[1] = next[1];
    }
}

/* The strip of warp `wid` of the grid. */
template <int FMT, int RGC, bool MORE>
CRAW_DEV void rcd_walk(const CRAWKDevelop &k, const CRAWKDevelopIO &io, const WalkGrid &g, int wid,
                       WalkSmem<RW_NQ> &smem)
{
    const int sx = wid % g.nx, sy = wid / g.nx;
    if (sy * g.seg >= g.nqy)
        return;
    const int nrows = min(g.seg, g.nqy - sy * g.seg);
    WalkOut<RW_NQ, RW_A, FMT, RGC, MORE> out(k, io, smem, min(RW_NQ, g.nqx - sx * RW_NQ), g.qx0 + sx * RW_NQ,
                                             g.qy0 + sy * g.seg);
    const int q = min(out.qx - RW_A + out.lane, k.width / 2 - 1), y0 = 2 * out.qy;
    const char *src = (const char *)io.src + 4 * (size_t)q;
    auto fetch = [&](int yr) {
        const int y = min(y0 + yr, k.height - 1);
        if (!craw_in_bounds(q >= 0 && 2 * q + 1 < k.width && y >= 0, io.err))
            return 0u;
        return walk_ld(src + (size_t)y * io.src_pitch);
    };
    RcdWalk t;
    memset(&t, 0, sizeof(t));
    /* Steps -3 .. nrows + 2, two a round (the first fills the pipeline
     * only); the rows of step -3 are -4 and -3, and four rows come before.
     * Every load is issued before the first is used. */
    uint32_t first[4], raw[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        first[i] = fetch(-8 + i);
#pragma unroll
    for (int i = 0; i < 4; i++)
        raw[i] = fetch(-4 + i);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        t.rows(walk_prep(k, io, first[2 * i], 0), walk_prep(k, io, first[2 * i + 1], 1));
#pragma unroll
        for (int c = 0; c < 6; c++) {
            t.v[2 * i][c] = t.v[4][c];
            t.v[2 * i + 1][c] = t.v[5][c];
        }
    }
#pragma unroll 1
    for (int s = -3; s <= nrows + 2; s += 2) {
        uint32_t next[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            next[i] = fetch(2 * s + 6 + i);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float o[2][2][3];
            t.rows(walk_prep(k, io, raw[2 * u], 0), walk_prep(k, io, raw[2 * u + 1], 1));
            t.step(o);
            const int r = s + u - 3;
            if (r >= 0 && r < nrows)
                out.quad_row(r, r == nrows - 1, o);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
            raw[i] = next[i];
    }
}

/* ------------------------------------------------------ bilinear, MHC */

/* The bilinear and MHC debayers of the whole frame by walking warps whose
 * lanes own four pixel columns each: one 4x4 block of the chroma path, half
 * an AWB block. A warp has LW_N output lanes (whole AWB blocks) and an apron
 * lane on either side. Outside the frame a sample is the one its position
 * mirrors to: the rows turn back at the frame's last row, and the lanes at
 * its left and right edge take the mirrored columns from their own.
 *
 * Bound: instruction issue for half-float output, DRAM and its latency for
 * the float layouts. At 5760x3240 (a frame without denoise, AWB on) MHC
 * takes 100 us with RGBA32F and 90 with RGBA16F out, against 155 by 64x16
 * tiles of shared memory with a pixel a thread. Two columns a lane (with the
 * block sums through shared memory) spend a third of their instructions on
 * addresses, constants and branches: 104 and 97 us; eight take too many
 * registers and too long a body for the instruction cache: 135 and 115. */
constexpr int LW_N = 30, LW_P = 4;

/* The four samples of a row from `p`, in the frame (8-byte aligned). */
CRAW_DEV uint2 walk_ld4(const char *p)
{
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

/* What a frame's epilogue is, fixed per kernel so that a row's code stays
 * small: the colour stage to one output layout (a CRAW_K_OUT_*); the chroma
 * path's (intermediate and block means); or any of it by tests (a kept
 * intermediate). */
constexpr int LW_CHROMA = 3, LW_ANY = 4;

template <int METHOD, int EPI>
struct LinearWalk {
    static constexpr bool CHROMA = EPI == LW_CHROMA, ANY = EPI == LW_ANY;
    static constexpr int RAD = METHOD == kMhc ? 2 : 1;   /* pixels around a quad that its debayer reads */
    static constexpr int WR = 2 + 2 * RAD, WC = LW_P + 2 * RAD;
    const CRAWKDevelop &k;
    const CRAWKDevelopIO &io;
    float v[WR][WC];         /* pixel rows 2r - RAD .. 2r + 1 + RAD, columns x0 - RAD .. x0 + 3 + RAD */
    int x0, nv;              /* the lane's first column; its columns inside the frame (output lanes) */
    bool edge;               /* the warp reaches the frame's left or right edge */
    bool inside, partial;    /* the lane's four columns are in the frame; its first two only */
    bool mine, right;        /* an output lane; the second of its AWB block */
    float as[3], hs[3];      /* the AWB block's sums so far; the block's above, waiting */
    bool held;               /* whether hs waits */
    float qs[3];             /* chroma: the sums of the 4x4 block so far */
    char *dst, *inter;       /* the lane's pixels in the row to store next */

    CRAW_DEV LinearWalk(const CRAWKDevelop &k_, const CRAWKDevelopIO &io_) : k(k_), io(io_) {}

    CRAW_DEV float at(int x, int y) const { return v[y][x]; }

    /* A row's four samples; of a lane that hangs over the right edge by two,
     * its two; of a lane outside the frame, none. (No lane combines what it
     * loads before it is used, a round later.) */
    CRAW_DEV uint2 load(const char *row) const
    {
        uint2 u = make_uint2(0u, 0u);
        if (!craw_in_bounds(row >= (const char *)io.src &&
                            row <= (const char *)io.src + (size_t)(k.height - 1) * io.src_pitch, io.err))
            return u;
        if (inside)
            u = walk_ld4(row + 2 * (size_t)x0);
        else if (partial)
            u.x = walk_ld(row + 2 * (size_t)x0);
        return u;
    }

    /* A raw row of parity py into window row `r`. The columns outside the
     * frame mirror into the lane's own or its left neighbour's. */
    CRAW_DEV void put(int r, uint2 raw, int py)
    {
        const float2 a = walk_prep(k, io, raw.x, py), b = walk_prep(k, io, raw.y, py);
        float p[LW_P] = { a.x, a.y, b.x, b.y }, l[RAD], q[RAD];   /* q: to the right */
#pragma unroll
        for (int i = 0; i < RAD; i++) {
            l[i] = walk_left(p[LW_P - RAD + i]);
            q[i] = walk_right(p[i]);
        }
        if (edge) {
            if (x0 == 0)
#pragma unroll
                for (int i = 0; i < RAD; i++)
                    l[i] = p[RAD - i];                   /* column -RAD + i */
            if (partial) {
                p[2] = p[0];                             /* column w: w - 2 */
                p[3] = l[RAD - 1];                       /* column w + 1: w - 3 */
            }
            if (x0 + LW_P == k.width)
#pragma unroll
                for (int i = 0; i < RAD; i++)
                    q[i] = p[LW_P - 2 - i];              /* column w + i: w - 2 - i */
        }
#pragma unroll
        for (int i = 0; i < RAD; i++) {
            v[r][i] = l[i];
            v[r][RAD + LW_P + i] = q[i];
        }
#pragma unroll
        for (int i = 0; i < LW_P; i++)
            v[r][RAD + i] = p[i];
    }

    /* The lane's pixels of row y of the RGB image at `base` (layout f), which
     * are at `d`. */
    CRAW_DEV void store(char *d, const void *base, size_t pitch, int y, int f, const float o[LW_P][3]) const
    {
        if (!mine || !craw_in_bounds(y >= 0 && y < k.height && x0 >= 0 && x0 + nv <= k.width &&
                                     d == (const char *)base + (size_t)y * pitch + (size_t)x0 * walk_bytes(f), io.err))
            return;
        if (nv == LW_P) {
            float *p = reinterpret_cast<float *>(d);
            if (f == CRAW_K_OUT_RGB32F) {
#pragma unroll
                for (int i = 0; i < 12; i += 4)
                    *reinterpret_cast<float4 *>(p + i) = make_float4(o[i / 3][i % 3], o[(i + 1) / 3][(i + 1) % 3],
                                                                     o[(i + 2) / 3][(i + 2) % 3],
                                                                     o[(i + 3) / 3][(i + 3) % 3]);
            } else if (f == CRAW_K_OUT_RGBA16F) {
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < LW_P; i++) {
                    const __half2 a = __floats2half2_rn(o[i][0], o[i][1]), b = __floats2half2_rn(o[i][2], 1.0f);
                    w[2 * i] = *reinterpret_cast<const uint32_t *>(&a);
                    w[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&b);
                }
                reinterpret_cast<uint4 *>(d)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                reinterpret_cast<uint4 *>(d)[1] = make_uint4(w[4], w[5], w[6], w[7]);
            } else if (!((uintptr_t)d & 31)) {
#pragma unroll
                for (int i = 0; i < LW_P; i += 2)
                    walk_store8(p + 4 * i, o[i][0], o[i][1], o[i][2], 1.0f, o[i + 1][0], o[i + 1][1], o[i + 1][2],
                                1.0f);
            } else {
#pragma unroll
                for (int i = 0; i < LW_P; i++)
                    reinterpret_cast<float4 *>(p)[i] = make_float4(o[i][0], o[i][1], o[i][2], 1.0f);
            }
        } else {
#pragma unroll
            for (int i = 0; i < LW_P; i++)
                if (i < nv)
                    craw_store_rgba(d, 0, i, 0, f, o[i][0], o[i][1], o[i][2]);
        }
    }

    /* The 4x4 block means of (R - G, B - G, G), added row by row over the
     * pixels inside the frame (reference lib/ref/ref_chroma.c:49-74). */
    CRAW_DEV void quarter(int y, bool last, bool odd, const float o[LW_P][3])
    {
        if (!(y & 3))
            qs[0] = qs[1] = qs[2] = 0.0f;
#pragma unroll
        for (int i = 0; i < LW_P; i++)
            if (i < nv) {
                qs[0] = __fadd_rn(qs[0], __fsub_rn(o[i][0], o[i][1]));
                qs[1] = __fadd_rn(qs[1], __fsub_rn(o[i][2], o[i][1]));
                qs[2] = __fadd_rn(qs[2], o[i][1]);
            }
        if (!odd || !((y & 3) == 3 || last) || !mine)
            return;
        const int bx = x0 / 4, by = y / 4;
        const float n = (float)(nv * ((y & 3) + 1));
        if (craw_in_bounds(bx >= 0 && bx < (k.width + 3) / 4 && by >= 0 && by < (k.height + 3) / 4, io.err))
            craw_store_rgba(io.quarter, io.quarter_pitch, bx, by, k.fp16, __fdiv_rn(qs[0], n), __fdiv_rn(qs[1], n),
                            __fdiv_rn(qs[2], n));
    }

    /* The statistic of the block whose sums are s, of `rows` pixel rows, on
     * the lanes that `go`. */
    CRAW_DEV void statistic(const float s[3], int rows, bool go)
    {
        const float n = (float)(min(8, k.width - (x0 & ~7)) * rows);
        uint64_t rec = 0;
        if (go)
            rec = craw_awb_block(__fdiv_rn(s[0], n), __fdiv_rn(s[1], n), __fdiv_rn(s[2], n), k.awb_wb,
                                 io.awb.deferred, io.awb.nb_deferred, craw_awb_blocks(k.width, k.height));
        __syncwarp();
        craw_awb_add(io.awb.hist, rec);
    }

    /* The AWB sums of a row, in the reference's order (lib/awb.c:239-253):
     * the left lane of a block adds its four pixels, the right lane its
     * four after them. The left lanes hold the sums; every second row of
     * blocks the right lanes take the row above's, so that the statistic
     * (over a hundred instructions) runs on all lanes at once. */
    CRAW_DEV void awb_row(int y, bool end, bool odd, const float o[LW_P][3])
    {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float t = as[c];
#pragma unroll
            for (int i = 0; i < LW_P; i++)
                t = nv == LW_P || i < nv ? __fadd_rn(t, o[i][c]) : t;
            float u = walk_left(t);
#pragma unroll
            for (int i = 0; i < LW_P; i++)
                u = nv == LW_P || i < nv ? __fadd_rn(u, o[i][c]) : u;
            as[c] = walk_right(u);
        }
        if (!odd || ((y & 7) != 7 && !end))
            return;
        if (!held && !end) {
#pragma unroll
            for (int c = 0; c < 3; c++)
                hs[c] = as[c];
            held = true;
        } else {
            float s[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float above = walk_left(hs[c]);
                s[c] = right ? above : as[c];
            }
            statistic(s, right ? 8 : (y & 7) + 1,
                      right ? held && x0 - LW_P < k.width && mine_pair() : mine);
            held = false;
        }
        as[0] = as[1] = as[2] = 0.0f;
    }
    /* Whether the lane's AWB block is an output of the strip (its right
     * lane may lie past the frame's edge). */
    CRAW_DEV bool mine_pair() const
    {
        const int lane = threadIdx.x & 31;
        return lane >= 1 && lane <= LW_N;
    }

    /* The epilogue of frame row y (`end`: the segment's last; `odd`: its
     * parity, constant where it is inlined): o the lane's camera RGB. */
    CRAW_DEV void row(int y, bool end, bool odd, float o[LW_P][3])
    {
        if (k.fp16) {
#pragma unroll
            for (int i = 0; i < LW_P; i++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    o[i][c] = craw_round_half(o[i][c]);
        }
        if (CHROMA || (ANY && io.inter)) {
            store(inter, io.inter, io.inter_pitch, y, k.fp16 ? CRAW_K_OUT_RGBA16F : CRAW_K_OUT_RGBA32F, o);
            inter += io.inter_pitch;
        }
        if constexpr (CHROMA) {
            quarter(y, end, odd, o);
            return;
        }
        if (io.awb.hist)
            awb_row(y, end, odd, o);
        if (!ANY || io.dst) {
            walk_colour<-1>(k.color, mine, o);
            store(dst, io.dst, io.dst_pitch, y, ANY ? io.dst_fmt : EPI, o);
            dst += io.dst_pitch;
        }
    }

    /* The lane's place in the strip of warp `wid` of the grid (the whole
     * frame's, in strips of LW_N lanes and segments of g.seg quad rows): its
     * segment's pixel rows are y0 .. y0 + rows; false where there is none. */
    CRAW_DEV bool place(const WalkGrid &g, int wid, int &y0, int &rows)
    {
        const int lane = threadIdx.x & 31, sx = wid % g.nx, sy = wid / g.nx;
        if (sy * g.seg >= g.nqy)
            return false;
        y0 = 2 * sy * g.seg;
        rows = 2 * min(g.seg, g.nqy - sy * g.seg);
        x0 = LW_P * (sx * LW_N - 1 + lane);
        edge = sx == 0 || LW_P * (sx * LW_N + 31) >= k.width;
        inside = x0 >= 0 && x0 + LW_P <= k.width;
        partial = x0 + 2 == k.width;
        mine = lane >= 1 && lane <= LW_N && x0 < k.width;
        right = !(lane & 1);
        nv = min(LW_P, k.width - x0);
        held = false;
#pragma unroll
        for (int c = 0; c < 3; c++)
            as[c] = hs[c] = qs[c] = 0.0f;
        const int f = ANY ? io.dst_fmt : EPI;
        dst = (char *)io.dst + (size_t)y0 * io.dst_pitch + (ptrdiff_t)x0 * walk_bytes(f);
        inter = (char *)io.inter + (size_t)y0 * io.inter_pitch + (ptrdiff_t)x0 * (k.fp16 ? 8 : 16);
        return true;
    }

    CRAW_DEV void run(const WalkGrid &g, int wid)
    {
        int y0, rows;
        if (!place(g, wid, y0, rows))
            return;
        int y = y0;
        const char *src = (const char *)io.src + (size_t)y0 * io.src_pitch;
        auto fetch = [&]() {
            const uint2 u = load(src);
            y++;
            src += y < k.height ? (ptrdiff_t)io.src_pitch : -(ptrdiff_t)io.src_pitch;
            return u;
        };
        /* The window's first rows, and the first two steps' two each; every
         * load is issued before the first is used. */
        uint2 first[2 * RAD], next[2][2];
#pragma unroll
        for (int i = 0; i < RAD; i++)
            first[i] = load((const char *)io.src + (size_t)craw_mirror(y0 - RAD + i, k.height) * io.src_pitch);
#pragma unroll
        for (int i = RAD; i < 2 * RAD; i++)
            first[i] = fetch();
#pragma unroll
        for (int i = 0; i < 4; i++)
            next[i >> 1][i & 1] = fetch();
#pragma unroll
        for (int i = 0; i < 2 * RAD; i++)
            put(i, first[i], (i + RAD) & 1);
#pragma unroll 1
        for (int r = 0; r < rows; r += 2) {
            put(2 * RAD, next[0][0], RAD & 1);
            put(2 * RAD + 1, next[0][1], (RAD + 1) & 1);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                next[0][i] = next[1][i];
                next[1][i] = fetch();
            }
#pragma unroll
            for (int b = 0; b < 2; b++) {
                float o[LW_P][3];
#pragma unroll
                for (int i = 0; i < LW_P; i++) {
                    if constexpr (METHOD == kMhc)
                        mhc_px(*this, RAD + i, RAD + b, 2 * b + (i & 1), o[i]);
                    else
                        bilinear_px(*this, RAD + i, RAD + b, 2 * b + (i & 1), o[i]);
                }
                /* A segment has whole quad rows: only their second row can
                 * end a block or the segment. */
                row(y0 + r + b, b && r + 2 == rows, b, o);
            }
#pragma unroll
            for (int i = 0; i < 2 * RAD; i++)
#pragma unroll
                for (int c = 0; c < WC; c++)
                    v[i][c] = v[i + 2][c];
        }
    }
};

} // namespace craw_dev
