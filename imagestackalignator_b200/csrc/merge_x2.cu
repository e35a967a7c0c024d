// Kernel-weighted Bayer accumulation at merge scales 2 (the reference's
// accumulateImagesSuperRes, DeBayerKernels.cu:379-468, and its whole-frame
// generalisation) and 1 (accumulateImages, :290-376; below), restructured so that no lane of a warp diverges from the
// others on the interior path.
//
// Geometry at s = 2. Output pixel (X, Y) (origin included) with shift
// (sx, sy) = round(2 * flow) reads, for its 5 x 5 taps, source samples
// q = (Xs + p) >> 1 with Xs = X + sx: a 3 x 3 block of cells starting at
// k0 = (Xs - 2) >> 1, j0 = (Ys - 2) >> 1. Tap p -> cell is 0 0 1 1 2 when
// Xs is even and 0 1 1 2 2 when it is odd (rows alike). The certainty of a
// tap comes from the half-resolution mask cell of the UNSHIFTED tap,
// (X + p) >> 2, so which of the two mask columns a tap reads depends only on
// X mod 4 (and rows on Y mod 4).
//
// Work layout. A warp covers 32 output pixels of one row, four columns apart
// (x = 128 bx + 4 lane + ph), so X mod 4 and Y mod 4 are the same for the
// whole warp. A CTA is the four ph of 128-pixel segments of four rows of one
// Y mod 4: its warps share the source lines they read, and the segments are
// written in whole lines through shared memory.
//
// The taps of a line fall into four groups of one cell and one mask line each,
// whatever the parity of Xs: that parity only moves the taps -1 and +1 between
// neighbouring groups, by multiply-adds with a 0 / 1 factor (the FMA pipe has
// room, the ALU pipe that selects run on does not). So the 5 x 5 weights (13
// distinct: w(-p) = w(p)) fold to 4 x 4 group weights, and the certainties
// meet them once per group:
//   W(cell) = sum over the cell's groups of (group weight) (certainty),
// with the certainty of the group's relative CFA class in its mask cell.
// The 3 x 3 cell weights multiply the 3 x 3 samples into the four relative
// CFA classes, which map to R, G, B through two bits per frame.
// Per frame and channel: acc_c += (sum w cert raw - black_c sum w cert) /
// white_c, wsum_c += sum w cert: the reference's per-tap
// (raw - black_c) / white_c * w * cert summed over the taps of the frame. (At
// scale 1 and tap by tap black is taken off each sample.)
// Pixels whose 3 x 3 block, mask window or flow cell reaches a border (and
// weights so large that their sums could overflow) take a per-tap path with
// the reference's clamps, out of line.
//
// Bound: instruction issue and instruction fetch, 316 instructions per pixel
// and frame over 8 frames (the pixel's own set-up among them) at an IPC of 2.5,
// the ALU pipe at 50 %. Code size decides as much as the count:
// the frame loop is one body per Y mod 4 (uniform in a CTA, and the rows of a
// 32-row band run one Y mod 4 after another) with a 35-instruction section
// per X mod 4. One body per (X mod 4, Y mod 4) pair inside a CTA took 157 ms
// at 20 x 6016x4000 (the instruction cache thrashes), the same bodies with
// CTA-uniform X mod 4 23.3 ms (the sixteen interleaved CTAs re-read each line
// from L2), four pixels per thread 36 ms (a 16 KB body), group weights in a
// shared-memory table 28-34 ms (no L1 left for the frames). This form: 23.4 ms,
// from 25.4 ms for per-tap selects; one 4096x3072 frame by itself 0.54 ms, from
// 0.87 ms. CTAs of 256 threads take 22.5 ms, but where bursts are merged side by
// side on several streams small CTAs refill every slot they free and keep the
// other streams' larger CTAs waiting (six bursts of 6 x 1024x768 on three
// streams: 7.78 ms with 256 threads, 7.48 ms with 512).
#include "isa_internal.cuh"

namespace {

constexpr int X2_W = 128, X2_ROWS = 4;  // row segment of a CTA's 128-thread part, rows (of one y mod 4) per CTA
constexpr int X2_NT = X2_W * X2_ROWS, X2_CTAS = 2;  // threads of a CTA, CTAs per SM

struct C3 { float v[3]; };

// Bayer description: green where (row parity ^ column parity) == g0, red on
// rows with parity ry.
struct Bayer { int g0, ry; };

__device__ __forceinline__ float4 sanitize(float4 m)
{
    m.x = isfinite(m.x) ? m.x : 0.f;
    m.y = isfinite(m.y) ? m.y : 0.f;
    m.z = isfinite(m.z) ? m.z : 0.f;
    return m;
}

// Certainties of the four relative CFA classes (class r = row parity * 2 +
// column parity, relative to (k0, j0)) in mask cell m. hG: relative class 0
// is green; fr: non-green cells on relative row 0 are red.
__device__ __forceinline__ void class_certs(const float4& m, bool hG, bool fr, float (&c)[4])
{
    const float rb0 = fr ? m.x : m.z, rb1 = fr ? m.z : m.x;
    c[0] = hG ? m.y : rb0;
    c[1] = hG ? rb0 : m.y;
    c[2] = hG ? rb1 : m.y;
    c[3] = hG ? m.y : rb1;
}

// The five taps of a line (-2 .. 2) into the four groups of X mod 4 == M (rows alike). P = 1, nP = 0 where the shifted
// position is odd, else P = 0, nP = 1. (Even: taps -2 -1 | 0 +1 | +2 share cells; odd: -2 | -1 0 | +1 +2.)
template <int M>
__device__ __forceinline__ void fold(float w0, float w1, float w2, float w3, float w4, float P, float nP, float (&g)[4])
{
    if constexpr (M == 0) {         // mask lines: -2 -1 | 0 +1 +2
        g[0] = fmaf(nP, w1, w0); g[1] = P * w1; g[2] = fmaf(nP, w3, w2); g[3] = fmaf(P, w3, w4);
    } else if constexpr (M == 1) {  // -2 | -1 0 +1 +2
        g[0] = w0; g[1] = nP * w1; g[2] = fmaf(nP, w3, fmaf(P, w1, w2)); g[3] = fmaf(P, w3, w4);
    } else if constexpr (M == 2) {  // -2 -1 0 +1 | +2
        g[0] = fmaf(nP, w1, w0); g[1] = fmaf(nP, w3, fmaf(P, w1, w2)); g[2] = P * w3; g[3] = w4;
    } else {                        // -2 -1 0 | +1 +2
        g[0] = fmaf(nP, w1, w0); g[1] = fmaf(P, w1, w2); g[2] = nP * w3; g[3] = fmaf(P, w3, w4);
    }
}

// Cell and mask line of group g for X mod 4 == M.
__host__ __device__ constexpr int cell_of(int M, int g) { return g == 0 ? 0 : (g == 3 ? 2 : (g == 1 ? (M == 1 ? 0 : 1) : (M == 2 ? 2 : 1))); }
__host__ __device__ constexpr int mline_of(int M, int g) { return g == 0 ? 0 : (g == 3 ? 1 : (g == 1 ? (M == 1 ? 1 : 0) : (M == 2 ? 0 : 1))); }

// Tap weights and certainties cq[mask row][mask column][class] -> cell weights: columns to groups, then rows, then the
// groups' certainties.
template <int XM, int YM>
__device__ __forceinline__ void cells(const float (&w)[5][5], float Q, float nQ, float P, float nP, const float (&cq)[2][2][4], float (&Wc)[3][3])
{
    bool set[3][3] = {};
    float G[5][4];
#pragma unroll
    for (int r = 0; r < 5; r++) fold<XM>(w[r][0], w[r][1], w[r][2], w[r][3], w[r][4], P, nP, G[r]);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float u[4];
        fold<YM>(G[0][c], G[1][c], G[2][c], G[3][c], G[4][c], Q, nQ, u);
        const int i = cell_of(XM, c);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int j = cell_of(YM, r);
            const float k = cq[mline_of(YM, r)][mline_of(XM, c)][(j & 1) * 2 + (i & 1)];
            Wc[j][i] = set[j][i] ? fmaf(u[r], k, Wc[j][i]) : u[r] * k;
            set[j][i] = true;
        }
    }
}

struct X2Args {
    isa_accum_geom g;
    unsigned cfa;
    Bayer bayer;
    int nframes;
    size_t raw_pitch, flow_pitch, mask_pitch;
    const float4* kparam;
    size_t kp_pitch;
    C3 rwhite, rwlow, black;  // 1 / white: at scale 2 rwhite, rounded, at scale 1 rwhite + rwlow
    isa_levels lv;            // of the samples tap by tap at scale 1
    float* acc;
    float* wsum;
    size_t out_pitch;
    int accumulate_into;
    isa_frame_in frames[ISA_ACC_MAX_FRAMES];
};

// What a frame without flow (two texels) or mask (up to three cells) reads, at offset 0.
__device__ const float4 g_zero_flow = {0.f, 0.f, 0.f, 0.f};
__device__ const float4 g_unit_mask[3] = {{1.f, 1.f, 1.f, 1.f}, {1.f, 1.f, 1.f, 1.f}, {1.f, 1.f, 1.f, 1.f}};

struct Sums { float a[3], w[3]; };

// Sample position of output pixel (x, y): texel and sub-pixel part.
struct Position { int ib, jb; float ax, by; };

__device__ __forceinline__ Position position(const isa_accum_geom& g, int x, int y)
{
    const float xb = ((float)x + 0.5f + (float)g.ox) / 2.0f - 0.5f;
    const float yb = ((float)y + 0.5f + (float)g.oy) / 2.0f - 0.5f;
    const float fxb = floorf(xb), fyb = floorf(yb);
    return {(int)fxb, (int)fyb, xb - fxb, yb - fyb};
}

// Kernel parameters: bilinear, clamp addressing.
__device__ __forceinline__ void kernel_params(const X2Args& A, const Position& p, float& k0, float& k1, float& k2)
{
    const isa_accum_geom& g = A.g;
    const int i0 = isa::clampi(p.ib, 0, g.W - 1), i1 = isa::clampi(p.ib + 1, 0, g.W - 1);
    const int j0 = isa::clampi(p.jb, 0, g.H - 1), j1 = isa::clampi(p.jb + 1, 0, g.H - 1);
    const float4 p00 = __ldg(isa::row_ptr(A.kparam, A.kp_pitch, j0) + i0), p10 = __ldg(isa::row_ptr(A.kparam, A.kp_pitch, j0) + i1);
    const float4 p01 = __ldg(isa::row_ptr(A.kparam, A.kp_pitch, j1) + i0), p11 = __ldg(isa::row_ptr(A.kparam, A.kp_pitch, j1) + i1);
    k0 = isa::lerp2(p00.x, p10.x, p01.x, p11.x, p.ax, p.by);
    k1 = isa::lerp2(p00.y, p10.y, p01.y, p11.y, p.ax, p.by);
    k2 = isa::lerp2(p00.z, p10.z, p01.z, p11.z, p.ax, p.by);
}

// The 13 distinct tap weights, w(-p) = w(p), from the kernel parameters; returns the largest.
__device__ __forceinline__ float tap_weights(float k0, float k1, float k2, float (&w)[5][5])
{
    float wmax = 1.f;
#pragma unroll
    for (int py = 0; py <= 2; py++)
#pragma unroll
        for (int px = -2; px <= 2; px++) {
            if (py == 0 && px < 0) continue;
            float v = 1.f;
            if (py != 0 || px != 0) {
                const float q = px * px * k0 + 2 * px * py * k2 + py * py * k1;
                v = expf(-0.5f * q);
                if (!isfinite(v)) v = px * py == 0 ? 1.f : 0.f;
                wmax = fmaxf(wmax, v);
            }
            w[2 + py][2 + px] = w[2 - py][2 - px] = v;
        }
    return wmax;
}

// One frame's sums of a pixel tap by tap at scale S (1 or 2), with the crop clamps and mirrored flow of the reference.
// Scale 1: a is normalised; scale 2: a holds the sums of w cert raw.
template <int S, bool SAME>
__device__ __noinline__ Sums frame_per_tap(const X2Args& A, int f, int x, int y)
{
    constexpr int SH = S - 1;
    const isa_accum_geom& g = A.g;
    const isa_frame_in fr = A.frames[f];
    const int X = x + g.ox, Y = y + g.oy;
    const Position p = S == 1 ? Position{X, Y, 0.f, 0.f} : position(g, x, y);
    float k0, k1, k2, w[5][5];
    kernel_params(A, p, k0, k1, k2);
    tap_weights(k0, k1, k2, w);
    Sums s = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    int sx = 0, sy = 0;
    if (fr.flow) {
        const int i0 = isa::mirror(p.ib, g.W), i1 = isa::mirror(p.ib + 1, g.W);
        const float2* r0 = isa::row_ptr(fr.flow, A.flow_pitch, isa::mirror(p.jb, g.H));
        const float2* r1 = isa::row_ptr(fr.flow, A.flow_pitch, isa::mirror(p.jb + 1, g.H));
        const float2 p00 = __ldg(r0 + i0), p10 = __ldg(r0 + i1), p01 = __ldg(r1 + i0), p11 = __ldg(r1 + i1);
        sx = (int)roundf(isa::lerp2(p00.x, p10.x, p01.x, p11.x, p.ax, p.by) * (float)S);
        sy = (int)roundf(isa::lerp2(p00.y, p10.y, p01.y, p11.y, p.ax, p.by) * (float)S);
    }
    int qx[5], ux[5];
#pragma unroll
    for (int d = 0; d < 5; d++) {
        qx[d] = isa::clampi((X + sx + d - 2) >> SH, g.cx0, g.cx1);
        ux[d] = (isa::clampi((X + d - 2) >> SH, g.cx0, g.cx1) >> 1) * 4;
    }
#pragma unroll
    for (int py = -2; py <= 2; py++) {
        const int qy = isa::clampi((Y + sy + py) >> SH, g.cy0, g.cy1);
        const int uy = isa::clampi((Y + py) >> SH, g.cy0, g.cy1) >> 1;
        const uint16_t* rr = isa::row_ptr(fr.raw, A.raw_pitch, qy);
        const float* mr = fr.mask ? (const float*)isa::row_ptr(fr.mask, A.mask_pitch, uy) : nullptr;
#pragma unroll
        for (int d = 0; d < 5; d++) {
            const int c = isa::cfa_at(A.cfa, qx[d], qy);
            float cert = 1.f;
            if (mr) {
                cert = __ldg(mr + ux[d] + c);
                if (!isfinite(cert)) cert = 0.f;
            }
            const float wc = __fmul_rn(w[py + 2][d], cert);
            float v = (float)__ldg(rr + qx[d]);
            if constexpr (S == 1)
                v = __fmaf_rn(v, A.lv.scale, SAME ? A.lv.nblack[0] : (c == 0 ? A.lv.nblack[0] : (c == 1 ? A.lv.nblack[1] : A.lv.nblack[2])));
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (k == c) { s.w[k] = __fadd_rn(s.w[k], wc); s.a[k] = __fmaf_rn(wc, v, s.a[k]); }
        }
    }
    if constexpr (S == 1) {
#pragma unroll
        for (int c = 0; c < 3; c++) s.a[c] = __fmaf_rn(s.a[c], A.lv.rhigh[c], s.a[c] * A.lv.rlow[c]);
    }
    return s;
}

// Frames f0, f0 + 1, ... of output pixel (x, y), y mod 4 (with the origin) == YM, up to the first whose 3 x 3 block
// reaches a border (returned); w: the tap weights; interior: neither the unshifted taps' mask cells nor the flow's
// texels reach a border.
template <int YM, bool SANE>
__device__ __forceinline__ int frames_x2(const X2Args& A, int f0, int x, int y, const float (&w)[5][5], bool interior, float (&a)[3], float (&ws)[3])
{
    const isa_accum_geom& g = A.g;
    const int X = x + g.ox, Y = y + g.oy, XM = X & 3;
    const Position p = position(g, x, y);
    // bilinear weights of the flow sample (never zero at scale 2), combined in lerp2's order and rounding
    const float f00 = (1.f - p.ax) * (1.f - p.by), f10 = p.ax * (1.f - p.by), f01 = (1.f - p.ax) * p.by, f11 = p.ax * p.by;
    const unsigned foff = (unsigned)isa::clampi(p.jb, 0, g.H - 2) * (unsigned)A.flow_pitch + (unsigned)isa::clampi(p.ib, 0, g.W - 2) * 8u;
    const unsigned moff = (unsigned)isa::clampi((Y - 2) >> 2, 0, g.H / 2 - 2) * (unsigned)A.mask_pitch + (unsigned)isa::clampi((X - 2) >> 2, 0, g.W / 2 - 2) * 16u;
    // the shifted 3 x 3 block lies inside the crop: k0 in [cx0, cx1 - 2], j0 in [cy0, cy1 - 2]
    const unsigned kspan = (unsigned)(g.cx1 - 2 - g.cx0), jspan = (unsigned)(g.cy1 - 2 - g.cy0);
    int f = f0;
#pragma unroll 1
    for (; f < A.nframes; f++) {
        const char* fl = (const char*)A.frames[f].flow;
        const char* fb = fl ? fl : (const char*)&g_zero_flow;
        const char* fb1 = fb + (fl ? A.flow_pitch : 0);
        const unsigned fo = fl ? foff : 0u;
        const float2 p00 = __ldg((const float2*)(fb + fo)), p10 = __ldg((const float2*)(fb + fo) + 1);
        const float2 p01 = __ldg((const float2*)(fb1 + fo)), p11 = __ldg((const float2*)(fb1 + fo) + 1);
        const float flx = __fmaf_rn(f11, p11.x, __fmaf_rn(f01, p01.x, __fmaf_rn(f10, p10.x, __fmul_rn(f00, p00.x))));
        const float fly = __fmaf_rn(f11, p11.y, __fmaf_rn(f01, p01.y, __fmaf_rn(f10, p10.y, __fmul_rn(f00, p00.y))));
        const int Xs = X + (int)roundf(flx * 2.0f), Ys = Y + (int)roundf(fly * 2.0f);
        const int k0 = (Xs - 2) >> 1, j0 = (Ys - 2) >> 1;
        if (!(interior && (unsigned)(k0 - g.cx0) <= kspan && (unsigned)(j0 - g.cy0) <= jspan)) {
            break;
        }
        const unsigned ro = (unsigned)j0 * (unsigned)A.raw_pitch + 2u * (unsigned)k0;
        float v[3][3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint16_t* rr = (const uint16_t*)((const char*)A.frames[f].raw + j * A.raw_pitch + ro);
            v[j][0] = (float)__ldg(rr);
            v[j][1] = (float)__ldg(rr + 1);
            v[j][2] = (float)__ldg(rr + 2);
        }
        const char* mk = (const char*)A.frames[f].mask;
        const char* mb = mk ? mk : (const char*)g_unit_mask;
        const char* mb1 = mb + (mk ? A.mask_pitch : 0);
        const unsigned mo = mk ? moff : 0u;
        float4 M00 = __ldg((const float4*)(mb + mo)), M01 = __ldg((const float4*)(mb + mo) + 1);
        float4 M10 = __ldg((const float4*)(mb1 + mo)), M11 = __ldg((const float4*)(mb1 + mo) + 1);
        const bool fx = k0 & 1, fy = j0 & 1;
        const bool hG = (int)(fx ^ fy) == A.bayer.g0, frr = (int)fy == A.bayer.ry;
        float cq[2][2][4];
        if (!SANE) { M00 = sanitize(M00); M01 = sanitize(M01); M10 = sanitize(M10); M11 = sanitize(M11); }
        class_certs(M00, hG, frr, cq[0][0]);
        class_certs(M01, hG, frr, cq[0][1]);
        class_certs(M10, hG, frr, cq[1][0]);
        class_certs(M11, hG, frr, cq[1][1]);
        const float P = (Xs & 1) ? 1.f : 0.f, nP = 1.f - P, Q = (Ys & 1) ? 1.f : 0.f, nQ = 1.f - Q;
        float Wc[3][3];
        // the same for the whole warp
        if (XM == 0) cells<0, YM>(w, Q, nQ, P, nP, cq, Wc);
        else if (XM == 1) cells<1, YM>(w, Q, nQ, P, nP, cq, Wc);
        else if (XM == 2) cells<2, YM>(w, Q, nQ, P, nP, cq, Wc);
        else cells<3, YM>(w, Q, nQ, P, nP, cq, Wc);
        // relative classes
        const float A0 = __fmaf_rn(Wc[2][2], v[2][2], __fmaf_rn(Wc[2][0], v[2][0], __fmaf_rn(Wc[0][2], v[0][2], __fmul_rn(Wc[0][0], v[0][0]))));
        const float A1 = __fmaf_rn(Wc[2][1], v[2][1], __fmul_rn(Wc[0][1], v[0][1]));
        const float A2 = __fmaf_rn(Wc[1][2], v[1][2], __fmul_rn(Wc[1][0], v[1][0]));
        const float A3 = __fmul_rn(Wc[1][1], v[1][1]);
        const float W0 = __fadd_rn(__fadd_rn(Wc[0][0], Wc[0][2]), __fadd_rn(Wc[2][0], Wc[2][2]));
        const float W1 = __fadd_rn(Wc[0][1], Wc[2][1]);
        const float W2 = __fadd_rn(Wc[1][0], Wc[1][2]);
        const float W3 = Wc[1][1];
        // relative classes -> R, G, B
        const float NA0 = hG ? A1 : A0, NA1 = hG ? A2 : A3, NW0 = hG ? W1 : W0, NW1 = hG ? W2 : W3;
        const float ga = __fadd_rn(hG ? A0 : A1, hG ? A3 : A2), gw = __fadd_rn(hG ? W0 : W1, hG ? W3 : W2);
        const float ra = frr ? NA0 : NA1, ba = frr ? NA1 : NA0, rw = frr ? NW0 : NW1, bw = frr ? NW1 : NW0;
        a[0] = __fmaf_rn(__fmaf_rn(-A.black.v[0], rw, ra), A.rwhite.v[0], a[0]);
        a[1] = __fmaf_rn(__fmaf_rn(-A.black.v[1], gw, ga), A.rwhite.v[1], a[1]);
        a[2] = __fmaf_rn(__fmaf_rn(-A.black.v[2], bw, ba), A.rwhite.v[2], a[2]);
        ws[0] = __fadd_rn(ws[0], rw);
        ws[1] = __fadd_rn(ws[1], gw);
        ws[2] = __fadd_rn(ws[2], bw);
    }
    return f;
}

template <bool SANE>
__global__ void __launch_bounds__(X2_NT, X2_CTAS) k_accumulate_x2(const __grid_constant__ X2Args A)
{
    __shared__ float so[X2_ROWS][2][3 * X2_W];
    const isa_accum_geom& g = A.g;
    const int tid = threadIdx.x % X2_W, lane = tid & 31, ph = tid >> 5, part = threadIdx.x / X2_W;
    // blocks in bands of 32 rows, eight CTA rows each, two per y mod 4: the CTAs of an SM run the same code
    const int nbx = (g.Wo + X2_W - 1) / X2_W;
    const int row = blockIdx.x / nbx, r = row & 7;
    const int x0 = (blockIdx.x - row * nbx) * X2_W, y = g.yb0 + 4 * (row & ~7) + 4 * (4 * (r & 1) + part) + (r >> 1);
    const bool yin = y < g.yb1;
    const int nx = yin ? 3 * min(X2_W, g.Wo - x0) : 0;
    float* arow = isa::row_ptr(A.acc, A.out_pitch, y) + 3 * x0;
    float* wrow = isa::row_ptr(A.wsum, A.out_pitch, y) + 3 * x0;
    if (A.accumulate_into) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int i = tid + k * X2_W;
            if (i < nx) { so[part][0][i] = arow[i]; so[part][1][i] = wrow[i]; }
        }
        __syncthreads();
    }
    const int lx = 4 * lane + ph, x = x0 + lx;
    if (yin && x < g.Wo) {
        float a[3] = {0.f, 0.f, 0.f}, ws[3] = {0.f, 0.f, 0.f};
        if (A.accumulate_into) {
#pragma unroll
            for (int c = 0; c < 3; c++) { a[c] = so[part][0][3 * lx + c]; ws[c] = so[part][1][3 * lx + c]; }
        }
        if (x >= 1 && y >= 1 && x < g.Wo - 1 && y < g.Ho - 1) {
            const int X = x + g.ox, Y = y + g.oy;
            const Position p = position(g, x, y);
            float k0, k1, k2, w[5][5];
            kernel_params(A, p, k0, k1, k2);
            const float wmax = tap_weights(k0, k1, k2, w);
            // the unshifted taps' mask cells are (X - 2) >> 2 + {0, 1} inside the crop, rows alike, the crop holds a 3 x 3
            // block, and the flow's four texels lie in the frame
            const bool interior = ((X - 2) >> 1) >= g.cx0 && ((X + 2) >> 1) <= g.cx1 && ((Y - 2) >> 1) >= g.cy0 && ((Y + 2) >> 1) <= g.cy1 &&
                                  g.cx1 - g.cx0 >= 2 && g.cy1 - g.cy0 >= 2 && p.ib >= 0 && p.ib + 1 < g.W && p.jb >= 0 && p.jb + 1 < g.H &&
                                  wmax < 1e30f;
            for (int f = 0;; f++) {
                switch (Y & 3) {  // the same for the whole CTA
                case 0: f = frames_x2<0, SANE>(A, f, x, y, w, interior, a, ws); break;
                case 1: f = frames_x2<1, SANE>(A, f, x, y, w, interior, a, ws); break;
                case 2: f = frames_x2<2, SANE>(A, f, x, y, w, interior, a, ws); break;
                default: f = frames_x2<3, SANE>(A, f, x, y, w, interior, a, ws); break;
                }
                if (f >= A.nframes) break;
                const Sums s = frame_per_tap<2, true>(A, f, x, y);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    a[c] += (s.a[c] - A.black.v[c] * s.w[c]) * A.rwhite.v[c];
                    ws[c] += s.w[c];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) { so[part][0][3 * lx + c] = a[c]; so[part][1][3 * lx + c] = ws[c]; }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int i = tid + k * X2_W;
        if (i < nx) { arow[i] = so[part][0][i]; wrow[i] = so[part][1][i]; }
    }
}

// ---- scale 1 (accumulateImages) ------------------------------------------------
// Output pixel (X, Y) reads the 5 x 5 samples around (X + sx, Y + sy), each
// with the certainty of the unshifted tap's mask cell: 3 x 3 cells, the taps
// of a line on cells 0 0 1 1 2 where X is even and 0 1 1 2 2 where it is odd.
// Relative to the block's first sample a tap's CFA class is its own parity, a
// compile-time constant; the certainty of a class is one of two values per
// mask cell and row parity. Row patterns (YM = Y mod 2) are a template
// parameter, uniform in a CTA; the column pattern is a select per lane.
// Black comes off each sample (see k_accumulate); SAME: one level for all
// channels, a constant instead of four selected ones (and their spills).
// Bound: issue and the loads' latency, 385 instructions per pixel and frame over
// 8 frames (100 additions and multiply-adds, about as many selects and loads) at
// an IPC of 2.2, 26 of 64 warps. 12 x 4000x3000: 2.74 ms, from 15.9 ms tap by tap
// with its clamps, divisions and indexed channels; one 3010x2006 frame by
// itself 0.22 ms, from 0.72 ms. CTAs of 512 threads: 2.9 ms and 0.24 ms; at 80
// registers (24 warps per SM) 3.0 ms.
constexpr int X1_NT = 2 * X2_W, X1_CTAS = 4;

template <int YM, bool SANE, bool SAME>
__device__ __forceinline__ int frames_x1(const X2Args& A, int f0, int X, int Y, const float (&w)[5][5], bool interior, float (&a)[3], float (&ws)[3])
{
    const isa_accum_geom& g = A.g;
    const unsigned foff = (unsigned)isa::clampi(Y, 0, g.H - 1) * (unsigned)A.flow_pitch + (unsigned)isa::clampi(X, 0, g.W - 1) * 8u;
    const unsigned moff = (unsigned)isa::clampi((Y - 2) >> 1, 0, g.H / 2 - 1) * (unsigned)A.mask_pitch + (unsigned)isa::clampi((X - 2) >> 1, 0, g.W / 2 - 1) * 16u;
    // the shifted 5 x 5 block lies inside the crop
    const unsigned kspan = (unsigned)(g.cx1 - 4 - g.cx0), jspan = (unsigned)(g.cy1 - 4 - g.cy0);
    const bool odd = X & 1;
    int f = f0;
#pragma unroll 1
    for (; f < A.nframes; f++) {
        int sx = 0, sy = 0;
        if (A.frames[f].flow) {
            const float2 fl = __ldg((const float2*)((const char*)A.frames[f].flow + foff));
            sx = (int)roundf(fl.x);
            sy = (int)roundf(fl.y);
        }
        const int k0 = X + sx - 2, j0 = Y + sy - 2;
        if (!(interior && (unsigned)(k0 - g.cx0) <= kspan && (unsigned)(j0 - g.cy0) <= jspan)) break;
        const unsigned ro = (unsigned)j0 * (unsigned)A.raw_pitch + 2u * (unsigned)k0;
        const char* mk = (const char*)A.frames[f].mask;
        const unsigned mo = mk ? moff : 0u;
        const size_t mp = mk ? A.mask_pitch : 0;
        const char* mb = mk ? mk : (const char*)g_unit_mask;
        const bool fx = k0 & 1, fy = j0 & 1;
        const bool hG = (int)(fx ^ fy) == A.bayer.g0, frr = (int)fy == A.bayer.ry;
        const float b1 = frr ? A.black.v[0] : A.black.v[2], b2 = frr ? A.black.v[2] : A.black.v[0], bg = A.black.v[1];
        const float bl[4] = {hG ? bg : b1, hG ? b1 : bg, hG ? b2 : bg, hG ? bg : b2};  // of the relative classes
        float Ac[4] = {0.f, 0.f, 0.f, 0.f}, Wc[4] = {0.f, 0.f, 0.f, 0.f};
        float4 M[3];
#pragma unroll
        for (int r = 0; r < 5; r++) {
            constexpr int MR[2][5] = {{0, 0, 1, 1, 2}, {0, 1, 1, 2, 2}};
            if (r == 0 || MR[YM][r] != MR[YM][r > 0 ? r - 1 : 0]) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    M[c] = __ldg((const float4*)(mb + MR[YM][r] * mp + mo) + c);
                    if (!SANE) M[c] = sanitize(M[c]);
                }
            }
            const int rp = r & 1;
            const bool red = rp ? !frr : frr, gE = rp ? !hG : hG;  // the row's other colour; green on its even taps
            float E[3], O[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const float rb = red ? M[c].x : M[c].z;
                E[c] = gE ? M[c].y : rb;
                O[c] = gE ? rb : M[c].y;
            }
            const float k[5] = {E[0], odd ? O[1] : O[0], E[1], odd ? O[2] : O[1], E[2]};
            const uint16_t* rr = (const uint16_t*)((const char*)A.frames[f].raw + r * A.raw_pitch + ro);
#pragma unroll
            for (int d = 0; d < 5; d++) {
                const float wc = __fmul_rn(w[r][d], k[d]);
                const int cl = rp * 2 + (d & 1);
                const float v = __fsub_rn((float)__ldg(rr + d), SAME ? A.black.v[0] : bl[cl]);
                Ac[cl] = __fmaf_rn(wc, v, Ac[cl]);
                Wc[cl] = __fadd_rn(Wc[cl], wc);
            }
        }
        // relative classes -> R, G, B
        const float NA0 = hG ? Ac[1] : Ac[0], NA1 = hG ? Ac[2] : Ac[3], NW0 = hG ? Wc[1] : Wc[0], NW1 = hG ? Wc[2] : Wc[3];
        const float ga = (hG ? Ac[0] : Ac[1]) + (hG ? Ac[3] : Ac[2]), gw = (hG ? Wc[0] : Wc[1]) + (hG ? Wc[3] : Wc[2]);
        const float ra = frr ? NA0 : NA1, ba = frr ? NA1 : NA0, rw = frr ? NW0 : NW1, bw = frr ? NW1 : NW0;
        a[0] = __fmaf_rn(ra, A.rwhite.v[0], __fmaf_rn(ra, A.rwlow.v[0], a[0]));
        a[1] = __fmaf_rn(ga, A.rwhite.v[1], __fmaf_rn(ga, A.rwlow.v[1], a[1]));
        a[2] = __fmaf_rn(ba, A.rwhite.v[2], __fmaf_rn(ba, A.rwlow.v[2], a[2]));
        ws[0] += rw;
        ws[1] += gw;
        ws[2] += bw;
    }
    return f;
}

template <bool SANE, bool SAME>
__global__ void __launch_bounds__(X1_NT, X1_CTAS) k_accumulate_x1(const __grid_constant__ X2Args A)
{
    const isa_accum_geom& g = A.g;
    // CTA rows in bands of four output rows: the two even rows, then the two odd ones
    const int nbx = (g.Wo + X2_W - 1) / X2_W;
    const int row = blockIdx.x / nbx;
    const int x = (blockIdx.x - row * nbx) * X2_W + threadIdx.x % X2_W;
    const int y = g.yb0 + 4 * (row >> 1) + 2 * (threadIdx.x / X2_W) + (row & 1);
    if (x >= g.Wo || y >= g.yb1) return;
    float* ap = isa::row_ptr(A.acc, A.out_pitch, y) + 3 * x;
    float* wp = isa::row_ptr(A.wsum, A.out_pitch, y) + 3 * x;
    if (x < 1 || y < 1 || x >= g.Wo - 1 || y >= g.Ho - 1) {
        if (!A.accumulate_into) { ap[0] = ap[1] = ap[2] = 0.f; wp[0] = wp[1] = wp[2] = 0.f; }
        return;
    }
    float a[3] = {0.f, 0.f, 0.f}, ws[3] = {0.f, 0.f, 0.f};
    if (A.accumulate_into) {
#pragma unroll
        for (int c = 0; c < 3; c++) { a[c] = ap[c]; ws[c] = wp[c]; }
    }
    const int X = x + g.ox, Y = y + g.oy;
    const float4 kp = __ldg(isa::row_ptr(A.kparam, A.kp_pitch, isa::clampi(Y, 0, g.H - 1)) + isa::clampi(X, 0, g.W - 1));
    float w[5][5];
    const float wmax = tap_weights(kp.x, kp.y, kp.z, w);
    // the unshifted taps lie inside the crop (and with them the flow's texel in the frame), the crop holds a 5 x 5 block
    const bool interior = X - 2 >= g.cx0 && X + 2 <= g.cx1 && Y - 2 >= g.cy0 && Y + 2 <= g.cy1 && wmax < 1e30f;
    for (int f = 0;; f++) {
        if ((Y & 1) == 0) f = frames_x1<0, SANE, SAME>(A, f, X, Y, w, interior, a, ws);  // the same for the whole CTA
        else f = frames_x1<1, SANE, SAME>(A, f, X, Y, w, interior, a, ws);
        if (f >= A.nframes) break;
        const Sums s = frame_per_tap<1, SAME>(A, f, x, y);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            a[c] += s.a[c];
            ws[c] += s.w[c];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) { ap[c] = a[c]; wp[c] = ws[c]; }
}

// The CFA is a Bayer pattern: codes 0/1/2 only, the two greens on one
// diagonal, red and blue on the other.
bool bayer_of(unsigned cfa, Bayer& b)
{
    int c[4];
    for (int i = 0; i < 4; i++) c[i] = (cfa >> (2 * i)) & 3;  // index = row parity * 2 + column parity
    if (c[1] == 1 && c[2] == 1 && c[0] != 1 && c[3] != 1 && c[0] != c[3]) {
        b.g0 = 1;
        b.ry = c[0] == 0 ? 0 : 1;
        return (c[0] == 0 || c[0] == 2) && (c[3] == 0 || c[3] == 2);
    }
    if (c[0] == 1 && c[3] == 1 && c[1] != 1 && c[2] != 1 && c[1] != c[2]) {
        b.g0 = 0;
        b.ry = c[1] == 0 ? 0 : 1;
        return (c[1] == 0 || c[1] == 2) && (c[2] == 0 || c[2] == 2);
    }
    return false;
}

}  // namespace

// Merge scales 1 and 2 of a Bayer layout, frames whose byte offsets fit 32 bits (the kernels' address arithmetic).
bool isa_accumulate_bayer_supported(const isa_accum_geom& g, unsigned cfa, int nframes, size_t raw_pitch, size_t flow_pitch, size_t mask_pitch)
{
    Bayer b;
    const unsigned long long lim = 1ull << 32, H = (unsigned long long)g.H;
    return (g.s_int == 1 || g.s_int == 2) && bayer_of(cfa, b) && nframes <= ISA_ACC_MAX_FRAMES && g.W >= 4 && g.H >= 4 && H * raw_pitch < lim &&
           H * flow_pitch < lim && H / 2 * mask_pitch < lim;
}

cudaError_t isa_launch_accumulate_bayer(const isa_accum_geom& g, unsigned cfa, const isa_frame_in* frames, int nframes, size_t raw_pitch,
                                        size_t flow_pitch, size_t mask_pitch, const float* kparam, size_t kparam_pitch, const float* white,
                                        const float* black, float* acc, float* wsum, size_t out_pitch, int accumulate_into, cudaStream_t st)
{
    X2Args A;
    if (!bayer_of(cfa, A.bayer) || nframes < 0 || nframes > ISA_ACC_MAX_FRAMES) return cudaErrorInvalidValue;
    A.g = g;
    A.cfa = cfa;
    A.nframes = nframes;
    for (int f = 0; f < nframes; f++) A.frames[f] = frames[f];
    A.raw_pitch = raw_pitch; A.flow_pitch = flow_pitch; A.mask_pitch = mask_pitch;
    A.kparam = (const float4*)kparam; A.kp_pitch = kparam_pitch;
    A.lv = isa_make_levels(white, black);
    for (int c = 0; c < 3; c++) {
        A.rwhite.v[c] = g.s_int == 2 ? (float)(1.0 / (double)white[c]) : A.lv.rhigh[c] * A.lv.scale;
        A.rwlow.v[c] = A.lv.rlow[c] * A.lv.scale;
        A.black.v[c] = black[c];
    }
    A.acc = acc; A.wsum = wsum; A.out_pitch = out_pitch; A.accumulate_into = accumulate_into;
    if (g.yb0 % 32 || g.yb0 < 0 || g.yb1 > g.Ho || g.yb1 <= g.yb0) return cudaErrorInvalidValue;
    const int rows = g.yb1 - g.yb0;  // CTA rows: four rows each in bands of 32, or two each in bands of 4
    const long long blocks = (long long)((g.Wo + X2_W - 1) / X2_W) * (g.s_int == 2 ? (rows + 31) / 32 * 8 : (rows + 3) / 4 * 2);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const auto kernel = g.s_int == 2 ? (g.masks_finite ? k_accumulate_x2<true> : k_accumulate_x2<false>)
                        : A.lv.same_black ? (g.masks_finite ? k_accumulate_x1<true, true> : k_accumulate_x1<false, true>)
                                          : (g.masks_finite ? k_accumulate_x1<true, false> : k_accumulate_x1<false, false>);
    kernel<<<(unsigned)blocks, g.s_int == 2 ? X2_NT : X1_NT, 0, st>>>(A);
    return cudaGetLastError();
}
