// pm_slots.cu -- CheckerboardUpdateFrame (MIStereo/AdaptMIPMFrame.cu:520-947)
// with pixel slots and pooled NCC evaluations.
//
// A CTA stages one micro-image and its neighbours and keeps up to 32 of its
// pixels in flight, one slot (half a warp) each.  It runs in rounds: every slot
// carries its pixel to the next point where costs are needed (the propagation
// candidates; the cross-view proposals and refinement candidates; a proposal or
// the candidates rebuilt because an earlier proposal won; the completion of the
// winner's cost vector), and puts the (hypothesis, neighbour) NCCs it needs into
// one list.  The list is sorted by the size of each NCC's tap rectangle, and the
// CTA's warps evaluate it 32 NCCs at a time, one per lane, whichever pixels they
// belong to.  A slot whose pixel is finished takes the next one.
//
// The tap rectangle of an NCC is the pixel's patch window cut down to the taps
// whose source sample can lie in the neighbour window under the hypothesis; a
// lane walks its own rectangle from its own origin, x offset outer, y offset
// inner, so each NCC keeps the reference's accumulation order, and a tap whose
// sample leaves the window adds nothing, as the reference skips it.
//
// Why: one pixel's NCCs fill 73% of the lanes of whole warps and the taps inside
// both windows 41-57% of a warp's tap slots; pooled over the slots and sorted,
// the lanes are full and 92% of the slots carry a tap of the lane's rectangle
// (500 warp-taps per pixel instead of 860, 2048x1536, 12 neighbours, 15x15).  The
// scalar code runs on half warps, the two halves of a warp on the same stage.
// Bound by instruction issue: a warp-tap is about 36 instructions (3 loads, 16
// FP32 operations, 6 integer products, 8 logical operations); packed pairs
// (f32x2) halve the issue slots of the coordinates, measured 3% of the sweep, and
// predicated sums take the place of selected zeros, 12% (with a blur channel 15%).
// The scalar code is bound by latency: what it took from a round was mostly chains of
// shuffles and loops that every lane ran.  So a plane, view, draw or candidate is one
// lane's wherever its order does not matter, the ordered sums read shared memory, the
// weight tables are filled by all warps and the finished pixels written by one.  Every
// lane on the loops -> one lane each: 28.7 -> 27.3 ms, 4.1 -> 3.6, 16.7 -> 10.6.
// Half-sweep, warp per pixel -> slots: 41 -> 23.4 ms (2048x1536, 12 neighbours,
// 15x15), 8.0 -> 3.2 ms (1024x768, 6, 11x11), 27 -> 9.6 ms (2048x1536, ACMM, 5x5).
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>
#include "pm_device.cuh"
#include "pm_kernels.h"
#include "pm_sweep_device.cuh"
#include "smem_limit.h"

namespace pfd {

namespace {

// Launch shapes: warps per CTA and CTAs per SM.  Shape 0, the default, is the
// fastest where two CTAs fit (2048x1536, 12 neighbours, 15x15: 23.5 ms, 12x2 24.4, 8x3
// 24.7, 16x1 27.5); one CTA with all the shared memory and registers (shape 3) where
// the quads of a blur channel leave two CTAs few slots (one_cta_shape).
template <int S> struct ShapeOf;
template <> struct ShapeOf<0> { static constexpr int warps = 16, min_ctas = 2; };
template <> struct ShapeOf<1> { static constexpr int warps = 12, min_ctas = 2; };
template <> struct ShapeOf<2> { static constexpr int warps = 8, min_ctas = 3; };
template <> struct ShapeOf<3> { static constexpr int warps = 16, min_ctas = 1; };
constexpr int kShapeWarps[kSweepShapes] = { ShapeOf<0>::warps, ShapeOf<1>::warps, ShapeOf<2>::warps, ShapeOf<3>::warps };
constexpr int kShapeCtas[kSweepShapes] = { ShapeOf<0>::min_ctas, ShapeOf<1>::min_ctas, ShapeOf<2>::min_ctas,
                                           ShapeOf<3>::min_ctas };

// What a slot keeps of its pixel between rounds.
struct __align__(16) SlotState {
    float4 best_plane;       // best plane so far
    float4 c0, rn;           // refinement draws: random plane, random normal
    float4 u;                // u1-u3 (perturbed normal), u4 (perturbed depth)
    uint64_t skip;           // request: rows not to be evaluated
    uint32_t slots;          // row of propagation slot s in bits [4s, 4s + 4)
    uint32_t tsel;           // selected views
    float best_cost;
    float best_d;            // disparity of the best plane at the pixel
    int best_min;            // view of the lowest cost of the best plane
    int best_row;            // 0: the current plane is still the best
    int row_lo, row_hi;      // request: rows
    int n_views;             // request: views; the first n_views entries of the slot's list, or every view (-1)
    int xy;                  // x | y << 8
    int r0;                  // row of the first refinement candidate
    int n, hs;               // walk over the proposals: next one, its speculative row
    uint32_t flags;          // candidate flags (bits 0-7), kFlag*
};
// A finished pixel's new state on its way to memory (xy -1: none).
struct __align__(16) SlotOut {
    float4 plane;
    float cost, d;
    uint32_t sel;
    int xy_view;             // x | y << 8 | (view of disp + 1) << 16, or -1
};
constexpr uint32_t kFlagChanged = 0x100u, kFlagPartial = 0x200u, kFlagSkip3 = 0x400u;

// Where a slot's pixel stands: what the evaluation in flight is for.
enum Stage : int { kIdle = 0, kNew, kProp, kSpec, kWalk, kRedo, kComplete, kWaits = 16, kFresh = 32 };

// Hypotheses one slot can hold: 9 propagation rows, or every selected view's
// proposal, the 5 refinement candidates and one rebuilt proposal.
__host__ __device__ inline int slot_rows(int K) { return K + 6 > 9 ? K + 6 : 9; }
// NCCs one request can ask for.
__host__ __device__ inline int slot_tasks(int K) { return slot_rows(K) * K; }

// Control words.
enum Ctl : int { kCtlItem = 0, kCtlPixel, kCtlTasks, kCtlPass, kCtlWords = 8 };

struct SlotPlan {
    int off_ctl, off_Q, off_QB, off_R, off_RB, off_geo, off_ok, off_as, off_ac, off_pc, off_ps, off_bins, off_id, off_order;
    int off_stage, off_wtab, off_plane, off_dp, off_cost, off_bvec, off_wgt, off_wres, off_wmin, off_aux, off_sel, off_state,
        off_out, off_stages;
    int rs, tx, ty, tab_n, rows, nbins, total;

    __host__ __device__ static int a16(int v) { return (v + 15) & ~15; }
    __host__ __device__ static SlotPlan make(int W, int H, int K, int ntap, bool blur, int tile_stride, int slots, int cap)
    {
        SlotPlan p;
        p.rs = H | 1;                                    // odd: columns start in different banks
        p.tx = ntap < W ? ntap : W;
        p.ty = ntap < H ? ntap : H;
        p.tab_n = p.tx * p.ty;
        p.rows = slot_rows(K);
        p.nbins = (p.tx / 2 + 1) * p.ty;
        int o = 16;                                      // the staging barrier is at offset 0 of every plan
        p.off_ctl = o;   o += kCtlWords * 4;
        const int q_bytes = a16(K * (H + 1) * (W + 1) * 4), r_bytes = a16((2 * W * p.rs + 2 * H) * 4);
        p.off_Q = o;     o += q_bytes;
        p.off_QB = o;    o += blur ? q_bytes : 0;
        p.off_R = o;     o += r_bytes;
        p.off_RB = o;    o += blur ? r_bytes : 0;
        p.off_geo = o;   o += a16(K * (int)sizeof(NbGeo));
        p.off_ok = o;    o += a16(K * 4);
        p.off_as = o;    o += a16(ntap * ntap * 4);
        p.off_ac = o;    o += 256 * 4;
        p.off_pc = o;    o += a16(W * H * 4);
        p.off_ps = o;    o += a16(W * H * 4);
        p.off_bins = o;  o += a16(p.nbins * 4);
        // the staging buffer shares what follows: it is filled and read only between
        // views, while no slot holds a pixel
        p.off_stage = o;
        const int stage_end = o + a16((1 + K) * tile_stride * (blur ? 2 : 1));
        p.off_wtab = o;  o += a16(slots * p.tab_n * 4);
        p.off_plane = o; o += slots * p.rows * 16;
        p.off_dp = o;    o += slots * p.rows * 16;
        p.off_cost = o;  o += a16(slots * p.rows * K * 4);
        p.off_bvec = o;  o += a16(slots * K * 4);
        p.off_wres = o;  o += a16(slots * p.rows * 4);
        p.off_wmin = o;  o += a16(slots * p.rows * 4);
        p.off_wgt = o;   o += a16(slots * K * 4);
        p.off_aux = o;   o += a16(slots * K * 2);
        p.off_sel = o;   o += a16(slots * K);
        p.off_state = o; o += slots * (int)sizeof(SlotState);
        p.off_out = o;   o += slots * (int)sizeof(SlotOut);
        p.off_stages = o; o += 64 * 4;
        p.off_id = o;    o += a16(cap * 2);
        p.off_order = o; o += a16(cap * 2);
        // a lane that walks past its own rectangle reads at most one window past the tables
        const int walk_end = p.off_wtab + (slots + 1) * p.tab_n * 4 + 64;
        if (o < stage_end) o = stage_end;
        if (o < walk_end) o = a16(walk_end);
        p.total = o;
        return p;
    }
};

// ---- packed pairs of single-precision values: two taps per instruction ----------
// Each half is the IEEE operation of the scalar instruction.
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2_rn(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t fma2_rm(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2_rn(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float lds_f32(uint32_t addr)
{
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// sb / 255 for sb = k / 256, 0 <= k < 2^16: the product with the rounded
// reciprocal and one fused correction give the correctly rounded quotient
// (division by a constant, Brisebarre and Muller), checked for all 2^16 values.
__device__ __forceinline__ float div255(float sb)
{
    const float r = 0x1.010102p-8f;                      // 1 / 255 rounded
    const float q = __fmul_rn(sb, r);
    return __fmaf_rn(__fmaf_rn(-q, 255.0f, sb), r, q);
}

// a / -0.18f, correctly rounded: the product with the rounded reciprocal and one fused
// correction (Markstein); for a 0 or in the normal range.
__device__ __forceinline__ float div_m018(float a)
{
    constexpr float v = -0.18f, y = 1.0f / -0.18f;
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-q, v, a), y, q);
}

// The six moment sums of one NCC (and the blur sums).
struct Moments {
    float sr, srr, ss, sss, srs, sw, bsx, bsy;
};

// Whether a sample position lies in the neighbour window (its bits compare below the
// window's), for the instructions that follow in the same statement.
#define PFD_IN_WINDOW(sx, sy, w, h) ".reg .pred v;\n\tsetp.lt.u32 v, " sx ", " w ";\n\tsetp.lt.and.u32 v, " sy ", " h ", v;\n\t"

// q = the word at q where the position is inside; otherwise q is unchanged.
__device__ __forceinline__ uint32_t lds_if(uint32_t q, float sx, float sy, uint32_t wb, uint32_t hb)
{
    asm("{\n\t" PFD_IN_WINDOW("%1", "%2", "%3", "%4") "@v ld.shared.u32 %0, [%0];\n\t}"
        : "+r"(q) : "r"(__float_as_uint(sx)), "r"(__float_as_uint(sy)), "r"(wb), "r"(hb));
    return q;
}

// One tap: sample position (sx, sy) with its texture coordinates (tx, ty), the
// tap's weight w and reference texel r.  A tap outside the neighbour window
// (wb 0: always outside) adds nothing: its load and its sums are predicated, two
// selects per tap less than adding zeros.
template <bool BLUR, bool SHIFT>
__device__ __forceinline__ void tap(Moments& M, float sx, float sy, float tx, float ty, float w, float r, float rb,
                                    float sh, uint32_t wb, uint32_t hb, uint32_t base, uint32_t kq, uint32_t qb_delta)
{
    // (a, b, ix, iy) in the four bytes; the entry's address is base + 4 ix + row iy
    const uint32_t p = __byte_perm(__float_as_uint(tx), __float_as_uint(ty), 0x5140);
    const uint32_t addr = __dp4a(p, kq, base);
    const uint32_t a = __float_as_uint(tx) & 0xFFu, b = __float_as_uint(ty) & 0xFFu;
    const uint32_t w11 = (a * b + 128u) >> 8;
    const uint32_t hi = w11 * 65535u + b;
    const uint32_t lo = a * 65535u + 256u - hi;
    const uint32_t q = lds_if(addr, sx, sy, wb, hb);
    float s = __fsub_rn(__uint_as_float(__dp2a_lo(lo, q, __dp2a_hi(hi, q, 0x47000000u))), 32768.0f);
    if (SHIFT) { s = __fsub_rn(s, sh); r = __fsub_rn(r, sh); }
    const float wr = __fmul_rn(w, r), ws = __fmul_rn(w, s);
    asm("{\n\t" PFD_IN_WINDOW("%11", "%12", "%13", "%14")
        "@v fma.rn.f32 %0, %6, %7, %0;\n\t"
        "@v fma.rn.f32 %1, %9, %7, %1;\n\t"
        "@v fma.rn.f32 %2, %6, %8, %2;\n\t"
        "@v fma.rn.f32 %3, %10, %8, %3;\n\t"
        "@v fma.rn.f32 %4, %9, %8, %4;\n\t"
        "@v add.rn.f32 %5, %5, %6;\n\t}"
        : "+f"(M.sr), "+f"(M.srr), "+f"(M.ss), "+f"(M.sss), "+f"(M.srs), "+f"(M.sw)
        : "f"(w), "f"(r), "f"(s), "f"(wr), "f"(ws), "r"(__float_as_uint(sx)), "r"(__float_as_uint(sy)), "r"(wb), "r"(hb));
    if (BLUR) {
        const uint32_t qb = lds_if(addr + qb_delta, sx, sy, wb, hb);
        const float sb = __fsub_rn(__uint_as_float(__dp2a_lo(lo, qb, __dp2a_hi(hi, qb, 0x47000000u))), 32768.0f);
        const float db = div255(sb);
        asm("{\n\t" PFD_IN_WINDOW("%4", "%5", "%6", "%7")
            "@v add.rn.f32 %0, %0, %2;\n\t@v add.rn.f32 %1, %1, %3;\n\t}"
            : "+f"(M.bsx), "+f"(M.bsy)
            : "f"(rb), "f"(db), "r"(__float_as_uint(sx)), "r"(__float_as_uint(sy)), "r"(wb), "r"(hb));
    }
}

// The NCC cost of its moments (ComputeBilateralNCC_Frame, AdaptMIPMFrame.cu:140-179).
template <bool BLUR>
__device__ __forceinline__ float ncc_cost(const Moments& M, float blur_gain)
{
    float c = kCostMax;
    if (M.sw > 1e-6f) {
        const float inv = __fdiv_rn(1.0f, M.sw);
        const float m_r = __fmul_rn(M.sr, inv), m_rr = __fmul_rn(M.srr, inv);
        const float m_s = __fmul_rn(M.ss, inv), m_ss = __fmul_rn(M.sss, inv);
        const float m_rs = __fmul_rn(M.srs, inv);
        const float var_r = __fmaf_rn(-m_r, m_r, m_rr);
        const float var_s = __fmaf_rn(-m_s, m_s, m_ss);
        if (!(var_r < 1e-5f || var_s < 1e-5f)) {
            const float cov = __fmaf_rn(-m_r, m_s, m_rs);
            const float vv = __fsqrt_rn(__fmul_rn(var_r, var_s));
            c = clamp_cost(__fsub_rn(1.0f, __fdiv_rn(cov, vv)));
        }
    }
    if (BLUR) {
        const float tb = __fsub_rn(M.bsx, M.bsy);
        const float bw = pfd_expf(__fmul_rn(__fmul_rn(-0.007368f, tb), tb));
        c = clamp_cost(__fmaf_rn(blur_gain, __fsub_rn(1.0f, bw), c));
    }
    return c;
}

// What the evaluation of a list entry reads, as shared-window addresses.
struct EvalEnv {
    uint32_t wtab, R, RB_delta, Q, QB_delta;
    int q_bytes, tab_n, rs, inc;
    uint32_t wb, hb, kq;
};

// One lane's NCC: the rectangle's tap columns and rows (nx, ny; 0 for a lane
// without an entry), the addresses of its first tap (weight wa, reference texel
// ra), the weight table's column step wstep in bytes, its first tap position
// (fx, fy) and the neighbour's quads (base).  All lanes walk the widest and
// tallest rectangle of the warp; taps past a lane's own rectangle add nothing.
// Two taps per iteration, their coordinates in packed pairs.
template <bool BLUR, bool SHIFT>
__device__ __forceinline__ void walk(Moments& M, const EvalEnv& E, float3 dp, float stx, float sty, int nx, int ny,
                                     uint32_t wa, uint32_t ra, uint32_t wstep, float fx, float fy, uint32_t base, float sh)
{
    const int NX = __reduce_max_sync(kFullMask, nx), NY = __reduce_max_sync(kFullMask, ny);
    const int NYm = __reduce_min_sync(kFullMask, nx > 0 ? ny : NY);      // rows every lane with an entry keeps
    const float finc = (float)E.inc;
    const uint32_t rinc = (uint32_t)E.inc * 4u, rstep = (uint32_t)(E.inc * E.rs) * 4u;
    const uint64_t dpy2 = pack2(dp.y, dp.y), dpz2 = pack2(dp.z, dp.z), stx2 = pack2(stx, stx), sty2 = pack2(sty, sty);
    const uint64_t half2 = pack2(0.5f, 0.5f), scale2 = pack2(256.0f, 256.0f), magic2 = pack2(8388480.5f, 8388480.5f);
    const uint64_t fy_start = pack2(fy, __fadd_rn(fy, finc)), fy_step = pack2(2.0f * finc, 2.0f * finc);
    for (int ix = 0; ix < NX; ++ix) {
        // a lane past its last column gets no sample position inside the window
        const float axr = ix < nx ? __fmul_rn(dp.x, fx) : __int_as_float(0x7fffffff);
        const uint64_t axr2 = pack2(axr, axr), fx2 = pack2(fx, fx);
        uint64_t fy2 = fy_start;
        uint32_t wp = wa, rp = ra;
        int iy = 0;
        auto pair = [&](uint32_t wb0, uint32_t wb1) {
            const uint64_t d2 = add2_rn(fma2_rn(dpy2, fy2, axr2), dpz2);
            const uint64_t sx2 = fma2_rn(stx2, d2, fx2), sy2 = fma2_rn(sty2, d2, fy2);
            const uint64_t tx2 = fma2_rm(add2_rn(sx2, half2), scale2, magic2);
            const uint64_t ty2 = fma2_rm(add2_rn(sy2, half2), scale2, magic2);
            float sx0, sx1, sy0, sy1, tx0, tx1, ty0, ty1;
            unpack2(sx2, sx0, sx1);
            unpack2(sy2, sy0, sy1);
            unpack2(tx2, tx0, tx1);
            unpack2(ty2, ty0, ty1);
            const float w0 = lds_f32(wp), w1 = lds_f32(wp + 4u);
            const float r0 = lds_f32(rp), r1 = lds_f32(rp + rinc);
            const float b0 = BLUR ? lds_f32(rp + E.RB_delta) : 0.0f, b1 = BLUR ? lds_f32(rp + rinc + E.RB_delta) : 0.0f;
            tap<BLUR, SHIFT>(M, sx0, sy0, tx0, ty0, w0, r0, b0, sh, wb0, E.hb, base, E.kq, E.QB_delta);
            tap<BLUR, SHIFT>(M, sx1, sy1, tx1, ty1, w1, r1, b1, sh, wb1, E.hb, base, E.kq, E.QB_delta);
            fy2 = add2_rn(fy2, fy_step);
            wp += 8u;
            rp += 2u * rinc;
        };
        for (; iy + 2 <= NYm; iy += 2) pair(E.wb, E.wb);
        // rows that some lanes keep: in pairs too (24.3 -> 23.9 ms, 2048x1536, 15x15), except
        // with a blur channel, where the registers do not suffice (22.0 -> 23.7 ms)
        if (!BLUR)
            for (; iy + 2 <= NY; iy += 2) pair(iy < ny ? E.wb : 0u, iy + 1 < ny ? E.wb : 0u);
        float fyr, fyr1;
        unpack2(fy2, fyr, fyr1);
        auto one = [&]() {
            const float d = __fadd_rn(__fmaf_rn(dp.y, fyr, axr), dp.z);
            const float sx = __fmaf_rn(stx, d, fx), sy = __fmaf_rn(sty, d, fyr);
            const float tx = __int_as_float(tex_coord_bits(sx)), ty = __int_as_float(tex_coord_bits(sy));
            const float b = BLUR ? lds_f32(rp + E.RB_delta) : 0.0f;
            tap<BLUR, SHIFT>(M, sx, sy, tx, ty, lds_f32(wp), lds_f32(rp), b, sh, iy < ny ? E.wb : 0u, E.hb, base, E.kq,
                             E.QB_delta);
        };
        if (!BLUR) {
            if (iy < NY) one();
        } else {
            for (; iy < NY; ++iy) {
                one();
                fyr = __fadd_rn(fyr, finc);
                wp += 4u;
                rp += rinc;
            }
        }
        fx = __fadd_rn(fx, finc);
        wa += wstep;
        ra += rstep;
    }
}

// pixel_window without its divisions for a tap step of 1.
__device__ __forceinline__ PixWin slot_window(const PmParams& P, int px, int py)
{
    if (P.inc != 1) return pixel_window(P, px, py);
    PixWin w;
    const int r = P.radius;
    w.x0 = max(0, px - r);
    w.y0 = max(0, py - r);
    w.ii0 = w.x0 - px + r;
    w.jj0 = w.y0 - py + r;
    w.nX = min(P.W - 1, px + r) - w.x0 + 1;
    w.nY = min(P.H - 1, py + r) - w.y0 + 1;
    return w;
}

// The tap indices [i0, i1] (positions p0 + i inc) whose sample p + s can lie in
// [0, lim) when the shift s is in [smin, smax]; eps covers the rounding of the
// sample positions.  Rounding to integers by the addition of 1.5 * 2^23.
__device__ __forceinline__ void cut_taps(float smin, float smax, float eps, float lim, float p0, float inv_inc, float& i0,
                                         float& i1)
{
    const float lo = __fadd_rn(__fadd_ru((-smax - eps - p0) * inv_inc - 0.001f, kRneMagic), -kRneMagic);
    const float hi = __fadd_rn(__fadd_rd((lim - smin + eps - p0) * inv_inc + 0.001f, kRneMagic), -kRneMagic);
    i0 = fmaxf(i0, lo);
    i1 = fminf(i1, hi);
}

// The rectangle of taps (first column and row, counts; 0 when empty) an NCC of
// plane dp against a neighbour with steps (stx, sty) can keep.  The disparity is
// affine over the window, so its range is at the corners.  (A second cut with the
// range over the first rectangle costs more than it saves: 24.4 against 24.1 ms,
// 2048x1536, 15x15; 10.1 against 9.8, ACMM, 5x5.)
__device__ __forceinline__ uint32_t tap_rect(const PixWin& pw, const PmParams& P, float3 dp, float stx, float sty,
                                             float inv_inc)
{
    float i0 = 0.0f, i1 = (float)(pw.nX - 1), j0 = 0.0f, j1 = (float)(pw.nY - 1);
    const float finc = (float)P.inc, X0 = (float)pw.x0, Y0 = (float)pw.y0;
    const float mag = fabsf(dp.x) * (float)P.W + fabsf(dp.y) * (float)P.H + fabsf(dp.z);
    if (mag * fmaxf(fabsf(stx), fabsf(sty)) < 1e6f) {    // false for NaN: the whole window
        const float ex = 0.01f + 4e-6f * mag * fabsf(stx), ey = 0.01f + 4e-6f * mag * fabsf(sty);
        const float dx = dp.x * finc, dy = dp.y * finc, d0 = dp.z + dp.x * X0 + dp.y * Y0;
        const float xb = dx * i1, yb = dy * j1;
        const float dmin = d0 + fminf(0.0f, xb) + fminf(0.0f, yb), dmax = d0 + fmaxf(0.0f, xb) + fmaxf(0.0f, yb);
        const float ax = stx * dmin, bx = stx * dmax, ay = sty * dmin, by = sty * dmax;
        cut_taps(fminf(ax, bx), fmaxf(ax, bx), ex, (float)P.W, X0, inv_inc, i0, i1);
        cut_taps(fminf(ay, by), fmaxf(ay, by), ey, (float)P.H, Y0, inv_inc, j0, j1);
    }
    if (!(i0 <= i1 && j0 <= j1)) return 0u;
    const uint32_t a = (uint32_t)(int)i0, b = (uint32_t)(int)j0, c = (uint32_t)(int)i1, d = (uint32_t)(int)j1;
    return a | (b << 8) | ((c - a + 1u) << 16) | ((d - b + 1u) << 24);
}

// Bin of a rectangle: columns in pairs from the widest down, rows up and down in
// turn, so that neighbours in the sorted list differ by little.
__device__ __forceinline__ int rect_bin(uint32_t rect, int tx, int ty)
{
    const int bx = ((int)((rect >> 16) & 0xFFu) - 1) >> 1, ry = (int)(rect >> 24) - 1;
    return ((tx - 1) / 2 - bx) * ty + ((bx & 1) ? ry : ty - 1 - ry);
}

// ---- staging, shared by the half-sweep and the initialisation -------------------
// Shared-memory arrays of the CTA's view.
struct StageDst {
    unsigned char* stage;    // 8-bit tiles of the view and its neighbours, filled by bulk copies
    uint64_t* bar;
    float* R;                // reference texels, column-major with stride rs
    float* RB;               // reference blur / 255
    uint32_t* Q;             // [K][H + 1][W + 1] quads
    uint32_t* QB;
    NbGeo* geo;
    int* ok;
    int rs;
};

// Thread 0 starts the bulk copies of view vid and its nc neighbours.  The threads'
// accesses to the shared area before the last barrier are ordered before them.
template <bool BLUR>
__device__ __forceinline__ void start_copies(const StageDst& D, const FrameDev& F, const PmParams& P, int vid, int nc)
{
    const int ts = P.tile_stride;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_arrive_expect_tx(D.bar, (uint32_t)((1 + nc) * ts * (BLUR ? 2 : 1)));
    for (int i = 0; i < 1 + nc; ++i) {
        const int v = (i == 0) ? vid : F.nb_ids[vid * P.K + i - 1];
        const int vv = (v < 0 || v >= F.V) ? vid : v;
        bulk_copy_g2s(D.stage + i * ts, F.gray + (size_t)vv * ts, (uint32_t)ts, D.bar);
        if (BLUR) bulk_copy_g2s(D.stage + (1 + nc + i) * ts, F.blur + (size_t)vv * ts, (uint32_t)ts, D.bar);
    }
}

// The neighbours' geometry; needs no copied tile.
__device__ __forceinline__ void stage_geo(const StageDst& D, const FrameDev& F, const PmParams& P, int vid, int nc, int* err)
{
    const float2 c0 = F.centers[vid];
    for (int k = threadIdx.x; k < P.K; k += blockDim.x) {
        int v = (k < nc) ? F.nb_ids[vid * P.K + k] : -1;
        if (v >= F.V) { atomicOr(err, PFD_DEVERR_SWEEP_CHECK); v = -1; }
        D.ok[k] = (v >= 0);
        D.geo[k] = make_geo(c0, F.centers[v >= 0 ? v : vid], P);
    }
}

// The copied tiles as floats (reference) and quads (neighbours); between barriers.
template <bool BLUR>
__device__ __forceinline__ void expand_tiles(const StageDst& D, const PmParams& P, int nc)
{
    const int W = P.W, H = P.H, ts = P.tile_stride;
    const uint8_t* stage = (const uint8_t*)D.stage;
    for (int e = threadIdx.x; e < W * H; e += blockDim.x) {
        const int ey = e / W, ex = e - ey * W;
        D.R[ex * D.rs + ey] = (float)stage[e];
        if (BLUR) D.RB[ex * D.rs + ey] = __fdiv_rn((float)stage[(1 + nc) * ts + e], 255.0f);
    }
    const int qs = W + 1, qn = (H + 1) * qs;
    for (int e = threadIdx.x; e < nc * qn; e += blockDim.x) {
        const int k = e / qn, r = e - k * qn;
        const int iy = r / qs, ix = r - iy * qs;
        const int y0 = min(iy, H - 1), y1 = min(iy + 1, H - 1);
        const int x0 = min(ix, W - 1), x1 = min(ix + 1, W - 1);
        const uint8_t* s = stage + (1 + k) * ts;
        D.Q[e] = (uint32_t)s[y0 * W + x0] | ((uint32_t)s[y0 * W + x1] << 8) | ((uint32_t)s[y1 * W + x0] << 16) |
                 ((uint32_t)s[y1 * W + x1] << 24);
        if (BLUR) {
            const uint8_t* sb = stage + (2 + nc + k) * ts;
            D.QB[e] = (uint32_t)sb[y0 * W + x0] | ((uint32_t)sb[y0 * W + x1] << 8) | ((uint32_t)sb[y1 * W + x0] << 16) |
                      ((uint32_t)sb[y1 * W + x1] << 24);
        }
    }
}

// The launch's weight tables (exponents of the spatial and the colour distance),
// and zeros behind the reference texels.
template <bool BLUR>
__device__ __forceinline__ void fill_tables(const PmParams& P, float* a_s, float* a_c, float* R, float* RB, int rs)
{
    for (int t = threadIdx.x; t < P.ntap * P.ntap; t += blockDim.x) {
        const float fi = (float)(-P.radius + (t / P.ntap) * P.inc);
        const float fj = (float)(-P.radius + (t % P.ntap) * P.inc);
        const float sd = __fsqrt_rn(__fmaf_rn(fj, fj, __fmul_rn(fi, fi)));
        a_s[t] = __fdiv_rn(-sd, P.ss2);
    }
    for (int c = threadIdx.x; c < 256; c += blockDim.x) a_c[c] = __fdiv_rn((float)c, P.cc2);
    for (int e = threadIdx.x; e < 2 * P.W * rs + 2 * P.H; e += blockDim.x) {
        R[e] = 0.0f;
        if (BLUR) RB[e] = 0.0f;
    }
}

// Bilateral weight of window tap (ix, iy) of pixel (x, y) with centre texel rc.
__device__ __forceinline__ float tap_weight(const float* R, int rs, const float* a_s, const float* a_c, const PmParams& P,
                                            const PixWin& pw, int ix, int iy, float rc)
{
    const float rv = R[(pw.x0 + ix * P.inc) * rs + pw.y0 + iy * P.inc];
    const float cd = fabsf(__fsub_rn(rv, rc));
    const int cdi = __float_as_int(__fadd_rn(cd, 8388608.0f)) & 0xFF;
    const int ti = (pw.ii0 + ix) * P.ntap + (pw.jj0 + iy);
    return pfd_expf_nonpos(__fsub_rn(a_s[ti], a_c[cdi]));
}

// Bin counts to bin offsets (one warp).
__device__ __forceinline__ int scan_bins(int* bins, int n, int lane)
{
    const int per = (n + 31) / 32;
    int sum = 0;
    for (int i = 0; i < per; ++i) {
        const int b = lane * per + i;
        if (b < n) sum += bins[b];
    }
    int off = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFullMask, off, o);
        if (lane >= o) off += t;
    }
    const int total = __shfl_sync(kFullMask, off, 31);
    off -= sum;
    for (int i = 0; i < per; ++i) {
        const int b = lane * per + i;
        if (b < n) { const int c = bins[b]; bins[b] = off; off += c; }
    }
    return total;
}

// ---- half-warp collectives -----------------------------------------------------
struct Half {
    uint32_t mask;           // the half's lanes in the warp
    int hl, shift;           // lane in the half; 0 or 16
    __device__ __forceinline__ float shfl(float v, int src) const { return __shfl_sync(mask, v, src, 16); }
    __device__ __forceinline__ int shfl(int v, int src) const { return __shfl_sync(mask, v, src, 16); }
    __device__ __forceinline__ uint32_t ballot(bool p) const { return (__ballot_sync(mask, p) >> shift) & 0xFFFFu; }
    __device__ __forceinline__ uint32_t below(uint32_t bits) const { return bits & ((1u << hl) - 1u); }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
};

// A pixel's draw stream whose first 32 draws are worked out by the half's lanes
// side by side (lane i holds draws i and 16 + i).
struct HalfDraws {
    const Half& hf;
    uint64_t seed;
    uint32_t sweep, pixel;
    float d0, d1;
    int n;
    __device__ __forceinline__ float one(int i) const
    {
        const uint4 b = philox4x32_10(make_uint4((uint32_t)i >> 2, sweep, pixel, 0u),
                                      make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
        const uint32_t w = (uint32_t)i & 3u;
        const uint32_t r = w == 0 ? b.x : (w == 1 ? b.y : (w == 2 ? b.z : b.w));
        return __fmul_rn((float)((r >> 8) + 1u), 0x1p-24f);
    }
    __device__ __forceinline__ HalfDraws(const Half& h, uint64_t s, uint32_t sw, uint32_t px)
        : hf(h), seed(s), sweep(sw), pixel(px), n(0)
    {
        d0 = one(h.hl);
        d1 = one(16 + h.hl);
    }
    __device__ __forceinline__ float uniform()
    {
        const int i = n++;
        if (i < 16) return hf.shfl(d0, i);
        if (i < 32) return hf.shfl(d1, i - 16);
        return one(i);
    }
};

// The CTA's view, as every slot sees it.
struct View {
    const float* R;          // [2 W][rs] reference texels, column-major, zeros past the window
    const NbGeo* geo;        // [K]
    const int* nb_ok;        // [K]
    const float* a_s;        // [ntap * ntap]
    const float* a_c;        // [256]
    const float* pc;         // [ppv] previous costs
    const uint32_t* ps;      // [ppv] previous selected views
    int vid, nc, rs;
    size_t vbase;
};

// A slot's arrays.
struct Slot {
    SlotState* st;
    SlotOut* out;
    float* wtab;             // [tab_n] bilateral weights of the pixel's window, x outer
    float4* plane;           // [rows]
    float4* dp;              // [rows] disparity plane and the disparity at the pixel
    float* cost;             // [rows][K]
    float* bvec;             // [K] cost vector of the best plane
    float* wgt;              // [K] view weights (draws per view)
    uint8_t* sel;            // [K] the selected views, ascending
    float* wres;             // [rows] weighted cost
    int* wmin;               // [rows] view of the lowest cost
    int16_t* aux;            // [K] proposals' sample positions, or -1
};

// ComputeWeightedCost_Frame (AdaptMIPMFrame.cu:284-317) of rows [lo, hi), one lane
// per row, on every view or on the selected ones (nsel of them; the others have
// weight 0 and unknown costs).
__device__ __forceinline__ void weigh_rows(const Half& hf, const Slot& S, int K, int lo, int hi, int nc, int nsel)
{
    const int n = nsel >= 0 ? nsel : nc;
    for (int h = lo + hf.hl; h < hi; h += 16) {
        WeightedCost wc;
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const int k = nsel >= 0 ? S.sel[i] : i;
            wc.add(k, S.cost[h * K + k], S.wgt[k]);
        }
        S.wres[h] = wc.result();
        S.wmin[h] = wc.min_idx;
    }
    hf.sync();
}

// The g-th pixel (row-major) whose colour (x + y) & 1 equals `colour`: two rows
// hold W of them.
__device__ __forceinline__ void nth_pixel(int g, int colour, int W, int& x, int& y)
{
    const int r2 = g / W;
    int rem = g - r2 * W;
    const int even = (W - colour + 1) >> 1;              // pixels of an even row
    y = 2 * r2;
    if (rem >= even) { rem -= even; ++y; }
    x = 2 * rem + ((colour ^ y) & 1);
}

__device__ __forceinline__ bool same_bits(float4 a, float4 b)
{
    return __float_as_uint(a.x) == __float_as_uint(b.x) && __float_as_uint(a.y) == __float_as_uint(b.y) &&
           __float_as_uint(a.z) == __float_as_uint(b.z) && __float_as_uint(a.w) == __float_as_uint(b.w);
}

__device__ __forceinline__ void request(SlotState& st, int row_lo, int row_hi, uint64_t skip, int n_views)
{
    st.row_lo = row_lo;
    st.row_hi = row_hi;
    st.skip = skip;
    st.n_views = n_views;
}

// The disparity planes of rows [lo, hi), one lane per row.
__device__ __forceinline__ void plane_rows(const Half& hf, const Slot& S, int lo, int hi, int x, int y)
{
    for (int h = lo + hf.hl; h < hi; h += 16) {
        const float3 dp = disparity_plane(x, y, S.plane[h]);
        S.dp[h] = make_float4(dp.x, dp.y, dp.z, to_disparity(x, y, dp));
    }
}

// Takes pixel g: the propagation candidates (AdaptMIPMFrame.cu:589-795) and the
// request for their costs (its weight table is made with the request's list).  Lane
// a < 8 works on direction a (up, down, left, right; near on even lanes, far on odd
// ones).  Row 0 holds the current plane, then one row per distinct candidate plane: a
// cost vector depends only on the pixel and the plane.  The current plane's vector is
// the stored one when that store is valid.
__device__ __forceinline__ void begin_pixel(const Half& hf, const Slot& S, const View& V, const PmParams& P,
                                            const StateDev& prev, int g, int phase)
{
    const int W = P.W, H = P.H, hl = hf.hl;
    int x, y;
    nth_pixel(g, phase, W, x, y);
    const int center = y * W + x;
    const size_t idx = V.vbase + center;
    const float4 cur = prev.plane[idx];
    const bool use_cvec = P.cvec_ok != 0;
    float cv[2] = { 0.0f, 0.0f };
    if (use_cvec) {
        if (hl < V.nc) cv[0] = P.cvec[idx * P.K + hl];
        if (hl + 16 < V.nc) cv[1] = P.cvec[idx * P.K + hl + 16];
    }
    const int a = hl & 7, dir = a >> 1;
    const bool vert = dir < 2, neg = (dir & 1) == 0;
    const int D = dir == 0 ? y : (dir == 1 ? H - 1 - y : (dir == 2 ? x : W - 1 - x));
    const int lat_lo = vert ? x : y, lat_hi = vert ? W - 1 - x : H - 1 - y;
    const int sp = vert ? 1 : W, su = neg ? -(vert ? W : 1) : (vert ? W : 1);
    const float* pc = V.pc;
    int pos = center;
    bool own = false;                                    // a sample of its own (not the near one's)
    auto take = [&](float& cm, int q) { if (pc[q] < cm) { cm = pc[q]; pos = q; } };
    if (!(a & 1)) {
        if (D > 0) {
            own = true;
            pos = center + su;
            float cm = pc[pos];
            const int s = pos;
            if (D > 1) take(cm, s + su);
            if (D > 2 && lat_lo > 1) take(cm, s + 2 * su - sp);
            if (D > 2 && lat_hi > 1) take(cm, s + 2 * su + sp);
        }
    } else if (D > 2) {
        own = true;
        pos = center + 3 * su;
        float cm = pc[pos];
        const int s = pos;
        if (D > 3) take(cm, s + su);
    }
    float4 q = cur;
    if (own) q = prev.plane[V.vbase + pos];
    const uint32_t flags = hf.ballot(D > 0) & 0xFFu, owns = hf.ballot(own) & 0xFFu;
    // the first earlier lane with the same plane; the planes side by side in the dp rows,
    // which are not in use yet
    if (hl < 8) S.dp[hl] = q;
    hf.sync();
    const bool eqcur = same_bits(q, cur);
    int match = -1;
#pragma unroll
    for (int t = 6; t >= 0; --t)
        if (t < a && ((owns >> t) & 1u) && same_bits(S.dp[t], q)) match = t;
    const bool lead = own && hl < 8 && !eqcur && match < 0;
    const uint32_t leads = hf.ballot(lead);
    int row = lead ? 1 + __popc(hf.below(leads)) : 0;
    const int mrow = hf.shfl(row, match < 0 ? 0 : match);
    if (own && !eqcur && match >= 0) row = mrow;
    const int nrow = hf.shfl(row, hl & ~1);              // the near sample's row
    if (!own) row = (D > 0) ? nrow : 0;
    if (lead) S.plane[row] = q;
    const uint32_t slots = __reduce_or_sync(hf.mask, hl < 8 ? (uint32_t)row << (4 * hl) : 0u);
    if (use_cvec) {
        if (hl < V.nc) S.cost[hl] = cv[0];
        if (hl + 16 < V.nc) S.cost[hl + 16] = cv[1];
    }
    if (hl == 0) {
        S.plane[0] = cur;
        S.st->xy = x | (y << 8);
        S.st->slots = slots;
        S.st->flags = flags;
        request(*S.st, use_cvec ? 1 : 0, 1 + __popc(leads), 0ull, -1);
    }
    hf.sync();
    plane_rows(hf, S, 0, 1 + __popc(leads), x, y);
}

// BuildCrossViewPlaneProposal (AdaptMIPMFrame.cu:350-398): the sample position (x | y
// << 8) of pixel (x, y) at disparity d in neighbour gk, or -1; and the plane from the
// neighbour's plane hn there.
__device__ __forceinline__ int proposal_at(const NbGeo& gk, int x, int y, int W, int H, float d)
{
    const float2 qf = geo_anchor(gk, x, y, d);
    const float fqx = floorf(__fadd_rn(qf.x, 0.5f)), fqy = floorf(__fadd_rn(qf.y, 0.5f));
    if (!(fqx >= 0.0f && fqx < (float)W && fqy >= 0.0f && fqy < (float)H)) return -1;
    return (int)fqx | ((int)fqy << 8);
}

__device__ __forceinline__ float4 proposal_from(const NbGeo& gk, float4 hn, int q, int x, int y)
{
    const float3 dpn = disparity_plane(q & 0xFF, q >> 8, hn);
    float denom = __fmaf_rn(dpn.y, gk.by, __fmaf_rn(dpn.x, gk.bx, 1.0f));
    denom = safe_denom(denom);
    return encode_plane(x, y, __fdiv_rn(dpn.x, denom), __fdiv_rn(dpn.y, denom), __fdiv_rn(dpn.z, denom));
}

// The five candidates of PlaneHypothesisRefinement_Frame (AdaptMIPMFrame.cu:400-471)
// for the best plane, from the draws already taken (c0: the random plane, rn: the
// random normal, u1-u3: the perturbation, u4: the depth perturbation), those from
// `from` on into rows r0 + i, one lane each.  Returns whether candidate 3 equals the
// best plane.  The caller synchronises before the rows are read.
__device__ __forceinline__ bool refine_rows(const Half& hf, const Slot& S, int x, int y, float4 best, float4 c0, float4 rn,
                                            float u1, float u2, float u3, float u4, float pert, int r0, int from)
{
    const float4 pn = perturbed_normal_u(x, y, best, u1, u2, u3, pert);
    const float dmin_p = __fmul_rn(__fsub_rn(1.0f, 0.02f), best.w), dmax_p = __fmul_rn(__fadd_rn(1.0f, 0.02f), best.w);
    const int i = hf.hl;
    float4 c = i == 0 ? c0 : (i == 1 ? rn : (i == 2 ? pn : best));
    if (i == 4) c.w = __fmaf_rn(u4, __fsub_rn(dmax_p, dmin_p), dmin_p);
    if (i > 0) c.w = to_disparity(x, y, disparity_plane(x, y, c));
    if (i >= from && i < 5) S.plane[r0 + i] = c;
    return __float_as_uint(hf.shfl(c.w, 3)) == __float_as_uint(best.w);
}

// After the propagation costs: view-selection priors and sampling (AdaptMIPMFrame.cu:
// 797-875), the best propagation plane, the refinement's draws, and the request for
// the cross-view proposals (:907-936) and the refinement candidates (:400-471), both
// built from the best plane so far.
__device__ __forceinline__ void after_propagation(const Half& hf, const Slot& S, const View& V, const FrameDev& F,
                                                  const PmParams& P, const StateDev& prev, uint32_t sweep_id, float thr,
                                                  float p_default)
{
    const int W = P.W, H = P.H, K = P.K, nc = V.nc, hl = hf.hl;
    SlotState& st = *S.st;
    const int x = st.xy & 0xFF, y = st.xy >> 8, center = y * W + x;
    const uint32_t slots = st.slots, flags = st.flags;
    HalfDraws g(hf, P.seed, sweep_id, (uint32_t)(V.vbase + center));
    const int dpos[4] = { (y > 0) ? center - W : -1, (y < H - 1) ? center + W : -1, (x > 0) ? center - 1 : -1,
                          (x < W - 1) ? center + 1 : -1 };
    // one view per lane (two above 16 views)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = hl + 16 * half;
        if (16 * half >= nc) break;
        if (i >= nc) continue;
        float prior = 0.0f;
#pragma unroll
        for (int ii = 0; ii < 4; ++ii)
            if (dpos[ii] >= 0) prior = __fadd_rn(prior, ((V.ps[dpos[ii]] >> i) & 1u) ? 0.9f : 0.1f);
        // the terms side by side, then their sum in order (a term that does not count is
        // +0, which leaves the sum as it is)
        float count = 0.0f, tmpw = 0.0f, p = 0.0f;
        int count_false = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const bool there = (flags >> j) & 1u;
            const float c = S.cost[(int)((slots >> (4 * j)) & 15u) * K + i];
            const bool low = there && c < thr;
            const float e = pfd_expf_nonpos(div_m018(__fmul_rn(c, c)));
            tmpw = __fadd_rn(tmpw, low ? e : 0.0f);
            count = __fadd_rn(count, low ? 1.0f : 0.0f);
            count_false += there && c > 1.2f;
        }
        if (count > 2.0f && count_false < 3) p = __fdiv_rn(tmpw, count);
        else if (count_false < 3) p = p_default;
        S.wgt[i] = __fmul_rn(p, prior);
    }
    hf.sync();
    // the sums over views run in view order, as the reference's loops do;
    // TransformPDFToCDF (CudaUtil.cu:491-507) and the 15 draws, one per lane: a draw's
    // view is the first whose CDF exceeds it (a CDF of NaN, all probabilities 0, exceeds
    // nothing)
    float psum = 0.0f;
#pragma unroll 4
    for (int i = 0; i < nc; ++i) psum = __fadd_rn(psum, S.wgt[i]);
    const float inv = __fdiv_rn(1.0f, psum);
    const float rp = __fsub_rn(g.d0, 1.1920928955078125e-07f);
    float cum = 0.0f;
    int id = 0;
    bool over = false;
#pragma unroll 4
    for (int i = 0; i < nc; ++i) {
        cum = __fmaf_rn(S.wgt[i], inv, cum);
        over |= cum > rp;
        id += !over;
    }
    hf.sync();                                           // the probabilities are read before they are replaced
    // draws per view, 4 bits each (at most 15), added up over the lanes
    uint32_t tsel = 0;
    {
        const uint32_t one = hl < 15 && id < nc ? 1u << (4 * (id & 7)) : 0u;
        uint32_t n0 = __reduce_add_sync(hf.mask, (id >> 3) == 0 ? one : 0u);
        uint32_t n1 = __reduce_add_sync(hf.mask, (id >> 3) == 1 ? one : 0u), n2 = 0u, n3 = 0u;
        if (nc > 16) {
            n2 = __reduce_add_sync(hf.mask, (id >> 3) == 2 ? one : 0u);
            n3 = __reduce_add_sync(hf.mask, (id >> 3) == 3 ? one : 0u);
        }
        if ((n0 | n1 | n2 | n3) == 0u) n0 = n1 = n2 = n3 = 0x11111111u;        // no draw hit: every view once
        const int c0 = (int)(((hl < 8 ? n0 : n1) >> (4 * (hl & 7))) & 15u), c1 = (int)(((hl < 8 ? n2 : n3) >> (4 * (hl & 7))) & 15u);
        tsel = hf.ballot(hl < nc && c0 > 0);
        if (nc > 16) tsel |= hf.ballot(16 + hl < nc && c1 > 0) << 16;
        if (hl < nc) {
            S.wgt[hl] = (float)c0;
            if ((tsel >> hl) & 1u) S.sel[__popc(tsel & ((1u << hl) - 1u))] = (uint8_t)hl;
        }
        if (16 + hl < nc) {
            S.wgt[16 + hl] = (float)c1;
            if ((tsel >> (16 + hl)) & 1u) S.sel[__popc(tsel & ((1u << (16 + hl)) - 1u))] = (uint8_t)(16 + hl);
        }
        hf.sync();
    }
    const int nh = st.row_hi;
    weigh_rows(hf, S, K, 0, nh, nc, -1);
    // current plane, then the candidates in slot order
    float best_cost = S.wres[0];
    int best_row = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int r = (int)((slots >> (4 * s)) & 15u);
        const float c = S.wres[r];
        if (((flags >> s) & 1u) && c < best_cost) { best_cost = c; best_row = r; }
    }
    const int best_min = S.wmin[best_row];
    const float4 best_plane = S.plane[best_row];
    const float best_d = S.dp[best_row].w;
    for (int k = hl; k < nc; k += 16) S.bvec[k] = S.cost[best_row * K + k];
    // the refinement's draws: 15 (depth_rand: drawn, never used), a normal by rejection
    // from pairs of draws 16 on, four uniforms, a depth, another normal.  Lanes 0-7 try
    // the pairs from even draws and lanes 8-14 those from odd draws side by side; the
    // first normal is the first accepted even pair, the second the first accepted odd
    // pair after the five draws between.
    float4 rn, c0;
    float u1, u2, u3, u4;
    {
        const int first = hl < 8 ? 2 * hl : 2 * hl - 15;
        const float q1 = __fmaf_rn(2.0f, hf.shfl(g.d1, first & 15), -1.0f);
        const float q2 = __fmaf_rn(2.0f, hf.shfl(g.d1, (first + 1) & 15), -1.0f);
        const float ss = __fmaf_rn(q2, q2, __fmul_rn(q1, q1));
        const uint32_t good = hf.ballot(hl < 15 && ss < 1.0f);
        const int a1 = __ffs(good & 0xFFu) - 1;
        const uint32_t odd = a1 >= 0 ? (good >> 8) & ~((1u << (a1 + 3)) - 1u) : 0u;
        if (odd) {
            const float sq = __fsqrt_rn(__fsub_rn(1.0f, ss));
            const float4 n = normalize3(make_float4(__fmul_rn(__fmul_rn(2.0f, q1), sq), __fmul_rn(__fmul_rn(2.0f, q2), sq),
                                                    __fmaf_rn(-2.0f, ss, 1.0f), 0.0f));
            const int b1 = 7 + __ffs(odd), at = 2 * a1 + 2;
            rn = make_float4(hf.shfl(n.x, a1), hf.shfl(n.y, a1), hf.shfl(n.z, a1), 0.0f);
            u1 = hf.shfl(g.d1, at);
            u2 = hf.shfl(g.d1, at + 1);
            u3 = hf.shfl(g.d1, at + 2);
            u4 = hf.shfl(g.d1, at + 3);
            const float depth = __fmaf_rn(hf.shfl(g.d1, at + 4), __fsub_rn(P.depth_max, P.depth_min), P.depth_min);
            c0 = make_float4(hf.shfl(n.x, b1), hf.shfl(n.y, b1), hf.shfl(n.z, b1), depth);
        } else {                                         // more than 16 draws: one after another
            g.n = 16;
            rn = random_normal(g);
            u1 = g.uniform();
            u2 = g.uniform();
            u3 = g.uniform();
            u4 = g.uniform();
            c0 = random_plane(g, P.depth_min, P.depth_max);
        }
    }
    hf.sync();                                           // every lane has read the rows before they are reused
    const int nsel = __popc(tsel);
    int nact = 0;
    for (int n0 = 0; n0 < nsel; n0 += 16) {
        const int n = n0 + hl;
        int q = -1, k = 0, nvid = -1;
        if (n < nsel) {
            k = S.sel[n];
            nvid = F.nb_ids[V.vid * K + k];
            if (nvid >= 0) q = proposal_at(V.geo[k], x, y, W, H, best_d);
        }
        const uint32_t act = hf.ballot(q >= 0);
        if (q >= 0)
            S.plane[nact + __popc(hf.below(act))] =
                proposal_from(V.geo[k], prev.plane[(size_t)nvid * P.ppv + (q >> 8) * W + (q & 0xFF)], q, x, y);
        if (n < nsel) S.aux[n] = (int16_t)q;
        nact += __popc(act);
    }
    // the candidate equal to the best plane has the best cost and cannot win
    const bool skip3 = refine_rows(hf, S, x, y, best_plane, c0, rn, u1, u2, u3, u4, P.pert_pi, nact, 0);
    if (hl == 0) {
        st.best_plane = best_plane;
        st.best_cost = best_cost;
        st.best_d = best_d;
        st.best_min = best_min;
        st.best_row = best_row;
        st.c0 = c0;
        st.rn = rn;
        st.u = make_float4(u1, u2, u3, u4);
        st.tsel = tsel;
        st.r0 = nact;
        st.n = 0;
        st.hs = 0;
        st.flags = skip3 ? kFlagSkip3 : 0u;
        request(st, 0, nact + 5, skip3 ? (1ull << (nact + 3)) : 0ull, nsel);
    }
    hf.sync();
    plane_rows(hf, S, 0, nact + 5, x, y);
}

// The walk over the proposals in reference order and the refinement candidates
// after it.  stage: what the costs that have just come in were for.  Returns the
// stage of the next request, or kNew when the pixel's best plane is final and its
// cost vector is known.
__device__ __forceinline__ int after_speculation(const Half& hf, const Slot& S, const View& V, const FrameDev& F,
                                                 const PmParams& P, const StateDev& prev, int stage)
{
    const int W = P.W, H = P.H, K = P.K, nc = V.nc, hl = hf.hl;
    SlotState& st = *S.st;
    const int x = st.xy & 0xFF, y = st.xy >> 8;
    const int nsel = __popc(st.tsel), r0 = st.r0;
    weigh_rows(hf, S, K, st.row_lo, st.row_hi, nc, nsel);
    float best_cost = st.best_cost, best_d = st.best_d;
    float4 best_plane = st.best_plane;
    int best_min = st.best_min, n = st.n, hs = st.hs;
    uint32_t flags = st.flags;
    hf.sync();
    if (stage == kSpec) {
        // nothing changes before the first proposal that wins: the lanes look for it side
        // by side
        for (int n0 = 0; n0 < nsel; n0 += 16) {
            const bool act = n0 + hl < nsel && S.aux[n0 + hl] >= 0;
            const uint32_t acts = hf.ballot(act);
            const uint32_t wins = hf.ballot(act && S.wres[hs + __popc(hf.below(acts))] < best_cost);
            if (wins) {
                const int w = __ffs(wins) - 1;
                n = n0 + w;
                hs += __popc(acts & ((1u << w) - 1u));
                break;
            }
            hs += __popc(acts);
            n = nsel;
        }
    }
    if (stage != kRedo) {
        bool resumed = stage == kWalk;
        for (; n < nsel; ++n) {
            const int spec_q = S.aux[n];
            int q = spec_q, k = 0, nvid = -1;
            if (flags & kFlagChanged) {
                k = S.sel[n];
                nvid = F.nb_ids[V.vid * K + k];
                q = (nvid >= 0) ? proposal_at(V.geo[k], x, y, W, H, best_d) : -1;
            }
            if (q >= 0) {
                const int row = (spec_q >= 0) ? hs : r0 + 5;
                if (q != spec_q && !resumed) {
                    // the best plane moved the sample position: rebuild this proposal in its
                    // own row (or the spare row after the refinement candidates)
                    const float4 proxy =
                        proposal_from(V.geo[k], prev.plane[(size_t)nvid * P.ppv + (q >> 8) * W + (q & 0xFF)], q, x, y);
                    if (hl == 0) {
                        S.plane[row] = proxy;
                        st.best_plane = best_plane;
                        st.best_cost = best_cost;
                        st.best_d = best_d;
                        st.best_min = best_min;
                        st.n = n;
                        st.hs = hs;
                        st.flags = flags;
                        request(st, row, row + 1, 0ull, nsel);
                    }
                    hf.sync();
                    plane_rows(hf, S, row, row + 1, x, y);
                    return kWalk;
                }
                const float c = S.wres[row];
                if (c < best_cost) {
                    best_cost = c;
                    best_plane = S.plane[row];
                    best_d = S.dp[row].w;
                    best_min = S.wmin[row];
                    flags |= kFlagChanged | kFlagPartial;
                }
            }
            resumed = false;
            if (spec_q >= 0) ++hs;
        }
        if (flags & kFlagChanged) {
            // candidates 2-4 follow the best plane: rebuild and evaluate them again
            hf.sync();                                   // proposal rows may be read above
            const bool skip3 = refine_rows(hf, S, x, y, best_plane, st.c0, st.rn, st.u.x, st.u.y, st.u.z, st.u.w, P.pert_pi,
                                           r0, 2);
            flags = (flags & ~kFlagSkip3) | (skip3 ? kFlagSkip3 : 0u);
            if (hl == 0) {
                st.best_plane = best_plane;
                st.best_cost = best_cost;
                st.best_d = best_d;
                st.best_min = best_min;
                st.flags = flags;
                request(st, r0 + 2, r0 + 5, skip3 ? (1ull << (r0 + 3)) : 0ull, nsel);
            }
            hf.sync();
            plane_rows(hf, S, r0 + 2, r0 + 5, x, y);
            return kRedo;
        }
    }
    {
        int won = -1;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float c = S.wres[r0 + i];
            if (!(i == 3 && (flags & kFlagSkip3)) && c < best_cost) { best_cost = c; won = i; }
        }
        if (won >= 0) {
            best_plane = S.plane[r0 + won];
            best_d = S.dp[r0 + won].w;
            best_min = S.wmin[r0 + won];
            flags |= kFlagPartial;
        }
    }
    hf.sync();
    // proposals and refinement candidates were evaluated on the selected views only,
    // which fixes their weighted cost; the winner's lowest-cost view runs over every
    // view, and its vector is stored, so the whole vector is evaluated
    if (hl == 0) {
        st.best_plane = best_plane;
        st.best_cost = best_cost;
        st.best_d = best_d;
        st.best_min = best_min;
        st.flags = flags;
        if (flags & kFlagPartial) {
            S.plane[0] = best_plane;
            request(st, 0, 1, 0ull, -1);
        }
    }
    hf.sync();
    if (!(flags & kFlagPartial)) return kNew;
    plane_rows(hf, S, 0, 1, x, y);
    return kComplete;
}

// The pixel's new state into the slot's out record.  completed: row 0 holds the
// winner's cost vector (a proposal or refinement candidate won); otherwise bvec does.
__device__ __forceinline__ void finish_pixel(const Half& hf, const Slot& S, const View& V, const PmParams& P,
                                             bool completed)
{
    const int K = P.K, nc = V.nc, hl = hf.hl, W = P.W;
    SlotState& st = *S.st;
    const int x = st.xy & 0xFF, y = st.xy >> 8;
    const size_t idx = V.vbase + y * W + x;
    const float* vec = completed ? S.cost : S.bvec;
    const float v0 = hl < nc ? vec[hl] : 2.0f, v1 = 16 + hl < nc ? vec[16 + hl] : 2.0f;
    // the stored vector of the new current plane (unchanged when the current
    // plane stays and its stored vector was used)
    if (P.cvec && (completed || st.best_row != 0 || !P.cvec_ok)) {
        if (hl < nc) P.cvec[idx * K + hl] = v0;
        if (16 + hl < nc) P.cvec[idx * K + 16 + hl] = v1;
    }
    uint32_t sel_out = st.tsel;
    float cost_out = st.best_cost;
    int disp_view = st.best_min;
    if (completed || P.acmm) {
        // the first view of the lowest cost, among the costs below 2 (-1: none)
        uint32_t low = min(v0 < 2.0f ? __float_as_uint(v0) : 0x40000000u, v1 < 2.0f ? __float_as_uint(v1) : 0x40000000u);
        low = __reduce_min_sync(hf.mask, low);           // costs are >= 0: their bits order as they do
        const uint32_t at = hf.ballot(__float_as_uint(v0) == low) | (hf.ballot(__float_as_uint(v1) == low) << 16);
        disp_view = low < 0x40000000u ? __ffs(at) - 1 : -1;
    }
    if (P.acmm) {
        // ACMM write-back (AdaptMIPMFrameACMM.cu:880-900, RecomputeSupportCostDisp_Frame
        // :259-280): the final plane's vector over every view gives the stored cost
        // (mean of the top-k), the selected views (the top-k mask) and the disp of the
        // lowest-cost view; DetailRestorer_FrameACMM does nothing without a warm start
        const int valid = __popc(hf.ballot(hl < nc && v0 < 2.0f)) + __popc(hf.ballot(16 + hl < nc && v1 < 2.0f));
        cost_out = 2.0f;
        sel_out = 0;
        if (valid > 0) {
            // the k smallest in ascending order: the lowest left, every time
            const int kk = min(valid, P.top_k);
            uint32_t b0 = hl < nc ? __float_as_uint(v0) : 0xffffffffu, b1 = 16 + hl < nc ? __float_as_uint(v1) : 0xffffffffu;
            float m = 0.0f;
            uint32_t low = 0u;
            for (int i = 0; i < kk; ++i) {
                low = __reduce_min_sync(hf.mask, min(b0, b1));
                m = __fadd_rn(m, __uint_as_float(low));
                const int lane = __ffs(hf.ballot(b0 == low || b1 == low)) - 1;
                if (hl == lane) { if (b0 == low) b0 = 0xffffffffu; else b1 = 0xffffffffu; }
            }
            cost_out = __fdiv_rn(m, (float)kk);
            const float thr = __uint_as_float(low);
            sel_out = hf.ballot(hl < nc && v0 <= thr) | (hf.ballot(16 + hl < nc && v1 <= thr) << 16);
        }
    }
    if (hl == 0) {
        S.out->plane = st.best_plane;
        S.out->cost = cost_out;
        S.out->d = st.best_d;
        S.out->sel = sel_out;
        S.out->xy_view = x | (y << 8) | ((disp_view + 1) << 16);
    }
    hf.sync();
}

// Writes a finished pixel's state (one lane per slot) and clears the record.
__device__ __forceinline__ void write_out(SlotOut& o, const View& V, const PmParams& P, const StateDev& next)
{
    const int xv = o.xy_view;
    if (xv < 0) return;
    const int x = xv & 0xFF, y = (xv >> 8) & 0xFF, view = (xv >> 16) - 1;
    const size_t idx = V.vbase + y * P.W + x;
    float4 disp = make_float4(0.f, 0.f, 0.f, 0.f);
    if (view >= 0) disp = geo_disp(V.geo[view], x, y, o.d);
    next.plane[idx] = o.plane;
    next.cost[idx] = o.cost;
    next.disp[idx] = disp;
    next.sel[idx] = o.sel;
    o.xy_view = -1;
}

}  // namespace

// One half-sweep of one frame by this CTA: it takes (micro-image, pixel part)
// items from P.view_queue until none is left.  parity: the staging barrier's
// phase, carried across frames.  Returns false when a staging wait gave up.
template <bool BLUR, bool SHIFT, int WARPS>
__device__ __forceinline__ bool sweep_slots(unsigned char* smem, const FrameDev& F, const PmParams& P,
                                            const StateDev& prev, const StateDev& next, int iter, int phase, int* err,
                                            uint32_t& parity)
{
    const int W = P.W, H = P.H, K = P.K, ts = P.tile_stride;
    const int n_slots = P.slots, cap = P.task_cap;
    const SlotPlan L = SlotPlan::make(W, H, K, P.ntap, BLUR, ts, n_slots, cap);
    {
        // the plan must fit what the launch has (the decision is the same in every thread)
        uint32_t dyn;
        asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (!(L.total <= (int)dyn && P.view_queue != nullptr && n_slots >= 1 && n_slots <= 2 * WARPS && n_slots <= 32 &&
              cap >= slot_tasks(K) && P.parts >= 1)) {
            if (threadIdx.x == 0) atomicOr(err, PFD_DEVERR_SWEEP_CHECK);
            return false;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    Half hf;
    hf.shift = lane & 16;
    hf.hl = lane & 15;
    hf.mask = 0xFFFFu << hf.shift;
    int* ctl = (int*)(smem + L.off_ctl);
    float* R = (float*)(smem + L.off_R);
    float* RB = (float*)(smem + L.off_RB);
    float* pc = (float*)(smem + L.off_pc);
    uint32_t* ps = (uint32_t*)(smem + L.off_ps);
    int* bins = (int*)(smem + L.off_bins);
    int* stages = (int*)(smem + L.off_stages), *next_stages = stages + 32;
    uint16_t* t_id = (uint16_t*)(smem + L.off_id);
    uint16_t* t_order = (uint16_t*)(smem + L.off_order);
    NbGeo* geo = (NbGeo*)(smem + L.off_geo);
    int* okk = (int*)(smem + L.off_ok);
    auto slot_at = [&](int s) {
        Slot S;
        S.st = (SlotState*)(smem + L.off_state) + s;
        S.out = (SlotOut*)(smem + L.off_out) + s;
        S.wtab = (float*)(smem + L.off_wtab) + s * L.tab_n;
        S.plane = (float4*)(smem + L.off_plane) + s * L.rows;
        S.dp = (float4*)(smem + L.off_dp) + s * L.rows;
        S.cost = (float*)(smem + L.off_cost) + s * L.rows * K;
        S.bvec = (float*)(smem + L.off_bvec) + s * K;
        S.wgt = (float*)(smem + L.off_wgt) + s * K;
        S.wres = (float*)(smem + L.off_wres) + s * L.rows;
        S.wmin = (int*)(smem + L.off_wmin) + s * L.rows;
        S.aux = (int16_t*)(smem + L.off_aux) + s * K;
        S.sel = (uint8_t*)(smem + L.off_sel) + s * K;
        return S;
    };
    const float inv_inc = 1.0f / (float)P.inc;
    const int n_upd = (P.ppv + (phase == 0 ? 1 : 0)) / 2;      // pixels with (x + y) & 1 == phase
    const uint32_t sweep_id = (uint32_t)(1 + 2 * iter + phase);
    const float thr = __fmul_rn(0.8f, pfd_expf(__fdiv_rn((float)(iter * iter), -90.0f)));
    const float p_default = pfd_expf(__fdiv_rn(__fmul_rn(thr, thr), -0.32f));

    fill_tables<BLUR>(P, (float*)(smem + L.off_as), (float*)(smem + L.off_ac), R, RB, L.rs);
    for (int e = tid; e < L.nbins; e += blockDim.x) bins[e] = 0;
    StageDst D;
    D.stage = smem + L.off_stage;
    D.bar = (uint64_t*)smem;
    D.R = R;
    D.RB = RB;
    D.Q = (uint32_t*)(smem + L.off_Q);
    D.QB = (uint32_t*)(smem + L.off_QB);
    D.geo = geo;
    D.ok = okk;
    D.rs = L.rs;
    EvalEnv E;
    E.wtab = smem_u32(smem + L.off_wtab);
    E.R = smem_u32(R);
    E.RB_delta = BLUR ? (uint32_t)(L.off_RB - L.off_R) : 0u;
    E.Q = smem_u32(smem + L.off_Q);
    E.QB_delta = BLUR ? (uint32_t)(L.off_QB - L.off_Q) : 0u;
    E.q_bytes = (H + 1) * (W + 1) * 4;
    E.tab_n = L.tab_n;
    E.rs = L.rs;
    E.inc = P.inc;
    E.wb = P.W_bits;
    E.hb = P.H_bits;
    E.kq = ((uint32_t)(W + 1) * 4u << 24) | (4u << 16);
    View V;
    V.R = R;
    V.geo = geo;
    V.nb_ok = okk;
    V.a_s = (const float*)(smem + L.off_as);
    V.a_c = (const float*)(smem + L.off_ac);
    V.pc = pc;
    V.ps = ps;
    V.rs = L.rs;

    // the CTAs take items one at a time from a shared counter, so a CTA that drew cheap
    // ones takes more; which CTA updates a pixel does not change its result
    for (;;) {
        __syncthreads();                                 // every thread has read the previous item
        if (tid == 0) ctl[kCtlItem] = atomicAdd(P.view_queue, 1);
        __syncthreads();
        const int item = ctl[kCtlItem];
        if (item >= F.V * P.parts) break;
        const int vid = item / P.parts, part = item - vid * P.parts;
        const int g_lo = (int)((long long)n_upd * part / P.parts), g_hi = (int)((long long)n_upd * (part + 1) / P.parts);
        const int nc = min(F.nb_counts[vid], K);
        const size_t vbase = (size_t)vid * P.ppv;
        V.vid = vid;
        V.nc = nc;
        V.vbase = vbase;
        if (nc > 0 && tid == 0) start_copies<BLUR>(D, F, P, vid, nc);
        // the other colour keeps its state; so does every pixel of a view without neighbours
        for (int e = tid; e < P.ppv; e += blockDim.x) {
            const int ey = e / W, ex = e - ey * W;
            const float c = prev.cost[vbase + e];
            const uint32_t sv = prev.sel[vbase + e];
            pc[e] = c;
            ps[e] = sv;
            if (part != 0 || (nc > 0 && ((ex + ey) & 1) == phase)) continue;
            next.plane[vbase + e] = prev.plane[vbase + e];
            next.cost[vbase + e] = c;
            next.disp[vbase + e] = prev.disp[vbase + e];
            next.sel[vbase + e] = sv;
        }
        if (nc <= 0) continue;
        stage_geo(D, F, P, vid, nc, err);
        if (tid == 0) {
            ctl[kCtlPixel] = g_lo;
            ctl[kCtlTasks] = 0;
        }
        const bool ok = mbar_wait_bounded((uint64_t*)smem, parity, err);
        if (__syncthreads_or(!ok)) return false;
        parity ^= 1u;
        expand_tiles<BLUR>(D, P, nc);
        __syncthreads();
        // stage of every slot; a slot whose request did not fit the list keeps it (kWaits set)
        if (tid < 32) {
            stages[tid] = tid < n_slots ? kNew : kIdle;
            next_stages[tid] = kIdle;
            if (tid < n_slots) slot_at(tid).out->xy_view = -1;
        }
        __syncthreads();

        for (;;) {
            // ---- every slot on to its next request.  The halves take the slots ordered by
            // stage, so the two halves of a warp mostly run the same code.
            {
                const int mine = stages[lane];
                int rank = 0, below = 0;
#pragma unroll
                for (int k = kComplete; k >= kIdle; --k) {
                    const uint32_t m = __ballot_sync(kFullMask, mine == k || (k == kIdle && (mine & kWaits)));
                    if (mine == k || (k == kIdle && (mine & kWaits))) rank = below + __popc(m & ((1u << lane) - 1u));
                    below += __popc(m);
                }
                int slot = -1;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t m = __ballot_sync(kFullMask, rank == 2 * warp + h);
                    if (h == (lane >> 4)) slot = __ffs(m) - 1;
                }
                int stage = slot >= 0 ? stages[slot] : kIdle;
                __syncwarp();
                if (stage != kIdle && !(stage & kWaits)) {
                    const Slot S = slot_at(slot);
                    if (stage == kProp) {
                        after_propagation(hf, S, V, F, P, prev, sweep_id, thr, p_default);
                        stage = kSpec;
                    } else {
                        if (stage == kComplete) {
                            finish_pixel(hf, S, V, P, true);
                            stage = kNew;
                        } else if (stage != kNew) {
                            stage = after_speculation(hf, S, V, F, P, prev, stage);
                            if (stage == kNew) finish_pixel(hf, S, V, P, false);
                        }
                        if (stage == kNew) {
                            int g = 0;
                            if (hf.hl == 0) g = atomicAdd(&ctl[kCtlPixel], 1);
                            g = hf.shfl(g, 0);
                            if (g < g_hi) {
                                begin_pixel(hf, S, V, P, prev, g, phase);
                                stage = kProp | kFresh;
                            } else {
                                stage = kIdle;
                            }
                        }
                    }
                    if (hf.hl == 0) next_stages[slot] = stage;
                } else if (slot >= 0 && hf.hl == 0) {
                    next_stages[slot] = stage & ~kWaits;
                }
            }
            __syncthreads();
            // ---- the requests' NCCs into the list, 32 (row, view) pairs per warp at a time.
            // Slots whose pairs do not fit the list wait for the next round.
            // A pair's place in the list is its index (0xFFFF: nothing to evaluate): no vote
            // and no shared counter per 32 pairs (1% of a half-sweep).
            int n_pairs;
            {
                const int entered = next_stages[lane], stage = entered & ~kFresh;
                int pairs = 0;
                if (stage != kIdle) {
                    const SlotState& st = *slot_at(lane).st;
                    pairs = (st.row_hi - st.row_lo) * (st.n_views >= 0 ? st.n_views : nc);
                }
                if (warp == WARPS - 1 && lane < n_slots) write_out(*slot_at(lane).out, V, P, next);
                if (!__any_sync(kFullMask, stage != kIdle)) break;       // the same in every warp
                // weight tables of the pixels just taken, 32 taps per warp at a time
                {
                    const int chunks = (L.tab_n + 31) >> 5;
                    uint32_t left = __ballot_sync(kFullMask, (entered & kFresh) != 0);
                    for (int i = 0; left; left &= left - 1, ++i) {
                        const int slot = __ffs(left) - 1, xy = slot_at(slot).st->xy, x = xy & 0xFF, y = xy >> 8;
                        // chunk c of the i-th such slot belongs to warp (i chunks + c) mod WARPS
                        const int u = (warp + WARPS - (i * chunks) % WARPS) % WARPS;
                        if (u >= chunks) continue;
                        const PixWin pw = slot_window(P, x, y);
                        const float rc = R[x * L.rs + y];
                        const int n = pw.nX * pw.nY;
                        const uint32_t magic = pw.nY > 1 ? 0xFFFFFFFFu / (uint32_t)pw.nY + 1u : 0u;
                        float* wtab = slot_at(slot).wtab;
                        for (int c = u; c < chunks; c += WARPS) {
                            const int t = c * 32 + lane;
                            if (t >= n) continue;
                            const int ix = pw.nY > 1 ? (int)__umulhi((uint32_t)t, magic) : t, iy = t - ix * pw.nY;
                            wtab[t] = tap_weight(R, L.rs, V.a_s, V.a_c, P, pw, ix, iy, rc);
                        }
                    }
                }
                int upto = pairs;
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(kFullMask, upto, o);
                    if (lane >= o) upto += t;
                }
                const bool fits = upto <= cap;
                const int start = upto - pairs;
                n_pairs = __reduce_max_sync(kFullMask, fits ? upto : 0);
                if (warp == 0) stages[lane] = fits ? stage : (stage | kWaits);
                int units = fits ? (pairs + 31) >> 5 : 0, first = units;
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(kFullMask, first, o);
                    if (lane >= o) first += t;
                }
                const int n_units = __shfl_sync(kFullMask, first, 31);
                first -= units;
                for (int u = warp; u < n_units; u += WARPS) {
                    __syncwarp();
                    const uint32_t holds = __ballot_sync(kFullMask, units > 0 && first <= u);
                    const int slot = 31 - __clz(holds);
                    const int e = (u - __shfl_sync(kFullMask, first, slot)) * 32 + lane, total = __shfl_sync(kFullMask, pairs, slot);
                    const int at = __shfl_sync(kFullMask, start, slot) + e;
                    if (e >= total) continue;
                    const Slot S = slot_at(slot);
                    const SlotState& st = *S.st;
                    const int nv = st.n_views, x = st.xy & 0xFF, y = st.xy >> 8;
                    const uint64_t skip = st.skip;
                    const PixWin pw = slot_window(P, x, y);
                    const int per = nv >= 0 ? nv : nc;
                    const uint32_t magic = per > 1 ? 0xFFFFFFFFu / (uint32_t)per + 1u : 0u;
                    const int hr = per > 1 ? (int)__umulhi((uint32_t)e, magic) : e;
                    const int h = st.row_lo + hr;
                    int k = e - hr * per;
                    uint32_t rect = 0u;
                    if (!((skip >> h) & 1ull)) {
                        if (nv >= 0) k = S.sel[k];
                        if (okk[k]) {
                            const float4 d = S.dp[h];
                            const NbGeo g = geo[k];
                            const float2 a = geo_anchor(g, x, y, d.w);
                            if ((__float_as_uint(a.x) < P.W_bits) && (__float_as_uint(a.y) < P.H_bits))
                                rect = tap_rect(pw, P, make_float3(d.x, d.y, d.z), g.stx, g.sty, inv_inc);
                        }
                        // no anchor in the window, or no tap: 2 without evaluation.  The cell of an
                        // NCC to be evaluated holds its rectangle until its cost is known.
                        S.cost[h * K + k] = rect ? __uint_as_float(rect) : kCostMax;
                    }
                    t_id[at] = rect ? (uint16_t)((slot << 11) | (h << 5) | k) : (uint16_t)0xFFFFu;
                    if (rect) atomicAdd(&bins[rect_bin(rect, L.tx, L.ty)], 1);
                }
            }
            __syncthreads();
            // ---- sort by rectangle: bin offsets, then the order
            if (warp == 0) {
                const int n = scan_bins(bins, L.nbins, lane);
                if (lane == 0) {
                    ctl[kCtlTasks] = n;
                    ctl[kCtlPass] = 0;
                }
            }
            __syncthreads();
            const int n_tasks = ctl[kCtlTasks];
            for (int i = tid; i < n_pairs; i += blockDim.x) {
                const int id = t_id[i];
                if (id == 0xFFFF) continue;
                const uint32_t rect = ((const uint32_t*)(smem + L.off_cost))[((id >> 11) * L.rows + ((id >> 5) & 63)) * K + (id & 31)];
                t_order[atomicAdd(&bins[rect_bin(rect, L.tx, L.ty)], 1)] = (uint16_t)id;
            }
            __syncthreads();
            for (int e = tid; e < L.nbins; e += blockDim.x) bins[e] = 0;
            // ---- evaluate, 32 NCCs per warp at a time
            for (;;) {
                int p = 0;
                if (lane == 0) p = atomicAdd(&ctl[kCtlPass], 1);
                p = __shfl_sync(kFullMask, p, 0);
                if (p * 32 >= n_tasks) break;
                const bool act = p * 32 + lane < n_tasks;
                const int id = act ? t_order[p * 32 + lane] : 0;
                const int s = id >> 11, h = (id >> 5) & 63, k = id & 31;
                float* cell = (float*)(smem + L.off_cost) + (s * L.rows + h) * K + k;
                const uint32_t rect = act ? __float_as_uint(*cell) : 0u;
                const float4 d = ((const float4*)(smem + L.off_dp))[s * L.rows + h];
                const int xy = ((const SlotState*)(smem + L.off_state))[s].xy;
                const int x = xy & 0xFF, y = xy >> 8;
                const PixWin pw = slot_window(P, act ? x : 0, act ? y : 0);
                const int i0 = rect & 0xFF, j0 = (rect >> 8) & 0xFF;
                const int X = pw.x0 + i0 * P.inc, Y = pw.y0 + j0 * P.inc;
                Moments M = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
                const float sh = SHIFT ? R[(act ? x * L.rs + y : 0)] : 0.0f;
                walk<BLUR, SHIFT>(M, E, make_float3(d.x, d.y, d.z), geo[k].stx, geo[k].sty, (int)((rect >> 16) & 0xFFu),
                                  (int)(rect >> 24), E.wtab + (uint32_t)(s * L.tab_n + i0 * pw.nY + j0) * 4u,
                                  E.R + (uint32_t)(X * L.rs + Y) * 4u, (uint32_t)pw.nY * 4u, (float)X, (float)Y,
                                  E.Q + (uint32_t)(k * E.q_bytes), sh);
                if (act) *cell = ncc_cost<BLUR>(M, P.blur_gain);
            }
            __syncthreads();
        }
    }
    return true;
}

// The staging barrier (offset 0 of every plan), once per launch.
__device__ __forceinline__ void init_barrier(unsigned char* smem)
{
    if (threadIdx.x == 0) mbar_init((uint64_t*)smem, 1);
    __syncthreads();
}

// ---- initialisation --------------------------------------------------------------
// RandomInitializationForFrame (AdaptMIPMFrame.cu:474-518): a random plane per
// pixel, its cost vector, and from it the stored cost, views and disp
// (ComputeSelectedViewsTopK_Frame, :227-282).  A CTA takes a micro-image and runs
// its pixels in chunks: the chunk's weight tables and planes, one list of all its
// (pixel, neighbour) NCCs sorted by tap rectangle and evaluated 32 at a time as in
// the half-sweep, then one thread per pixel for the views.  With refit set a pixel
// keeps its plane (PostRefineMetadataFrame, AdaptMIPMFrameACMM.cu:903-929).
// Bound by instruction issue, as the half-sweep.  Against one thread per pixel
// over chunks of neighbours (the lanes' windows and taps differ, IEEE divisions per
// blur tap): 16.0 -> 4.2 ms (2048x1536, 12 neighbours, 15x15), 51.8 -> 3.6 ms
// (1531x1147, 17, 13x13, blur, shifted), 1.78 -> 0.58 ms (1024x768, 6, 11x11).
namespace {

constexpr int kInitWarps = 16, kInitCtas = 2;

struct InitPlan {
    int off_ctl, off_Q, off_QB, off_R, off_RB, off_geo, off_ok, off_as, off_ac, off_bins;
    int off_stage, off_wtab, off_plane, off_dp, off_cost, off_id, off_order;
    int rs, tx, ty, tab_n, nbins, kc, total;

    __host__ __device__ static int a16(int v) { return (v + 15) & ~15; }
    __host__ __device__ static InitPlan make(int W, int H, int K, int ntap, bool blur, int tile_stride, int chunk)
    {
        InitPlan p;
        p.rs = H | 1;
        p.tx = ntap < W ? ntap : W;
        p.ty = ntap < H ? ntap : H;
        p.tab_n = p.tx * p.ty;
        p.nbins = (p.tx / 2 + 1) * p.ty;
        p.kc = K | 1;                                    // odd: threads read rows side by side
        int o = 16;
        p.off_ctl = o;   o += 16;
        const int q_bytes = a16(K * (H + 1) * (W + 1) * 4), r_bytes = a16((2 * W * p.rs + 2 * H) * 4);
        p.off_Q = o;     o += q_bytes;
        p.off_QB = o;    o += blur ? q_bytes : 0;
        p.off_R = o;     o += r_bytes;
        p.off_RB = o;    o += blur ? r_bytes : 0;
        p.off_geo = o;   o += a16(K * (int)sizeof(NbGeo));
        p.off_ok = o;    o += a16(K * 4);
        p.off_as = o;    o += a16(ntap * ntap * 4);
        p.off_ac = o;    o += 256 * 4;
        p.off_bins = o;  o += a16(p.nbins * 4);
        p.off_stage = o;                                 // shares what follows, as in the half-sweep
        const int stage_end = o + a16((1 + K) * tile_stride * (blur ? 2 : 1));
        p.off_wtab = o;  o += a16(chunk * p.tab_n * 4);
        p.off_plane = o; o += chunk * 16;
        p.off_dp = o;    o += chunk * 16;
        p.off_cost = o;  o += a16(chunk * p.kc * 4);
        p.off_id = o;    o += a16(chunk * K * 2);
        p.off_order = o; o += a16(chunk * K * 2);
        const int walk_end = p.off_wtab + (chunk + 1) * p.tab_n * 4 + 64;
        if (o < stage_end) o = stage_end;
        if (o < walk_end) o = a16(walk_end);
        p.total = o;
        return p;
    }
};

}  // namespace

template <bool BLUR, bool SHIFT>
__global__ void __launch_bounds__(32 * kInitWarps, kInitCtas)
pm_init_kernel(FrameDev F, PmParams P, StateDev out, int* err, int refit, int chunk, int parts)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int W = P.W, H = P.H, K = P.K;
    const InitPlan L = InitPlan::make(W, H, K, P.ntap, BLUR, P.tile_stride, chunk);
    {
        uint32_t dyn;
        asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (L.total > (int)dyn || chunk < 1 || chunk * 32 > 65536 || parts < 1) {
            if (threadIdx.x == 0) atomicOr(err, PFD_DEVERR_SWEEP_CHECK);
            return;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    int* ctl = (int*)(smem + L.off_ctl);                 // 0: tasks, 1: next pass
    float* R = (float*)(smem + L.off_R);
    int* bins = (int*)(smem + L.off_bins);
    const float* a_s = (const float*)(smem + L.off_as);
    const float* a_c = (const float*)(smem + L.off_ac);
    float* wtab = (float*)(smem + L.off_wtab);
    float4* plane = (float4*)(smem + L.off_plane);
    float4* dps = (float4*)(smem + L.off_dp);
    float* cost = (float*)(smem + L.off_cost);
    uint16_t* t_id = (uint16_t*)(smem + L.off_id);
    uint16_t* t_order = (uint16_t*)(smem + L.off_order);
    StageDst D;
    D.stage = smem + L.off_stage;
    D.bar = (uint64_t*)smem;
    D.R = R;
    D.RB = (float*)(smem + L.off_RB);
    D.Q = (uint32_t*)(smem + L.off_Q);
    D.QB = (uint32_t*)(smem + L.off_QB);
    D.geo = (NbGeo*)(smem + L.off_geo);
    D.ok = (int*)(smem + L.off_ok);
    D.rs = L.rs;
    EvalEnv E;
    E.wtab = smem_u32(wtab);
    E.R = smem_u32(R);
    E.RB_delta = BLUR ? (uint32_t)(L.off_RB - L.off_R) : 0u;
    E.Q = smem_u32(D.Q);
    E.QB_delta = BLUR ? (uint32_t)(L.off_QB - L.off_Q) : 0u;
    E.q_bytes = (H + 1) * (W + 1) * 4;
    E.tab_n = L.tab_n;
    E.rs = L.rs;
    E.inc = P.inc;
    E.wb = P.W_bits;
    E.hb = P.H_bits;
    E.kq = ((uint32_t)(W + 1) * 4u << 24) | (4u << 16);
    const float inv_inc = 1.0f / (float)P.inc;
    if (tid == 0) mbar_init(D.bar, 1);
    fill_tables<BLUR>(P, (float*)(smem + L.off_as), (float*)(smem + L.off_ac), R, D.RB, L.rs);
    for (int e = tid; e < L.nbins; e += blockDim.x) bins[e] = 0;
    uint32_t parity = 0;
    for (int item = blockIdx.x; item < F.V * parts; item += gridDim.x) {
        const int vid = item / parts, part = item - vid * parts;
        const int p_lo = (int)((long long)P.ppv * part / parts), p_hi = (int)((long long)P.ppv * (part + 1) / parts);
        const int nc = min(F.nb_counts[vid], K);
        const size_t vbase = (size_t)vid * P.ppv;
        __syncthreads();                                 // the previous item's shared memory is free
        if (tid == 0) {
            start_copies<BLUR>(D, F, P, vid, nc > 0 ? nc : 0);
            ctl[0] = 0;
        }
        stage_geo(D, F, P, vid, nc, err);
        const bool ok = mbar_wait_bounded(D.bar, parity, err);
        if (__syncthreads_or(!ok)) return;
        parity ^= 1u;
        expand_tiles<BLUR>(D, P, nc > 0 ? nc : 0);
        __syncthreads();
        for (int e0 = p_lo; e0 < p_hi; e0 += chunk) {
            const int np = min(chunk, p_hi - e0);
            // ---- planes, weight tables
            for (int p = tid; p < np; p += blockDim.x) {
                const int e = e0 + p, y = e / W, x = e - y * W;
                const size_t idx = vbase + e;
                float4 h;
                if (refit) {
                    h = out.plane[idx];
                } else {
                    DrawStream g;
                    g.init(P.seed, 0u, (uint32_t)idx);
                    h = random_plane(g, P.depth_min, P.depth_max);
                }
                plane[p] = h;
                const float3 dp = disparity_plane(x, y, h);
                dps[p] = make_float4(dp.x, dp.y, dp.z, to_disparity(x, y, dp));
            }
            for (int p = warp; p < np; p += kInitWarps) {
                const int e = e0 + p, y = e / W, x = e - y * W;
                const PixWin pw = slot_window(P, x, y);
                const float rc = R[x * L.rs + y];
                const int n = pw.nX * pw.nY;
                const uint32_t magic = pw.nY > 1 ? 0xFFFFFFFFu / (uint32_t)pw.nY + 1u : 0u;
                for (int t = lane; t < n; t += 32) {
                    const int ix = pw.nY > 1 ? (int)__umulhi((uint32_t)t, magic) : t, iy = t - ix * pw.nY;
                    wtab[p * L.tab_n + t] = tap_weight(R, L.rs, a_s, a_c, P, pw, ix, iy, rc);
                }
            }
            __syncthreads();
            // ---- the NCCs of the chunk, sorted by rectangle
            const int total = np * nc;
            for (int i0 = warp * 32; i0 < total; i0 += 32 * kInitWarps) {
                const int i = i0 + lane;
                const int p = i / nc, k = i - p * nc;
                uint32_t rect = 0u;
                if (i < total) {
                    const int e = e0 + p, y = e / W, x = e - y * W;
                    if (D.ok[k]) {
                        const float4 d = dps[p];
                        const NbGeo g = D.geo[k];
                        const float2 a = geo_anchor(g, x, y, d.w);
                        if ((__float_as_uint(a.x) < P.W_bits) && (__float_as_uint(a.y) < P.H_bits))
                            rect = tap_rect(slot_window(P, x, y), P, make_float3(d.x, d.y, d.z), g.stx, g.sty, inv_inc);
                    }
                    cost[p * L.kc + k] = rect ? __uint_as_float(rect) : kCostMax;
                }
                const uint32_t m = __ballot_sync(kFullMask, rect != 0u);
                if (!m) continue;
                int at = 0;
                if (lane == 0) at = atomicAdd(&ctl[0], __popc(m));
                at = __shfl_sync(kFullMask, at, 0) + __popc(m & ((1u << lane) - 1u));
                if (rect) {
                    t_id[at] = (uint16_t)((p << 5) | k);
                    atomicAdd(&bins[rect_bin(rect, L.tx, L.ty)], 1);
                }
            }
            __syncthreads();
            const int n_tasks = ctl[0];
            if (warp == 0) {
                scan_bins(bins, L.nbins, lane);
                if (lane == 0) ctl[1] = 0;
            }
            __syncthreads();
            for (int i = tid; i < n_tasks; i += blockDim.x) {
                const int id = t_id[i];
                const uint32_t rect = __float_as_uint(cost[(id >> 5) * L.kc + (id & 31)]);
                t_order[atomicAdd(&bins[rect_bin(rect, L.tx, L.ty)], 1)] = (uint16_t)id;
            }
            __syncthreads();
            for (int e = tid; e < L.nbins; e += blockDim.x) bins[e] = 0;
            if (tid == 0) ctl[0] = 0;
            for (;;) {
                int q = 0;
                if (lane == 0) q = atomicAdd(&ctl[1], 1);
                q = __shfl_sync(kFullMask, q, 0);
                if (q * 32 >= n_tasks) break;
                const bool act = q * 32 + lane < n_tasks;
                const int id = act ? t_order[q * 32 + lane] : 0;
                const int p = id >> 5, k = id & 31;
                const int e = e0 + p, y = e / W, x = e - y * W;
                float* cell = cost + p * L.kc + k;
                const uint32_t rect = act ? __float_as_uint(*cell) : 0u;
                const float4 d = dps[p];
                const PixWin pw = slot_window(P, x, y);
                const int i0 = rect & 0xFF, j0 = (rect >> 8) & 0xFF;
                const int X = pw.x0 + i0 * P.inc, Y = pw.y0 + j0 * P.inc;
                Moments M = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
                const float sh = SHIFT ? R[x * L.rs + y] : 0.0f;
                walk<BLUR, SHIFT>(M, E, make_float3(d.x, d.y, d.z), D.geo[k].stx, D.geo[k].sty,
                                  (int)((rect >> 16) & 0xFFu), (int)(rect >> 24),
                                  E.wtab + (uint32_t)(p * L.tab_n + i0 * pw.nY + j0) * 4u,
                                  E.R + (uint32_t)(X * L.rs + Y) * 4u, (uint32_t)pw.nY * 4u, (float)X, (float)Y,
                                  E.Q + (uint32_t)(k * E.q_bytes), sh);
                if (act) *cell = ncc_cost<BLUR>(M, P.blur_gain);
            }
            __syncthreads();
            // ---- the pixel's cost, views and disp: the top-k of its vector
            for (int p = tid; p < np; p += blockDim.x) {
                const int e = e0 + p, y = e / W, x = e - y * W;
                const size_t idx = vbase + e;
                const float* cs = cost + p * L.kc;
                int best_idx = -1, valid = 0;
                for (int i = 0; i < nc; ++i) {
                    const float c = cs[i];
                    if (c < 2.0f) {
                        ++valid;
                        if (best_idx < 0 || c < cs[best_idx]) best_idx = i;
                    }
                }
                float mean = 2.0f;
                uint32_t mask = 0;
                if (valid > 0) {
                    // the k smallest in ascending order
                    const int kk = min(valid, P.top_k);
                    uint32_t used = 0;
                    float m = 0.0f, low = 0.0f;
                    for (int i = 0; i < kk; ++i) {
                        int at = -1;
                        for (int j = 0; j < nc; ++j)
                            if (!((used >> j) & 1u) && (at < 0 || cs[j] < low)) { at = j; low = cs[j]; }
                        used |= 1u << at;
                        m = __fadd_rn(m, low);
                    }
                    mean = __fdiv_rn(m, (float)kk);
                    for (int i = 0; i < nc; ++i)
                        if (cs[i] <= low) mask |= (1u << i);
                }
                const float4 h = plane[p];
                float4 disp = make_float4(0.f, 0.f, 0.f, 0.f);
                if (best_idx >= 0) disp = geo_disp(D.geo[best_idx], x, y, to_disparity(x, y, disparity_plane(x, y, h)));
                if (!refit) out.plane[idx] = h;
                out.cost[idx] = mean;
                out.disp[idx] = disp;
                out.sel[idx] = mask;
            }
            if (P.cvec)
                for (int i = tid; i < total; i += blockDim.x) {
                    const int p = i / nc, k = i - p * nc;
                    P.cvec[(vbase + e0 + p) * K + k] = cost[p * L.kc + k];
                }
            __syncthreads();                             // the chunk's planes and costs are free
        }
    }
}

template <bool BLUR, bool SHIFT, int SHAPE>
__global__ void __launch_bounds__(32 * ShapeOf<SHAPE>::warps, ShapeOf<SHAPE>::min_ctas)
pm_slots_kernel(FrameDev F, PmParams P, StateDev prev, StateDev next, int iter, int phase, int* err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    init_barrier(smem);
    uint32_t parity = 0;
    sweep_slots<BLUR, SHIFT, ShapeOf<SHAPE>::warps>(smem, F, P, prev, next, iter, phase, err, parity);
}

// Several frames' half-sweeps in one launch, in list order: a CTA that finds a
// frame's queue empty moves on to the next frame at once, so one frame's tail
// overlaps the next one's start.  The dynamic shared memory is the largest of
// the frames' plans.
template <bool BLUR, bool SHIFT, int SHAPE>
__global__ void __launch_bounds__(32 * ShapeOf<SHAPE>::warps, ShapeOf<SHAPE>::min_ctas)
pm_slots_batch_kernel(const SweepItem* items, int n, int* err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    init_barrier(smem);
    uint32_t parity = 0;
    for (int b = 0; b < n; ++b) {
        const SweepItem it = items[b];
        if (!sweep_slots<BLUR, SHIFT, ShapeOf<SHAPE>::warps>(smem, it.F, it.P, it.prev, it.next, it.iter, it.phase, err,
                                                             parity))
            return;
    }
}

cudaError_t launch_init(const FrameDev& F, const PmParams& P, const StateDev& out, int* err, cudaStream_t st, bool refit)
{
    const bool blur = F.blur != nullptr;
    if (F.V <= 0) return cudaSuccess;
    // chunk: the pixels whose tables fit two CTAs per SM, or one
    int chunk = 0, smem = 0;
    for (int ctas = kInitCtas; ctas >= 1 && !smem; --ctas) {
        const int budget = std::min(227 * 1024, (228 * 1024) / ctas - 1024);
        for (int c = std::min(128, P.ppv); c >= 1; --c) {
            if (ctas > 1 && c < std::min(32, P.ppv)) break;
            const InitPlan L = InitPlan::make(P.W, P.H, P.K, P.ntap, blur, P.tile_stride, c);
            if (L.total > budget) continue;
            chunk = c;
            smem = L.total;
            break;
        }
    }
    if (!smem) return cudaErrorInvalidValue;
    const int chunks = (P.ppv + chunk - 1) / chunk;
    chunk = (P.ppv + chunks - 1) / chunks;               // equal chunks
    const void* k = P.shifted ? (blur ? (const void*)pm_init_kernel<true, true> : (const void*)pm_init_kernel<false, true>)
                              : (blur ? (const void*)pm_init_kernel<true, false> : (const void*)pm_init_kernel<false, false>);
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * kInitWarps, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    // a frame of few micro-images splits them by chunks, so that every SM has work
    int parts = 1;
    while (parts < chunks && (long long)F.V * parts < 4LL * sms * per_sm) parts = std::min(chunks, parts * 2);
    const int grid = (int)std::min<long long>((long long)sms * per_sm, (long long)F.V * parts);
    FrameDev f = F; PmParams p = P; StateDev o = out; int* er = err; int r = refit ? 1 : 0;
    void* args[] = { &f, &p, &o, &er, &r, &chunk, &parts };
    return cudaLaunchKernel(k, dim3(grid), dim3(32 * kInitWarps), args, (size_t)smem, st);
}

int slots_shape_warps(int shape) { return kShapeWarps[(shape >= 0 && shape < kSweepShapes) ? shape : 0]; }
int slots_shape_ctas(int shape) { return kShapeCtas[(shape >= 0 && shape < kSweepShapes) ? shape : 0]; }

// Slots, list capacity and parts of a half-sweep; returns the dynamic shared
// memory of its plan, or 0 when none fits.  A launch of fewer than six items per
// CTA splits its micro-images, so that no CTA is without work and the last ones end
// together; a part stages the micro-image anew and drains its slots.  Measured at 1, 2, 4
// and 8 parts over 63 frames, 0.3 to 22 micro-images per CTA, windows of 10x10 to
// 20x20, patches of 5x5 to 15x15, with and without blur and ACMM: the rule's choice is
// 1.1% off the best on average, 2.4% with the line at two items.  Half-sweep, ms (16x16,
// 12 neighbours, 15x15, 296 CTAs): 195 micro-images 1.19, .92, .93, .98; 1554 (5.3 items)
// 6.02, 5.85, 6.13, 6.77; 1840 (6.2) 6.84, 6.90, 7.23, 7.98; 6612 23.3, 24.1, 25.5, 28.4.
// ACMM (5x5) gains 2-5% from two parts also above six items.  No part gets fewer pixels
// than slots: 10x10 windows (50 pixels, 32 slots) at one and two parts .41 and .43 ms at
// 2.2 items, .72 and .75 at 4.1; the smallest frames would gain (100 of them, .3 items:
// .141 and .123 ms).
int slots_plan(PmParams& P, bool blur, int shape, int n_views)
{
    const int warps = slots_shape_warps(shape);
    for (int ctas = slots_shape_ctas(shape); ctas >= 1; --ctas) {
        const int budget = std::min(227 * 1024, (228 * 1024) / ctas - 1024);
        for (int s = std::min(32, 2 * warps); s >= 1; --s) {
            if (ctas > 1 && s < warps) break;            // fewer slots than warps: fewer CTAs instead
            const int cap = std::max(slot_tasks(P.K), s * 9 * P.K);
            const SlotPlan L = SlotPlan::make(P.W, P.H, P.K, P.ntap, blur, P.tile_stride, s, cap);
            if (L.total > budget) continue;
            P.slots = s;
            P.task_cap = cap;
            int dev = 0, sms = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            const int n_upd = (P.ppv + 1) / 2;
            P.parts = 1;
            while ((long long)n_views * P.parts < 6LL * sms * ctas && n_upd / (2 * P.parts) >= s) P.parts *= 2;
            return L.total;
        }
    }
    return 0;
}

template <int SHAPE>
static const void* slots_kernel_of(bool blur, bool shift)
{
    if (shift) return blur ? (const void*)pm_slots_kernel<true, true, SHAPE> : (const void*)pm_slots_kernel<false, true, SHAPE>;
    return blur ? (const void*)pm_slots_kernel<true, false, SHAPE> : (const void*)pm_slots_kernel<false, false, SHAPE>;
}

static const void* slots_kernel(int shape, bool blur, bool shift)
{
    switch (shape) {
    case 1: return slots_kernel_of<1>(blur, shift);
    case 2: return slots_kernel_of<2>(blur, shift);
    case 3: return slots_kernel_of<3>(blur, shift);
    default: return slots_kernel_of<0>(blur, shift);
    }
}

template <int SHAPE>
static const void* slots_batch_kernel_of(bool blur, bool shift)
{
    if (shift) return blur ? (const void*)pm_slots_batch_kernel<true, true, SHAPE>
                           : (const void*)pm_slots_batch_kernel<false, true, SHAPE>;
    return blur ? (const void*)pm_slots_batch_kernel<true, false, SHAPE>
                : (const void*)pm_slots_batch_kernel<false, false, SHAPE>;
}

static const void* slots_batch_kernel(int shape, bool blur, bool shift)
{
    switch (shape) {
    case 1: return slots_batch_kernel_of<1>(blur, shift);
    case 2: return slots_batch_kernel_of<2>(blur, shift);
    case 3: return slots_batch_kernel_of<3>(blur, shift);
    default: return slots_batch_kernel_of<0>(blur, shift);
    }
}

// A plan of more than half of an SM's shared memory runs one CTA per SM whatever the
// kernel's registers are bounded for: the default shape then runs the kernel of as many
// warps with the registers of one CTA (a half-sweep at 1531x1147, 17
// neighbours, 13x13, blur: 21.7 -> 20.3 ms).  Where two CTAs fit, the default's kernel:
// 23.5 against 27.5 ms (2048x1536, 12, 15x15).
static_assert(ShapeOf<0>::warps == ShapeOf<3>::warps && ShapeOf<3>::min_ctas == 1, "shapes of one_cta_shape");
static int one_cta_shape(int shape, int smem) { return shape == 0 && smem > (228 * 1024) / 2 - 1024 ? 3 : shape; }

static cudaError_t slots_grid(const void* k, int threads, int smem, int* n_ctas)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    *n_ctas = sms * per_sm;
    return cudaSuccess;
}

cudaError_t slots_sweep_grid(const FrameDev& F, const PmParams& P, int smem, int* n_ctas, int shape)
{
    shape = one_cta_shape(shape, smem);
    return slots_grid(slots_kernel(shape, F.blur != nullptr, P.shifted != 0), 32 * slots_shape_warps(shape), smem, n_ctas);
}

cudaError_t launch_slots_sweep(const FrameDev& F, const PmParams& P, const StateDev& prev, const StateDev& next, int iter,
                               int phase, int smem, int n_ctas, int* err, cudaStream_t st, int shape)
{
    if (smem <= 0 || smem > 227 * 1024) return cudaErrorInvalidConfiguration;
    shape = one_cta_shape(shape, smem);
    const void* k = slots_kernel(shape, F.blur != nullptr, P.shifted != 0);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(P.view_queue, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, (int)std::min<long long>(n_ctas, (long long)F.V * P.parts));
    FrameDev f = F; PmParams p = P; StateDev a = prev, b = next; int it = iter, ph = phase; int* er = err;
    void* args[] = { &f, &p, &a, &b, &it, &ph, &er };
    return cudaLaunchKernel(k, dim3(grid), dim3(32 * slots_shape_warps(shape)), args, (size_t)smem, st);
}

cudaError_t slots_batch_grid(int smem, bool blur, bool shift, int* n_ctas, int shape)
{
    shape = one_cta_shape(shape, smem);
    return slots_grid(slots_batch_kernel(shape, blur, shift), 32 * slots_shape_warps(shape), smem, n_ctas);
}

cudaError_t launch_slots_batch(const SweepItem* items, int n, bool blur, bool shift, int smem, int n_ctas, int* err,
                               cudaStream_t st, int shape)
{
    if (n <= 0) return cudaSuccess;
    if (smem <= 0 || smem > 227 * 1024) return cudaErrorInvalidConfiguration;
    shape = one_cta_shape(shape, smem);
    const void* k = slots_batch_kernel(shape, blur, shift);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    const SweepItem* it = items; int nn = n; int* er = err;
    void* args[] = { &it, &nn, &er };
    return cudaLaunchKernel(k, dim3(std::max(1, n_ctas)), dim3(32 * slots_shape_warps(shape)), args, (size_t)smem, st);
}

}  // namespace pfd
