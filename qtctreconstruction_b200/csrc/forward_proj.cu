// forward_proj.cu — the forward projector (the RadonTransform stage of the
// FBP path).
//
// The reference's forward projector (SerialBackend::computeSinogram,
// SerialBackend.cpp:59-136) splats every non-zero pixel onto the two detector
// bins around s = (x-cx)cos + (y-cy)sin + floor(nd/2) with weights
// (1 - frac, frac), frac = s - floor(s). For bins 1 .. nd-2 that is the hat
// function: bin b = sum over pixels of v * max(0, 1 - |s - b|). Bins 0 and
// nd-1 follow the reference's own rules instead (a pixel with floor(s) = -1
// adds nothing to bin 0; floor(s) = nd-1 adds its full value to bin nd-1).
//
// Here a warp computes a strip of K consecutive output bins of one angle for
// 4 NP slices, walking the image along the axis the detector is closest to
// (rows when |cos| >= |sin|, else columns of the transposed copy). At walked
// row p the strip's pixels are the 32 consecutive columns from the crossing
// q*(p) of its lower bin edge: lane l owns column rint(q*) + S l (S the sign
// of ds/dq), whose offset from the crossing is u = (l + phi) |kq| in bins,
// phi = S (rint(q*) - q*) in [-1/2, 1/2]. So every row is one coalesced load
// of 32 neighbouring pixels (each the 8 slices of a plane pair, 32 bytes, one
// 256-bit load per lane), and lane l's pixel
// always falls in bin m_l or m_l + 1 of the strip, m_l = floor((l - 1/2)
// |kq|), whatever the row: the lane keeps three accumulators, for bins m_l,
// m_l + 1 and m_l + 2, adding v times the hat weights of its pixel. At the
// end of the walk the warp adds, per output bin, the accumulators of the few
// lanes that reach it, in lane order, gathered by warp shuffles. K is chosen per
// angle group so that K + 1 <= 31.5 |kq|: the lanes' pixels cover the
// strip's bins and the bin on either side.
//
// What a row needs beside the pixels is the same for all lanes: its column and
// phi. So the warp prepares 32 rows at a time, lane r evaluating row r's crossing
// in double and testing its 32 columns against the non-zero pixels of the row's
// 8-row band; the walk then reads each row's two values from shared memory (one
// broadcast) where every lane computing them for itself took 12 more
// instructions per row. 8-row groups without a needed row are skipped. Reading
// rows within one row of the range where the strip's columns, at most 31.5 wide,
// come within kReach = 2 columns of the non-zero box (or of the image without
// bounds), or at most 7 rows beyond it, with |dq*/dp| <= 1, the 32-column window
// stays within 50 columns of the image on either side: inside the kFwdGuard = 64
// border, which reads as zeros.
//
// Bound by the L1 data path (about 9 wavefronts per row of 1 KB, 74 % busy at 512^2
// x 32 x 720 without zeros) and issue (28 instructions per row, 12 of them packed
// FP32x2 of two issue cycles): 5.56 -> 4.51 ms at 512^3 x 720 of the benchmark
// phantom, 3.00 -> 2.53 ms at 512^2 x 64 x 720 without zeros, against each lane
// preparing its rows. Measured there and not kept: 16 slices per lane (3.53 ms), 8
// angles per CTA (2.92), 6 or 8 CTAs per SM (2.77, 3.37), four rows' loads ahead
// (2.55), prefetching the next rows into L1 (2.61), saturating weights (2.54).
//
// The warps of a CTA are the up to GMAX = 4 angles of a group that share the
// walked axis, on the same strip index; after one barrier that ends the set-up
// (per-angle constants from the plan's FwdAngleRec table) they walk the same rows
// at nearly the same columns and share the L1 lines, and never wait on one
// another again.
// Bins 0 and nd-1 are recomputed by the warp whose strip holds them, with one
// lane per row deciding on the reference's own float s for the few pixels
// around those bins.
#include <climits>
#include <cmath>

#include "ctb_internal.h"

namespace ctb {
namespace {

constexpr int LANES = 32;
constexpr int PCH = kFwdRows;  // zero rows below the image
constexpr int GMAX = kFwdGroup;
constexpr int THREADS = LANES * GMAX;
constexpr int NP = kFwdPlanes;          // float4 planes (4 slices each) per thread
static_assert(kFwdGuard >= 50, "the walked windows reach 50 columns outside the image");
static_assert(PCH >= 8, "an 8-row group may start at the image's last row");
static_assert(NP == 2, "a pixel holds the 8 slices of a plane pair: two float4, one 32-byte load");

struct FAngle {
    double q0;   // crossing of the strip's lower edge (bin b_lo = k K - 1) at p = 0
    double inv;  // dq*/db = 1 / kq
    double dq;   // dq*/dp = -kp / kq
    float akq;     // |kq|: bins per pixel step along the walked row
    float cf, sf;  // the reference's float cos/sin
    int a;
    int p_lo, p_hi;  // rows where the strip meets the non-zero box and disc
    int c_lo, c_hi;  // columns of the non-zero box
    int neg;         // kq < 0: the strip's columns decrease with the bin
};

__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
// One pixel of a plane pair: 8 slices in 32 bytes (32-byte aligned), one load, not
// through the read-only path (the normalisation before this kernel may still run when
// it starts). It stays behind chain_wait without being volatile, because its address
// comes from a row record written after the block's barrier; volatile keeps the loads
// from being spread over a row group's arithmetic (1148 -> 1165 us at 387^2 x 50 x 580).
__device__ __forceinline__ void ld_pixel(const float4* p, float4 (&v)[NP]) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[0].z), "=f"(v[0].w), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[1].z),
          "=f"(v[1].w)
        : "l"(p));
}
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Lane l's first bin (relative to b_lo): floor((l - 1/2) |kq|). The combine
// step evaluates exactly this expression again for other lanes.
__device__ __forceinline__ int lane_bin(int l, float akq) {
    return static_cast<int>(floorf((static_cast<float>(l) - 0.5f) * akq));
}

// One walked row of the strip, as one lane prepares it for the warp.
struct RowRec {
    float dy;      // S (rint(q*) - q*) |kq|: the pixels' offset from their nominal place, in bins
    unsigned col;  // pixel index of column rint(q*) from the block's first row, left border included
};

// Eight rows of a block. Lane l's pixel of a row lies y = cl1 + dy bins from bin
// m_l + 1 (cl1 = l |kq| - m_l - 1), y in [-1, 1], which gives its hat weights
// for bins m_l, m_l + 1, m_l + 2: max(-y, 0), 1 - |y|, max(y, 0).
__device__ __forceinline__ void walk_rows(const float4* lane_base, const RowRec* __restrict__ rr,
                                          float cl1, float2 (&acc)[3][2 * NP]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float y = cl1 + rr[i].dy;
        const float w0 = fmaxf(-y, 0.0f), w2 = fmaxf(y, 0.0f), w1 = 1.0f - fabsf(y);
        const float2 W0 = make_float2(w0, w0), W1 = make_float2(w1, w1), W2 = make_float2(w2, w2);
        float4 v[NP];
        ld_pixel(lane_base + 2ull * rr[i].col, v);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            acc[0][2 * k] = __ffma2_rn(W0, lo2(v[k]), acc[0][2 * k]);
            acc[0][2 * k + 1] = __ffma2_rn(W0, hi2(v[k]), acc[0][2 * k + 1]);
            acc[1][2 * k] = __ffma2_rn(W1, lo2(v[k]), acc[1][2 * k]);
            acc[1][2 * k + 1] = __ffma2_rn(W1, hi2(v[k]), acc[1][2 * k + 1]);
            acc[2][2 * k] = __ffma2_rn(W2, lo2(v[k]), acc[2][2 * k]);
            acc[2][2 * k + 1] = __ffma2_rn(W2, hi2(v[k]), acc[2][2 * k + 1]);
        }
    }
}

// The same for a single slice (4-byte pixels), two rows at a time: the two lanes
// of a packed operation hold an even and an odd row, so the weights need no copies.
__device__ __forceinline__ void walk_rows(const float* lane_base, const RowRec* __restrict__ rr, float cl1,
                                          float2 (&acc)[3]) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float2 v = make_float2(ld_chained(lane_base + rr[i].col), ld_chained(lane_base + rr[i + 1].col));
        const float2 y = make_float2(cl1 + rr[i].dy, cl1 + rr[i + 1].dy);
        acc[0] = __ffma2_rn(make_float2(fmaxf(-y.x, 0.0f), fmaxf(-y.y, 0.0f)), v, acc[0]);
        acc[1] = __ffma2_rn(make_float2(1.0f - fabsf(y.x), 1.0f - fabsf(y.y)), v, acc[1]);
        acc[2] = __ffma2_rn(make_float2(fmaxf(y.x, 0.0f), fmaxf(y.y, 0.0f)), v, acc[2]);
    }
}

// Bins 0 and nd-1 by the reference's rules (SerialBackend.cpp:109-120), on
// its own float s: bin 0 takes (1 - frac) v from the pixels with floor(s) =
// 0, bin nd-1 takes frac v from floor(s) = nd-2 and v from floor(s) = nd-1.
// Lane l takes rows r_lo + l, r_lo + l + 32, ... up to r_hi; in each row the
// candidates are the columns whose exact s lies within 1/64 of [lo, hi] =
// [0, 1] (bin 0) or [nd-2, nd] (bin nd-1), the reference's float s being
// much closer than that to the exact one. The lanes' sums are added by a
// fixed shuffle tree; every lane returns the total.
__device__ __noinline__ void edge_bin(const float4* plane, int pitch, int nq,
                                      const FAngle& f, int b_lo, int e, int nd, int r_lo, int r_hi, bool rows,
                                      float cxf, float cyf, int lane, float2 (&sum)[2 * NP]) {
#pragma unroll
    for (int j = 0; j < 2 * NP; ++j) sum[j] = make_float2(0.0f, 0.0f);
    const double lo = e == 0 ? 0.0 : nd - 2.0, hi = e == 0 ? 1.0 : static_cast<double>(nd);
    const double da = (lo - 1.0 / 64 - b_lo) * f.inv, db = (hi + 1.0 / 64 - b_lo) * f.inv;
    const float dcs = static_cast<float>(nd / 2);
    for (int p = r_lo + lane; p <= r_hi; p += LANES) {
        const double qp = fma(static_cast<double>(p), f.dq, f.q0);
        const int c0 = static_cast<int>(ceil(qp + fmin(da, db)));
        const int c1 = min(static_cast<int>(floor(qp + fmax(da, db))), c0 + 5);
        for (int c = max(c0, 0); c <= min(c1, nq - 1); ++c) {
            const float xg = static_cast<float>(rows ? c : p);
            const float yg = static_cast<float>(rows ? p : c);
            const float ss = __fadd_rn(__fadd_rn(__fmul_rn(__fsub_rn(xg, cxf), f.cf),
                                                 __fmul_rn(__fsub_rn(yg, cyf), f.sf)), dcs);
            const float fl = floorf(ss);
            const int i0 = static_cast<int>(fl);
            const float fr = __fsub_rn(ss, fl);
            float wgt = 0.0f;
            if (e == 0) wgt = i0 == 0 ? __fsub_rn(1.0f, fr) : 0.0f;
            else wgt = i0 == nd - 2 ? fr : (i0 == nd - 1 ? 1.0f : 0.0f);
            if (wgt == 0.0f) continue;
            const float2 W = make_float2(wgt, wgt);
            const float4* px = plane + 2 * (static_cast<long long>(p) * pitch + c);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const float4 v = ld_chained(px + k);
                sum[2 * k] = __ffma2_rn(W, lo2(v), sum[2 * k]);
                sum[2 * k + 1] = __ffma2_rn(W, hi2(v), sum[2 * k + 1]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2 * NP; ++j)
        for (int o = 16; o > 0; o >>= 1) {
            sum[j].x += __shfl_xor_sync(0xffffffffu, sum[j].x, o);
            sum[j].y += __shfl_xor_sync(0xffffffffu, sum[j].y, o);
        }
}

// edge_bin of a single slice.
__device__ __noinline__ float edge_bin(const float* plane, int pitch, int nq, const FAngle& f, int b_lo, int e,
                                       int nd, int r_lo, int r_hi, bool rows, float cxf, float cyf, int lane) {
    float sum = 0.0f;
    const double lo = e == 0 ? 0.0 : nd - 2.0, hi = e == 0 ? 1.0 : static_cast<double>(nd);
    const double da = (lo - 1.0 / 64 - b_lo) * f.inv, db = (hi + 1.0 / 64 - b_lo) * f.inv;
    const float dcs = static_cast<float>(nd / 2);
    for (int p = r_lo + lane; p <= r_hi; p += LANES) {
        const double qp = fma(static_cast<double>(p), f.dq, f.q0);
        const int c0 = static_cast<int>(ceil(qp + fmin(da, db)));
        const int c1 = min(static_cast<int>(floor(qp + fmax(da, db))), nq - 1);
        // at most (2 + 1/32) sqrt(2) < 3 columns; the loads do not wait for the weights
        float wgt[3], v[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int c = c0 + i;
            const bool in = c >= 0 && c <= c1;
            v[i] = ld_chained(plane + static_cast<long long>(p) * pitch + (in ? c : 0));
            const float xg = static_cast<float>(rows ? c : p);
            const float yg = static_cast<float>(rows ? p : c);
            const float ss = __fadd_rn(__fadd_rn(__fmul_rn(__fsub_rn(xg, cxf), f.cf),
                                                 __fmul_rn(__fsub_rn(yg, cyf), f.sf)), dcs);
            const float fl = floorf(ss);
            const int i0 = static_cast<int>(fl);
            const float fr = __fsub_rn(ss, fl);
            if (e == 0) wgt[i] = i0 == 0 ? __fsub_rn(1.0f, fr) : 0.0f;
            else wgt[i] = i0 == nd - 2 ? fr : (i0 == nd - 1 ? 1.0f : 0.0f);
            if (!in) wgt[i] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (wgt[i] != 0.0f) sum = fmaf(wgt[i], v[i], sum);
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// PER_SM: the CTAs per SM the registers are held to. Seven (72 registers) for
// launches that fill the SMs. A launch that does not is bound by the latency of its
// loads: four per SM (127 registers) let a warp have all eight rows of a group on
// their way (us of a whole call, seven against four: 45.1 and 33.4 at 160^2 x 1 x
// 180, 39.0 and 29.8 at 128^2 x 8 x 180, 28.7 and 22.6 at 64^2 x 1 x 90; but 72.0
// and 73.3 at 256^2 x 1 x 360 with 1620 CTAs, 2563 and 2714 at 512^2 x 64 x 720). A
// single slice in planes of its own needs 72 registers either way.
constexpr int FULL = 7, SPARSE = 4;
// ONE: a single slice in planes of 4-byte pixels (img, imgT then point to floats):
// a row of 32 columns is one or two L1 wavefronts instead of nine and a row takes a
// quarter of the instructions (us of a whole call: 27.3 -> 18.8 at 160^2 x 180, 66.5 ->
// 34.6 at 256^2 x 360, 348 -> 154 at 512^2 x 720, 2336 -> 991 at 1024^2 x 1440).
template <int PER_SM, bool ONE>
__global__ void __launch_bounds__(THREADS, PER_SM)
    k_forward(const float4* img, const float4* imgT, int w, int h, int nz, int na, int nd,
              const int4* __restrict__ groups, const FwdAngleRec* __restrict__ arec, const int4* box,
              const int2* band, float* __restrict__ sino) {
    __shared__ FAngle fa[GMAX];
    __shared__ int erow[GMAX][4];                      // edge-pass rows: bin 0 [lo, hi], bin nd-1 [lo, hi]
    __shared__ __align__(16) RowRec rows_sm[GMAX][LANES];  // the block of rows each warp walks

    const int4 grp = groups[blockIdx.y];  // the plan: its upload was waited for
    const int cnt = grp.y;
    const bool rows = grp.z == 0;
    const int K = grp.w;  // output bins per strip for this group
    if (blockIdx.x * K >= nd) return;  // the group has fewer strips than the grid (uniform per CTA)
    chain_wait();
    const int b_lo = blockIdx.x * K - 1;       // the strip's lower edge bin
    const int nout = min(K, nd - 1 - b_lo);    // output bins b_lo + 1 .. b_lo + nout
    const bool has0 = b_lo < 0, has_last = b_lo + nout == nd - 1;
    const int lane = threadIdx.x, ja = threadIdx.y;
    const int tid = ja * LANES + lane;

    const int np = rows ? h : w;  // walked axis
    const int nq = rows ? w : h;  // gathered axis
    const double cq = rows ? 0.5 * (w - 1) : 0.5 * (h - 1);
    const double cp = rows ? 0.5 * (h - 1) : 0.5 * (w - 1);
    const double dcf = static_cast<double>(nd / 2);
    constexpr double kReach = 2.0;  // margin of the row ranges (columns)

    // p range (within rows [rl, rh]) where crossings [qa, qb] (at p = 0) come
    // within reach of columns [cl, ch]; idq = 1 / dq (the margins of one row
    // and kReach columns absorb its rounding)
    auto prange = [&](double qa, double qb, double dq, double idq, int cl, int ch, int rl, int rh, int& lo,
                      int& hi) {
        lo = rl;
        hi = rh;
        if (dq != 0.0) {
            const double pa0 = (cl - kReach - qa) * idq, pb0 = (ch + kReach - qa) * idq;
            const double pa1 = (cl - kReach - qb) * idq, pb1 = (ch + kReach - qb) * idq;
            // clamped to [rl, rh + 1] and [rl - 1, rh] before the conversion: at an
            // angle one float step off an axis (90 degrees of 670 uniform ones) idq
            // is 7.5e6, and the rows of columns 286 away do not fit an int
            lo = static_cast<int>(fmin(fmax(floor(fmin(fmin(pa0, pb0), fmin(pa1, pb1))) - 1.0, rl), rh + 1.0));
            hi = static_cast<int>(fmax(fmin(ceil(fmax(fmax(pa0, pb0), fmax(pa1, pb1))) + 1.0, rh), rl - 1.0));
        } else if (fmax(qa, qb) < cl - kReach || fmin(qa, qb) > ch + kReach) {
            hi = -1;
        }
    };

    if (tid < cnt) {
        // the non-zero box of the CTA's slices (all its 4-slice groups), as
        // walked rows [rl, rh] and gathered columns [cl, ch]
        const int ng4 = (nz + 3) / 4;
        // without bounds: the whole image and a disc through its corners
        int4 bx = box ? box[2 * blockIdx.z * NP] : make_int4(0, w - 1, 0, h - 1);
        int r4 = box ? box[2 * blockIdx.z * NP + 1].x : (w - 1) * (w - 1) + (h - 1) * (h - 1);
        for (int k = 1; k < NP && box; ++k) {
            if (blockIdx.z * NP + k >= ng4) break;
            const int4 b2 = box[2 * (blockIdx.z * NP + k)];
            bx = make_int4(min(bx.x, b2.x), max(bx.y, b2.y), min(bx.z, b2.z), max(bx.w, b2.w));
            r4 = max(r4, box[2 * (blockIdx.z * NP + k) + 1].x);
        }
        const int rl = rows ? bx.z : bx.x, rh = rows ? bx.w : bx.y;
        const int cl = rows ? bx.x : bx.z, ch = rows ? bx.y : bx.w;
        const FwdAngleRec R = arec[grp.x + tid];
        const int a = R.a;
        const double kq = R.kq;
        const double kp = R.kp;
        // s(q, p) = (q - cq) kq + (p - cp) kp + dcf = b  <=>  q = q0(b) + p dq
        FAngle f;
        f.inv = R.inv;
        f.dq = -kp * f.inv;
        f.q0 = cq + (static_cast<double>(b_lo) - dcf + cp * kp) * f.inv;
        f.akq = static_cast<float>(fabs(kq));
        f.neg = kq < 0.0 ? 1 : 0;
        f.cf = R.cf;
        f.sf = R.sf;
        f.a = a;
        f.c_lo = cl;
        f.c_hi = ch;
        f.p_lo = 0;
        f.p_hi = -1;
        int e0 = 0, e1 = -1, e2 = 0, e3 = -1;
        if (ch >= cl) {  // an empty box (all slices zero) leaves no rows
            // the strip's pixels have s in (b_lo, b_lo + K + 1)
            const double idq = R.idq;
            prange(f.q0, f.q0 + (K + 1) * f.inv, f.dq, idq, cl, ch, rl, rh, f.p_lo, f.p_hi);
            // Rows where the strip meets the disc: in the frame
            // u' = (q - cq) kq + (p - cp) kp, v = (p - cp) kq - (q - cq) kp the
            // strip is u' in [U0, U1], the disc u'^2 + v^2 <= rad^2, and p - cp
            // = u' kp + v kq. The rectangle u' in [max(U0, -rad), min(U1, rad)],
            // |v| <= sqrt(rad^2 - m^2) (m the smallest |u'| there) holds their
            // intersection.
            // (single-precision roots: their error, ~1e-4 pixels, is far inside
            // the margins of 1.5 pixels and 2 rows)
            const double rad = 0.5 * sqrtf(static_cast<float>(r4)) + 1.5;
            const double u0 = static_cast<double>(b_lo) - dcf, u1 = u0 + K + 1;
            const double a0 = fmax(fmin(u0, u1), -rad), a1 = fmin(fmax(u0, u1), rad);
            if (a0 > a1) {
                f.p_hi = -1;
            } else {
                const double m = (a0 <= 0.0 && a1 >= 0.0) ? 0.0 : fmin(fabs(a0), fabs(a1));
                const double vm = sqrtf(static_cast<float>(fmax(0.0, rad * rad - m * m)));
                const double e0d = a0 * kp, e1d = a1 * kp, ev = vm * fabs(kq);
                const int dlo = static_cast<int>(floor(cp + fmin(e0d, e1d) - ev)) - 2;
                const int dhi = static_cast<int>(ceil(cp + fmax(e0d, e1d) + ev)) + 2;
                f.p_lo = max(f.p_lo, dlo);
                f.p_hi = min(f.p_hi, dhi);
            }
            // rows of the edge passes: s within [-1, 2] of bin 0, [nd-3, nd+1] of bin nd-1
            if (has0)
                prange(f.q0 + (-1 - b_lo) * f.inv, f.q0 + (2 - b_lo) * f.inv, f.dq, idq, cl, ch, rl, rh, e0, e1);
            if (has_last)
                prange(f.q0 + (nd - 3 - b_lo) * f.inv, f.q0 + (nd + 1 - b_lo) * f.inv, f.dq, idq, cl, ch, rl, rh, e2,
                       e3);
        }
        fa[tid] = f;
        erow[tid][0] = e0;
        erow[tid][1] = e1;
        erow[tid][2] = e2;
        erow[tid][3] = e3;
    }
    __syncthreads();
    const bool has_a = ja < cnt;
    const int ng4 = (nz + 3) / 4;    // float4 planes
    const int g0 = blockIdx.z * NP;  // first plane of the CTA
    bool any = false;
    for (int k = 0; k < cnt; ++k) any = any || fa[k].p_hi >= fa[k].p_lo;
    if (!any) {  // the strip meets no non-zero pixel at any angle of the group
        if (has_a && lane < nout)
            for (int z = 4 * g0; z < min(nz, 4 * (g0 + NP)); ++z)
                sino[(static_cast<long long>(z) * na + fa[ja].a) * nd + b_lo + 1 + lane] = 0.0f;
        return;
    }

    const int pitch = nq + 2 * kFwdGuard;
    // the CTA's plane pair: (np + PCH) rows of pitch pixels of 8 slices (two
    // float4). Pairs are allocated whole: a half past the last slice is read
    // but its sums are not stored
    const long long pstride = 2LL * (np + PCH) * pitch;
    const float4* plane = (rows ? img : imgT) + blockIdx.z * pstride + 2 * kFwdGuard;
    // 8-row bands of the walked axis: row bands (x ranges) of the group when
    // walking rows, its column bands (y ranges) when walking columns
    const int nby = (h + 7) / 8, nbx = (w + 7) / 8;
    const int nb_all = nby + nbx, nb_off = rows ? 0 : nby, nb_p = rows ? nby : nbx;

    float2 acc[3][ONE ? 1 : 2 * NP];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int j = 0; j < (ONE ? 1 : 2 * NP); ++j) acc[r][j] = make_float2(0.0f, 0.0f);
    const float* plane1 = reinterpret_cast<const float*>(rows ? img : imgT) + kFwdGuard;  // of a single slice
    if (has_a) {
        const FAngle& f = fa[ja];
        const float akq = f.akq;
        const int ml = lane_bin(lane, akq);
        const float cl1 = fmaf(static_cast<float>(lane), akq, -static_cast<float>(ml + 1));
        RowRec* rr = rows_sm[ja];
        // blocks start on multiples of 32 rows, so that warps whose row ranges
        // overlap walk the same rows at about the same time
        for (int p0 = f.p_lo & ~(LANES - 1); p0 <= f.p_hi; p0 += LANES) {
            // lane r prepares row p0 + r: its crossing in double, and whether
            // the 32 columns from there meet the row's non-zero columns (the
            // range of its 8-row band over the CTA's slice groups, none past the
            // image; or the box without bands)
            const int p = p0 + lane;
            const double q = fma(static_cast<double>(p), f.dq, f.q0);
            const double qr = rint(q);
            const int col = static_cast<int>(qr);
            const float d = static_cast<float>(qr - q);
            int cl = f.c_lo, ch = f.c_hi;
            if (band) {
                cl = INT_MAX;
                ch = -1;
                const int bi = p >> 3;
                for (int k = 0; k < NP && bi < nb_p; ++k) {
                    if (g0 + k >= ng4) break;
                    const int2 r = ld_chained(band + static_cast<long long>(g0 + k) * nb_all + nb_off + bi);
                    cl = min(cl, r.x);
                    ch = max(ch, r.y);
                }
            }
            const int first = f.neg ? col - (LANES - 1) : col;
            const unsigned need = __ballot_sync(
                0xffffffffu, p >= f.p_lo && p <= f.p_hi && ch >= cl && first + LANES - 1 >= cl && first <= ch);
            if (!need) continue;
            __syncwarp();  // the last block's rows are read
            rr[lane] = RowRec{(f.neg ? -d : d) * akq, static_cast<unsigned>(lane * pitch + col + kFwdGuard)};
            __syncwarp();
            const float4* lane_base =
                plane + 2 * (static_cast<long long>(p0) * pitch - kFwdGuard + (f.neg ? -lane : lane));
            // groups of 8 rows without a needed one add only zeros
#pragma unroll 1
            for (int g = 0; g < LANES; g += 8) {
                if (!((need >> g) & 0xffu)) continue;
                if constexpr (ONE) {
                    float2 a[3] = {acc[0][0], acc[1][0], acc[2][0]};
                    walk_rows(plane1 + (static_cast<long long>(p0) * pitch - kFwdGuard + (f.neg ? -lane : lane)), rr + g,
                              cl1, a);
#pragma unroll
                    for (int r = 0; r < 3; ++r) acc[r][0] = a[r];
                } else {
                    walk_rows(lane_base, rr + g, cl1, acc);
                }
            }
        }
    }
    if (!has_a) return;
    const FAngle& f = fa[ja];
    const long long zst = static_cast<long long>(na) * nd;  // slice stride of the sinograms
    const long long ob = static_cast<long long>(f.a) * nd;
    // Output bin t = lane + 1 of the strip is the sum, in lane order, of
    // accumulator t - m_l of every lane l with m_l in [t - 2, t]. Lanes with
    // equal m_l form runs of one or two (m_l + 2 - m_l >= 2|kq| > 1) and the
    // runs' values are -1, 0, 1, ... in lane order (consecutive m differ by at
    // most |kq| <= 1, and m_0 = -1), so run m starts at the (m + 1)-th set bit
    // (counting from 0) of `firsts`. The terms come by warp shuffles.
    constexpr unsigned kAll = 0xffffffffu;
    const int ml = lane_bin(lane, f.akq);
    const int mprev = __shfl_up_sync(kAll, ml, 1);
    const unsigned firsts = __ballot_sync(kAll, lane == 0 || mprev != ml);
    const int t = lane + 1;
    constexpr int NS = ONE ? 1 : 2 * NP;
    if constexpr (ONE)  // the even and the odd rows
        for (int r = 0; r < 3; ++r) acc[r][0] = make_float2(acc[r][0].x + acc[r][0].y, 0.0f);
    float2 sum[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) sum[j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int r = 2; r >= 0; --r) {
        const unsigned l0 = __fns(firsts, 0, t - r + 2);  // first lane of run t - r (or ~0u: none)
        const bool ok0 = l0 < LANES;
        const bool ok1 = ok0 && l0 + 1 < LANES && !((firsts >> (l0 + 1)) & 1u);
        const int s0 = ok0 ? static_cast<int>(l0) : lane, s1 = ok1 ? static_cast<int>(l0) + 1 : lane;
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            const float2 a0 = make_float2(__shfl_sync(kAll, acc[r][j].x, s0),
                                          ONE ? 0.0f : __shfl_sync(kAll, acc[r][j].y, s0));
            const float2 a1 = make_float2(__shfl_sync(kAll, acc[r][j].x, s1),
                                          ONE ? 0.0f : __shfl_sync(kAll, acc[r][j].y, s1));
            if (ok0) sum[j] = __fadd2_rn(sum[j], a0);
            if (ok1) sum[j] = __fadd2_rn(sum[j], a1);
        }
    }
    const int b = b_lo + t;
    if (lane < nout && b != 0 && b != nd - 1) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            const int z = 4 * g0 + 2 * j;  // slices z, z + 1 of pair j
            if (z < nz) sino[z * zst + ob + b] = sum[j].x;
            if (!ONE && z + 1 < nz) sino[(z + 1) * zst + ob + b] = sum[j].y;
        }
    }
    // bins 0 and nd-1 on the reference's own rules
    const float cxf = static_cast<float>(w - 1) * 0.5f, cyf = static_cast<float>(h - 1) * 0.5f;
    for (int side = 0; side < 2; ++side) {
        if (!(side == 0 ? has0 : has_last)) continue;
        const int eb = side == 0 ? 0 : nd - 1;
        if constexpr (ONE) {
            const float v = edge_bin(plane1, pitch, nq, f, b_lo, eb, nd, erow[ja][2 * side], erow[ja][2 * side + 1], rows,
                                     cxf, cyf, lane);
            if (lane == 0) sino[ob + eb] = v;
            continue;
        }
        float2 sum[2 * NP];
        edge_bin(plane, pitch, nq, f, b_lo, eb, nd, erow[ja][2 * side], erow[ja][2 * side + 1], rows, cxf,
                 cyf, lane, sum);
        if (lane == 0) {
#pragma unroll
            for (int j = 0; j < 2 * NP; ++j) {
                const int z = 4 * g0 + 2 * j;
                if (z < nz) sino[z * zst + ob + eb] = sum[j].x;
                if (z + 1 < nz) sino[(z + 1) * zst + ob + eb] = sum[j].y;
            }
        }
    }
}

// One thread per angle group: the per-angle constants of its angles (the
// expressions the projector's set-up evaluated itself before).
__global__ void k_fwd_angles(const int4* __restrict__ groups, int ngroups, const int* __restrict__ order,
                             Trig trig, FwdAngleRec* __restrict__ rec) {
    const int gi = blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= ngroups) return;
    const int4 grp = groups[gi];
    const bool rows = grp.z == 0;
    for (int k = 0; k < grp.y; ++k) {
        const int a = order[grp.x + k];
        const double2 tc = trig.cs[a];
        FwdAngleRec r;
        r.kq = rows ? tc.x : tc.y;
        r.kp = rows ? tc.y : tc.x;
        r.inv = 1.0 / r.kq;
        const double dq = -r.kp * r.inv;
        r.idq = dq != 0.0 ? 1.0 / dq : 0.0;
        const float2 tf = trig.csf[a];
        r.cf = tf.x;
        r.sf = tf.y;
        r.a = a;
        r.pad = 0;
        rec[grp.x + k] = r;
    }
}

}  // namespace

cudaError_t launch_forward(const float4* d_img, const float4* d_imgT, int w, int h, int nz,
                           int na, int nd, const int4* d_groups, int ngroups, int max_strips,
                           const FwdAngleRec* d_rec, const int4* d_box, const int2* d_band, float* d_sino,
                           cudaStream_t st, bool single) {
    const dim3 grid(max_strips, ngroups, ((nz + 3) / 4 + NP - 1) / NP);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool sparse = static_cast<long long>(grid.x) * grid.y * grid.z <= static_cast<long long>(SPARSE) * sms;
    auto kernel = single ? k_forward<FULL, true> : sparse ? k_forward<SPARSE, false> : k_forward<FULL, false>;
    return launch_chained(kernel, grid, dim3(LANES, GMAX), 0, st, d_img, d_imgT, w,
                          h, nz, na, nd, d_groups, d_rec, d_box, d_band, d_sino);
}

cudaError_t launch_fwd_angles(const int4* d_groups, int ngroups, const int* d_order, Trig trig,
                              FwdAngleRec* d_rec, cudaStream_t st) {
    k_fwd_angles<<<(ngroups + 127) / 128, 128, 0, st>>>(d_groups, ngroups, d_order, trig, d_rec);
    return cudaGetLastError();
}

}  // namespace ctb
