// backproject.cu — pixel-driven backprojection (the BP stage of
// SerialBackend::reconstructSlice, SerialBackend.cpp:197-252).
//
// For a voxel (x, y) of an n x n slice, with r = floor(n/2), xx = x - r,
// yy = y - r and dc = floor(sq/2), the reference sums over angles the linear
// interpolation of the filtered row at u = xx cos - yy sin + dc, taking a
// contribution only when both taps floor(u) and floor(u)+1 lie in [0, sq), and
// zeroes voxels outside the inscribed circle xx^2 + yy^2 > r^2. The result is
// scaled by pi/(2 na) (folded into the filter output here) and, for volume
// reconstruction, denormalised with the slice's span and minimum (span folded
// into the filter output, minimum added in the epilogue).
//
// Work decomposition: a work item is a TX x TY voxel tile of one or two groups of
// four slices (the float4 lanes of the filtered rows) of one job. Per angle, the
// detector window that the tile can touch (WIN bins) is staged into shared memory
// by the bulk-copy engine (cp.async.bulk), in a ring of stages; the warps take
// turns as the producer and meet only through the stages' mbarriers. The tile
// origin's detector coordinate is evaluated in double precision once per angle
// and split into the window start and a fractional offset, so each thread
// evaluates u in float on small numbers (|u_local| < WIN): the interpolation
// position is ~10x more accurate than the reference's float u of magnitude ~sq.
// Six shapes are compiled: four tile shapes (32x32, the default; 64x32; 32x16;
// 16x16) and the 32x32 tile with half and twice the ring; bp_default_variant
// picks among 32x32, 32x16 and 16x16 from the job's size, the context's autotuner
// times all six per size bucket.
//
// What bounds it and why this split: interpolating each voxel on its own reads
// two 16-byte taps per voxel and angle, and such a kernel ran at 0.92 of the
// shared-memory load bandwidth (18.28 ms at 512^3 x 720). Neighbouring voxels
// share taps along the axis where u changes slowly (coefficient at most
// sqrt(1/2) bins per voxel), so a thread owns columns of four voxels along that
// slow axis and its lanes run along the other (fast) one: a column's taps are 3,
// 4 or 5 consecutive bins (3.6 on average over the angles, against 8), read
// once, and lanes next to each other read bins next to each other, without bank
// conflicts. Each voxel adds three taps with hat weights; which three depends on
// the slow coefficient alone (four patterns, column_taps), and two slice groups
// share the weights. The kernel is then bound by issue: 44 packed FP32x2 FMAs of
// two issue cycles (6.2 ms on their own) and about 43 other instructions per column
// and angle of 8 slices: 10.55 ms at 512^3 x 720, FMA pipe 69 %, shared memory 78 %
// busy (11.03 ms with smaller stages, see Shape). Measured then, against 11.03: with
// two of the taps read only, 10.95 ms; not kept: tap differences with saturating
// weights, which share the first tap's sum within a column (11.72), one slice group
// per item (13.4) or four (11.07), 64 or 128 registers (12.4 and 11.3 against 80).
//
// The slow axis is x for angles with |sin| > |cos| and y for the others, so a
// tile runs through the angles in the order of the table (Trig): first those
// with columns along x, then, after the accumulators changed places through
// shared memory, those with columns along y; within each, the angles whose slow
// coefficient is positive, then (columns walked from the other end) negative,
// and within those one tap pattern after the other. Small tiles split the angles
// of a stage over SPLIT groups of threads, whose sums are added in a fixed order
// at the end, so that a thread always has columns to share taps in and its
// serial chain of angles is short.
//
// Jobs of few angles (bp_default_variant) have a tile function without columns.
//
// One kernel serves both shapes of work: a single job with one CTA per item,
// or a batch of jobs (BpBatch) on a persistent grid that takes items from an
// atomic counter. An item's arithmetic depends only on its job and tile shape,
// so a job's output is bit-identical alone and in any mix of the same shape.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <type_traits>

#include "ctb_internal.h"

namespace ctb {
namespace {

constexpr int THREADS = 256;
constexpr float kRound = 12582912.0f;   // 1.5 * 2^23: x + kRound rounds x to an integer
constexpr int kRoundBits = 0x4B400000;  // bit pattern of kRound

// A tile shape: TX x TY voxels in columns of V, a ring of NST stages of SW windows
// (one per angle and slice group; CA is a nominal count that bp_shape reports, the
// stages do not follow it) and WIN bins per window: with
// a span of sqrt((TX-1)^2 + (TY-1)^2) bins, the taps of every column lie in bins 0
// .. floor(span + 2) + 2 of the window. MINB is the launch-bounds occupancy target
// (registers 65536 / (256 MINB)). A stage costs every warp about 80 instructions
// beside its angles, so few large stages beat many small ones as long as three CTAs
// fit an SM (32x32 tile at 512^2 x 256 x 720: 5.58 ms with 5 stages of 16 windows,
// 5.75 with 6 of 12, 5.51 with 4 of 20, 5.28 with 3 of 26).
constexpr int V = 4;
template <int TX_, int TY_, int CA_, int WIN_, int SW_, int NST_, int MINB_, bool PAIR_>
struct Shape {
    static constexpr int TX = TX_, TY = TY_, CA = CA_, WIN = WIN_, MINB = MINB_;
    static constexpr bool PAIR = PAIR_, FEW = false;
    // Stages, and how many the producer works ahead: it refills the slot of two
    // stages back, so a warp may lag one stage without holding it up (refilling
    // the last stage's slot made every producer wait for the slowest warp: 13.3
    // against 11.4 ms at 512^3 x 720).
    static constexpr int NST = NST_, AHEAD = NST - 2;
    static constexpr int SW = SW_;                                   // windows per stage
    static constexpr int COLS = TX * TY / V;                         // columns of a tile
    static constexpr int SPLIT = COLS >= THREADS ? 1 : THREADS / COLS;  // groups that share a chunk's angles
    static constexpr int GT = THREADS / SPLIT;                       // threads per group
    static constexpr int NC = COLS / GT;                             // columns per thread
    static_assert(NC * GT == COLS && GT * SPLIT == THREADS, "whole columns per thread");
    static_assert(TX % 16 == 0 && TY % 16 == 0 && GT % TX == 0 && GT % TY == 0, "lanes along either axis");
    static_assert(GT % 32 == 0, "a warp is in one group");
    static_assert(SW <= 32 && SW % (2 * SPLIT) == 0, "a lane per staged angle, whole turns of the groups");
    static_assert(WIN <= kBpWindowMax, "window within the filtered-row guard");
    static_assert(SPLIT * V * GT <= SPLIT * TX * TY, "the exchange buffer holds every group's sums");
};
using V0 = Shape<32, 32, 32, 48, 26, 3, 3, true>;  // the general-purpose shape
using V1 = Shape<64, 32, 32, 76, 16, 4, 2, false>;  // wide tiles: less staging per voxel
using V2 = Shape<32, 16, 32, 40, 24, 4, 3, true>;  // half-height tiles: twice the CTAs
using V3 = Shape<16, 16, 32, 28, 24, 4, 3, true>;  // small tiles for small slices
using V4 = Shape<32, 32, 16, 48, 12, 3, 3, true>;  // the general shape with half the ring
using V5 = Shape<32, 32, 64, 48, 32, 4, 2, true>;  // the general shape with twice the ring (half the stages)

// A tile shape of jobs with few angles (few_tile): TX x TY voxels of four slices, VPT
// voxels per thread along x (TX / VPT apart), 32 angles per staged chunk.
template <int TX_, int TY_, int VPT_, int WIN_>
struct Few {
    static constexpr int TX = TX_, TY = TY_, VPT = VPT_, CA = 32, WIN = WIN_, MINB = 4;
    static constexpr bool PAIR = false, FEW = true;
    static constexpr int XS = TX / VPT;
    static_assert(XS * TY == THREADS, "256 threads per CTA");
    static_assert(WIN <= kBpWindowMax, "window within the filtered-row guard");
};
using F0 = Few<32, 32, 4, 52>;
using F2 = Few<32, 16, 2, 40>;
using F3 = Few<16, 16, 1, 28>;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes,
                                          unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// 16 bytes from a 32-bit shared address (volatile: stays between the barriers
// around it).
__device__ __forceinline__ float4 lds128(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float2 lds64(unsigned a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" :
        "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
constexpr unsigned long long kWaitLimitNs = 2000000000ull;
// Bounded wait: gives up once `limit_ns` nanoseconds of the GPU's global timer
// have passed since the first unsuccessful poll (2 s in the kernels; a poll may
// itself suspend for a hardware-defined interval, so the bound is on time, with
// 2^22 polls as a second cap), and reports `code` through the device error word. With
// `stop` it also gives up, reporting nothing, once another wait of the block did.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity,
                                                  unsigned* err,
                                                  unsigned long long limit_ns = kWaitLimitNs,
                                                  unsigned code = 1u, const volatile int* stop = nullptr) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (unsigned it = 0; it < (1u << 22); ++it) {
        __nanosleep(32);  // leave the issue slots to the warps that work
        if (mbar_try_wait(bar, parity)) return true;
        if (stop && *stop) return false;
        if (global_ns() - t0 > limit_ns) break;
    }
    if (err) atomicOr(err, code);
    return false;
}

// Self-test of the timeout path: one CTA initialises an mbarrier that expects
// one arrival which never comes (no copy or thread arrives on it), and every
// thread waits on it through the same bounded wait the kernels use. Each wait
// gives up after `limit_us` microseconds and records kWaitSelftestCode; the
// kernel then returns normally. Nothing is in flight when it exits.
constexpr unsigned kWaitSelftestCode = 1u << 4;
__global__ void k_wait_selftest(unsigned limit_us, unsigned* err) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    mbar_wait_bounded(&bar, 0, err, 1000ull * limit_us, kWaitSelftestCode);
    __syncthreads();
}

// The fields the inner loop reads every angle come first: one 16-byte
// shared-memory broadcast per warp and angle.
struct AngleRec {
    float f0;      // u of the tile corner with the lowest slow term, minus the window start
    float cf, as;  // u per voxel along the fast axis; |u per voxel| along the slow axis
    int edge;      // the window reaches a detector edge: decide taps like the reference
    float rc, rs;  // the reference's float cos/sin (edge decisions only)
    int pad[2];
};

template <class C>
struct BpSmem {
    static constexpr int NST = C::NST;
    float4 win[NST][C::SW][C::WIN];
    float2 ex[C::SPLIT * C::TX * C::TY];     // exchange of accumulators between threads
    AngleRec rec[NST][C::SW + C::SPLIT];     // a record is read ahead of its use
    unsigned long long full[NST], empty[NST];
    int meta[NST];                           // stage: angles | group << 8 | some angle has `edge` set << 16
    unsigned sent[NST];                      // stages whose copies were issued into the slot
    int first[kBpGroups];                    // first stage of each group of the angle order
    int start[kBpGroups + 1];                // first angle of each group; na
    int total;                               // stages of the item
    int dead;                                // a wait gave up
};

// A stage whose copies the self-test leaves out, and its waits' limit.
struct BpLost {
    int stage;
    unsigned long long limit_ns;
};

// One column of V = 4 voxels at one angle. w: shared address of the window bin of the column's
// lowest voxel, f1 its fraction minus 1, as <= sqrt(1/2) (to rounding) the step
// in u. Voxel v lies frac + v as bins above w, in interval m_v or m_v + 1, where
// m_v = floor(v as) depends on the pattern P alone (the range of as):
//   P = 0: as in [0, 1/3):   m = 0 0 0 0, taps 0..2      P = 2: [1/2, 2/3): m = 0 0 1 1, taps 0..3
//   P = 1: as in [1/3, 1/2): m = 0 0 0 1, taps 0..3      P = 3: [2/3, ..]:  m = 0 0 1 2, taps 0..4
// so with y = frac + v as - m_v - 1 in [-1, 1] its value is max(-y, 0) w[m_v] +
// (1 - |y|) w[m_v + 1] + max(y, 0) w[m_v + 2] (two taps for v = 0): 11 packed
// FP32x2 operations per pair of slices and column and 3 to 5 shared loads, where
// a tap pair per voxel takes 8 of each. ZG groups of four slices share the
// weights; group p's window lies p WIN bins on. With MASK the voxels whose bit of
// `keep` is clear get zero weights; the others' sums do not depend on MASK.
template <int P, int ZG, int WIN, bool MASK>
__device__ __forceinline__ void column_taps(unsigned w, float f1, float as, unsigned keep,
                                            float2 (&acc)[V][2 * ZG]) {
    constexpr int T = P == 0 ? 3 : P == 3 ? 5 : 4;
    constexpr int m0[V] = {0, 0, P >= 2 ? 1 : 0, P == 0 ? 0 : P == 3 ? 2 : 1};
    float c[V][3];
    c[0][0] = -f1;
    c[0][1] = 1.0f + f1;
    c[0][2] = 0.0f;
#pragma unroll
    for (int v = 1; v < V; ++v) {
        const float y = fmaf(static_cast<float>(v), as, f1 - static_cast<float>(m0[v]));
        c[v][0] = fmaxf(-y, 0.0f);
        c[v][1] = 1.0f - fabsf(y);
        c[v][2] = fmaxf(y, 0.0f);
    }
    if constexpr (MASK) {
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int i = 0; i < 3; ++i) c[v][i] = keep & (1u << v) ? c[v][i] : 0.0f;
    }
#pragma unroll
    for (int m = 0; m < T; ++m) {
        float2 q[2 * ZG];
#pragma unroll
        for (int p = 0; p < ZG; ++p) {
            const float4 r = lds128(w + static_cast<unsigned>((p * WIN + m) * sizeof(float4)));
            q[2 * p] = make_float2(r.x, r.y);
            q[2 * p + 1] = make_float2(r.z, r.w);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            if (m < m0[v] || m > m0[v] + (v == 0 ? 1 : 2)) continue;
            const float2 W = make_float2(c[v][m - m0[v]], c[v][m - m0[v]]);
#pragma unroll
            for (int h = 0; h < 2 * ZG; ++h) acc[v][h] = __ffma2_rn(W, q[h], acc[v][h]);
        }
    }
}

// Backproject one tile (x0, y0) of ZG slice groups from zg on of job J. `stages`
// counts the stages this CTA has consumed so far (mbarrier phases continue
// across items). Returns false when a bounded wait gave up (block-uniform): from
// then on no warp issues a copy, waits or reads a window, but all go through the
// stages' barriers of the block, whose place follows from the angle order alone, and
// the copies under way are waited for before the return.
template <class C, int ZG, bool LOST = false>
__device__ __forceinline__ bool bp_tile(BpSmem<C>& S, const BpJob& J, int zg, int x0, int y0, unsigned& stages,
                                        unsigned* err, BpLost lost = {}) {
    constexpr int TX = C::TX, TY = C::TY, WIN = C::WIN, NC = C::NC;
    constexpr int SA = C::SW / ZG;           // angles per stage
    constexpr int NST = C::NST, AHEAD = C::AHEAD;
    constexpr int NS = 4 * ZG, NH = 2 * ZG;  // slices, pairs of slices
    const int t = threadIdx.x;
    const int n = J.n, nz = J.nz, na = J.na, sq = J.sq;
    const double ctr = J.ctr;  // voxel-grid centre (the mask radius too)
    const float radf = static_cast<float>(ctr);

    auto offset = [&](int z) {  // the slice's minimum (0 in normalised units)
        if (!J.stats || J.denorm == CTB_DENORM_NONE || z >= nz) return 0.0f;
        const float4 st = J.stats[z];
        // CUDABackend.cu:676-681 adds the minimum only when max > min
        return (J.denorm == CTB_DENORM_CUDA && !(st.y - st.x > 0.0f)) ? 0.0f : st.x;
    };

    // Tiles entirely outside the reconstruction circle hold only the offset.
    {
        const int xe = min(x0 + TX - 1, n - 1), ye = min(y0 + TY - 1, n - 1);
        const double dx = fmax(0.0, fmax(x0 - ctr, ctr - xe));
        const double dy = fmax(0.0, fmax(y0 - ctr, ctr - ye));
        if (dx * dx + dy * dy > ctr * ctr) {
            for (int z = 4 * zg; z < min(nz, 4 * zg + NS); ++z) {
                const float o = offset(z);
                for (int i = t; i < TX * TY; i += THREADS) {
                    const int x = x0 + i % TX, y = y0 + i / TX;
                    if (x < n && y < n) J.out[(static_cast<long long>(z) * n + y) * n + x] = o;
                }
            }
            return true;
        }
    }

    // A stage is up to SA angles of one group of the angle order (Trig), so
    // its tap pattern is the same for all. Warp 0 lists the groups' first stages.
    const int warp = t / 32, lane = t & 31;
    if (warp == 0) {
        const int begin = lane > 0 && lane <= kBpGroups ? J.trig.end[lane - 1] : 0;
        const int count = lane < kBpGroups ? J.trig.end[lane] - begin : 0;
        int sum = (count + SA - 1) / SA;
        const int own = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += q;
        }
        if (lane < kBpGroups) {
            S.first[lane] = sum - own;
            S.start[lane] = begin;
        }
        if (lane == 31) {
            S.total = sum;
            S.start[kBpGroups] = na;
        }
    }
    __syncthreads();
    const int total = S.total;
    auto wait = [&](unsigned long long* bar, unsigned parity) {
        const bool ok = mbar_wait_bounded(bar, parity, err, LOST ? lost.limit_ns : kWaitLimitNs, 1u, &S.dead);
        if (!ok) *static_cast<volatile int*>(&S.dead) = 1;
        return ok;
    };

    // One warp fills the item's stage i (the CTA's stage s).
    // Its slot was last used NST stages ago: every warp arrived on `empty` after
    // reading it.
    auto produce = [&](unsigned s, int i) {
        const int slot = s % NST;
        const unsigned use = s / NST;
        bool ok = *static_cast<volatile int*>(&S.dead) == 0;
        if (ok && use > 0) ok = wait(&S.empty[slot], (use - 1) & 1);
        if (!__all_sync(0xffffffffu, ok)) return;  // nothing is copied any more
        // the last group that starts at or before stage i
        const int grp = __popc(__ballot_sync(0xffffffffu, lane < kBpGroups && S.first[lane & (kBpGroups - 1)] <= i)) - 1;
        const int pos = S.start[grp] + (i - S.first[grp]) * SA;
        const int cnt = min(SA, S.start[grp + 1] - pos);
        const bool along = grp < kBpGroups / 2, flip = (grp / 4) & 1;
        int a = 0, ws = 0, edge = 0;
        if (lane < cnt) {
            a = J.trig.order[pos + lane];
            const double2 tc = J.trig.cs[a];
            const float2 tf = J.trig.csf[a];
            const double uo = (x0 - ctr) * tc.x - (y0 - ctr) * tc.y + J.dc;
            const double umin = uo + fmin(0.0, (TX - 1) * tc.x) + fmin(0.0, -(TY - 1) * tc.y);
            const double umax = uo + fmax(0.0, (TX - 1) * tc.x) + fmax(0.0, -(TY - 1) * tc.y);
            ws = static_cast<int>(floor(umin)) - 1;
            // u = uo + x cos - y sin over the tile's voxels (x, y): columns
            // along x or along y, walked from the end where the slow term is
            // lowest
            const double fast = along ? -tc.y : tc.x, slow = along ? tc.x : -tc.y;
            AngleRec r;
            r.f0 = static_cast<float>(uo + (flip ? ((along ? TX : TY) - 1) * slow : 0.0) - ws);
            r.cf = static_cast<float>(fast);
            r.as = static_cast<float>(flip ? -slow : slow);
            // taps near bin 0 or bin sq-1: the reference's float u decides them
            // (the CUDA backend's per-tap bounds need no rule: bins outside
            // [0, sq) are zeros of the guard)
            edge = J.edge_rule && (umin < 2.0 || umax > sq - 3.0);
            r.edge = edge;
            r.rc = tf.x;
            r.rs = tf.y;
            r.pad[0] = r.pad[1] = 0;
            S.rec[slot][lane] = r;
        }
        edge = __any_sync(0xffffffffu, edge);
        const bool send = !LOST || i != lost.stage;
        if (lane == 0) {
            S.meta[slot] = cnt | grp << 8 | (edge ? 1 << 16 : 0);
            if (send) S.sent[slot] = use + 1;
        }
        __syncwarp();
        // the arrival publishes the records; the copies complete the stage
        if (lane == 0) mbar_expect_tx(&S.full[slot], static_cast<unsigned>(cnt * ZG * WIN * sizeof(float4)));
        __syncwarp();
        if (lane < cnt && send) {
            const float4* row = J.filt + (static_cast<long long>(zg) * na + a) * J.pitch + J.guard + ws;
#pragma unroll
            for (int p = 0; p < ZG; ++p)
                bulk_load(&S.win[slot][lane * ZG + p][0], row + static_cast<long long>(p) * na * J.pitch,
                          WIN * sizeof(float4), &S.full[slot]);
        }
    };

    // this thread's columns: group g takes the angles g, g + SPLIT, ... of a
    // stage; column k has fast coordinate `fast` and slow coordinates 4 col(k)
    // .. 4 col(k) + 3 (counted from the other end of the tile when flipped)
    const int g = t / C::GT, tg = t % C::GT;
    float2 acc[NC][V][NH];
#pragma unroll
    for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int h = 0; h < NH; ++h) acc[k][v][h] = make_float2(0.f, 0.f);
    bool along_x = S.start[kBpGroups / 2] > 0, flipped = false;
    int fast = 0, col[NC];
    bool live[NC];  // some voxel of the column inside the circle
    auto inside = [&](int x, int y) {  // SerialBackend.cpp:220-224
        const float xx = static_cast<float>(x) - radf, yy = static_cast<float>(y) - radf;
        return !(xx * xx + yy * yy > radf * radf);
    };
    auto map_columns = [&] {
        const int F = along_x ? TY : TX;
        fast = tg % F;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            col[k] = tg / F + (C::GT / F) * k;
            live[k] = false;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int s = V * col[k] + v;
                live[k] |= along_x ? inside(x0 + s, y0 + fast) : inside(x0 + fast, y0 + s);
            }
        }
    };
    auto flip_columns = [&] {  // the columns' voxels in the other order
        flipped = !flipped;
        const int ncol = (along_x ? TX : TY) / V;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            col[k] = ncol - 1 - col[k];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                float2 q = acc[k][0][h];
                acc[k][0][h] = acc[k][3][h];
                acc[k][3][h] = q;
                q = acc[k][1][h];
                acc[k][1][h] = acc[k][2][h];
                acc[k][2][h] = q;
            }
        }
    };
    // Hand the sums of columns along x to the threads of the columns along y,
    // two slices at a time. Voxel (x, y) of group g sits at y TX + (x ^ y mod
    // 16): distinct banks for 16 lanes in x or in y.
    auto exchange = [&] {
        if (flipped) flip_columns();
        float2* buf = S.ex + g * TX * TY;
        const int yf = fast;
        int xs[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) xs[k] = V * col[k];
        along_x = false;
        map_columns();
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NC; ++k)
#pragma unroll
                for (int v = 0; v < V; ++v) buf[yf * TX + ((xs[k] + v) ^ (yf & 15))] = acc[k][v][h];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NC; ++k)
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int y = V * col[k] + v;
                    acc[k][v][h] = buf[y * TX + (fast ^ (y & 15))];
                }
        }
    };
    map_columns();

    // The warps take turns as the producer and meet only through the stages'
    // barriers.
    if (warp < min(AHEAD, total)) produce(stages + warp, warp);
    bool landed = true;
    for (int i = 0; i < total; ++i, ++stages) {
        const int slot = stages % NST;
        if (warp == i % (THREADS / 32) && i + AHEAD < total) produce(stages + AHEAD, i + AHEAD);
        // A failed wait leaves stale records and windows: the warp takes nothing of
        // them, and the block stops as a whole at the end of the item.
        landed = landed && wait(&S.full[slot], (stages / NST) & 1);
        // cnt | grp << 8 of the stage; without the stage its group alone, so that every
        // warp passes the block's barriers in exchange() at the same stage
        int meta = 0;
        if (landed) {
            meta = S.meta[slot];
        } else {
            for (int q = 1; q < kBpGroups; ++q) meta += S.first[q] <= i ? 1 << 8 : 0;
        }
        const int cnt = meta & 0xff, grp = (meta >> 8) & 0xff;
        if (along_x && grp >= kBpGroups / 2) exchange();
        if (flipped != (((grp / 4) & 1) != 0)) flip_columns();
        const float fi = static_cast<float>(fast);
        float fj[NC];
        bool some = false;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            fj[k] = static_cast<float>(V * col[k]);
            some |= live[k];
        }
        if (some && g < cnt) {
            // 32-bit shared addresses of this group's first record and window;
            // the window's is offset so that adding 16 times the bits of
            // floor(u) + kRound gives the tap's
            unsigned ra = smem_u32(&S.rec[slot][g]);
            unsigned wa = smem_u32(&S.win[slot][g * ZG][0]) - (static_cast<unsigned>(kRoundBits) << 4);
            // Which voxels of column k take part in an angle whose window reaches a
            // detector edge: SerialBackend.cpp:229-239 evaluates u = (xx cos - yy sin)
            // + dc in float without fused multiply-add and keeps the tap pair only
            // when 0 <= floor(u) and floor(u) + 1 < sq. That decision is reproduced
            // here exactly; the interpolation itself uses the accurate u.
            auto in_range = [&](int k, float2 rcs) {
                const float dcf = static_cast<float>(J.dc);
                unsigned keep = 0;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int sl = V * col[k] + v;
                    const int sa = flipped ? (along_x ? TX : TY) - 1 - sl : sl;
                    const float xs = static_cast<float>(x0 + (along_x ? sa : fast)) - radf;
                    const float ys = static_cast<float>(y0 + (along_x ? fast : sa)) - radf;
                    const float us = __fadd_rn(__fsub_rn(__fmul_rn(xs, rcs.x), __fmul_rn(ys, rcs.y)), dcf);
                    const int is = static_cast<int>(floorf(us));
                    if (is >= 0 && is + 1 < sq) keep |= 1u << v;
                }
                return keep;
            };
            // EDGES: some angle of the stage has `edge` set. An angle's sums depend on
            // its own flag only: what else is in its stage must not change a bit.
            auto run = [&](auto pattern, auto edges) {
                constexpr int P = decltype(pattern)::value;
                constexpr bool EDGES = decltype(edges)::value;
                float4 rec = lds128(ra);
                const unsigned end = wa + static_cast<unsigned>((cnt - g + C::SPLIT - 1) / C::SPLIT) * (C::SPLIT * ZG * WIN * 16u);
                while (wa != end) {
                    const float rf0 = rec.x, rcf = rec.y, ras = rec.z;
                    const bool edge = EDGES && __float_as_int(rec.w);
                    const unsigned rest = ra + offsetof(AngleRec, rc);
                    ra += C::SPLIT * sizeof(AngleRec);
                    rec = lds128(ra);  // the next angle's
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        if (NC > 1 && !live[k]) continue;
                        const float u = fmaf(fi, rcf, fmaf(fj[k], ras, rf0));
                        const float tr = __fadd_rd(u, kRound);  // floor(u), no conversion-unit instruction
                        const unsigned keep = edge ? in_range(k, lds64(rest)) : ~0u;
                        column_taps<P, ZG, WIN, EDGES>(wa + (__float_as_uint(tr) << 4), u - (tr - (kRound - 1.0f)),
                                                       ras, keep, acc[k]);
                    }
                    wa += C::SPLIT * ZG * WIN * sizeof(float4);
                }
            };
            auto run_pattern = [&](auto edges) {
                const int pat = grp % 4;
                if (pat == 0) run(std::integral_constant<int, 0>(), edges);
                else if (pat == 1) run(std::integral_constant<int, 1>(), edges);
                else if (pat == 2) run(std::integral_constant<int, 2>(), edges);
                else run(std::integral_constant<int, 3>(), edges);
            };
            if (meta >> 16) run_pattern(std::true_type());
            else run_pattern(std::false_type());
        }
        __syncwarp();
        if ((t & 31) == 0 && landed) mbar_arrive(&S.empty[slot]);
    }
    if (!__syncthreads_and(landed)) {
        if (t < NST && S.sent[t] > 0) mbar_wait_bounded(&S.full[t], (S.sent[t] - 1) & 1, err);
        __syncthreads();
        return false;
    }
    if (along_x) exchange();
    if (flipped) flip_columns();
    if constexpr (C::SPLIT > 1) {
        // add the groups' sums in group order
        static_assert(NC == 1, "one column per thread of a group");
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            __syncthreads();
            if (g > 0)
#pragma unroll
                for (int v = 0; v < V; ++v) S.ex[((g - 1) * V + v) * C::GT + tg] = acc[0][v][h];
            __syncthreads();
            if (g == 0)
#pragma unroll
                for (int s = 0; s < C::SPLIT - 1; ++s)
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[0][v][h] = __fadd2_rn(acc[0][v][h], S.ex[(s * V + v) * C::GT + tg]);
        }
        if (g > 0) return true;
    }
    const int x = x0 + fast;
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const int z = 4 * zg + j;
        if (z >= nz) break;
        const float o = offset(z);
#pragma unroll
        for (int k = 0; k < NC; ++k)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int y = y0 + V * col[k] + v;
                if (x >= n || y >= n) continue;
                const float r = j & 1 ? acc[k][v][j / 2].y : acc[k][v][j / 2].x;
                J.out[(static_cast<long long>(z) * n + y) * n + x] = (inside(x, y) ? r : 0.0f) + o;
            }
    }
    return true;
}

// ------------------------------------------------------------ few angles
// A job of few angles gains nothing from the columns: its 16 groups make as many
// nearly empty stages, each with another of the unrolled tap patterns, and the
// exchange of sums and 3 CTAs per SM stand against writing the output. So each
// voxel interpolates on its own between two taps, in the angles' given order, with
// four CTAs per SM (FBP of 512^2 x 64: 73.7 -> 60.6 us at 8 angles, 103.3 -> 89.3 at 16).
struct FewRec {
    float f0;      // tile-origin u minus window start
    float c, s;
    int edge;      // the window reaches a detector edge: decide taps like the reference
    float rc, rs;  // the reference's float cos/sin (edge decisions only)
    int pad[2];
};
template <class C>
struct FewSmem {
    float4 win[2][C::CA][C::WIN];
    FewRec rec[2][C::CA];
};
template <class C>
using SmemOf = std::conditional_t<C::FEW, FewSmem<C>, BpSmem<C>>;
// The shape of a launch's jobs of few angles: the same tiles, in the windows' space.
template <class C>
struct FewOf {
    static constexpr bool ANY = false;
    using type = F0;
};
template <class F, class C>
struct FewIn {
    static constexpr bool ANY = true;
    using type = F;
    static_assert(F::TX == C::TX && F::TY == C::TY, "one grid of tiles for both");
    static_assert(sizeof(FewSmem<F>) <= sizeof(BpSmem<C>::win), "clear of the barriers");
};
template <> struct FewOf<V0> : FewIn<F0, V0> {};
template <> struct FewOf<V2> : FewIn<F2, V2> {};
template <> struct FewOf<V3> : FewIn<F3, V3> {};

// Backproject one tile (x0, y0) of slice group zg of job J. bar: one per buffer.
// `chunks` counts the chunks this CTA has consumed so far (mbarrier phases continue
// across items).
// Returns false when a bounded wait gave up (block-uniform), the copies under way
// waited for.
template <class C>
__device__ __forceinline__ bool few_tile(FewSmem<C>& S, unsigned long long* bar, const BpJob& J, int zg, int x0, int y0,
                                         unsigned& chunks, unsigned* err) {
    constexpr int TX = C::TX, TY = C::TY, VPT = C::VPT, XS = C::XS, CA = C::CA, WIN = C::WIN;
    const int t = threadIdx.x;
    const int lx = t % XS, ly = t / XS;
    const int n = J.n, nz = J.nz, na = J.na, sq = J.sq;
    const double ctr = J.ctr;  // voxel-grid centre (the mask radius too)
    const float radf = static_cast<float>(ctr);

    float add[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int z = 4 * zg + j;
        float a = 0.0f;
        if (J.stats && J.denorm != CTB_DENORM_NONE && z < nz) {
            const float4 st = J.stats[z];
            // CUDABackend.cu:676-681 adds the minimum only when max > min
            a = (J.denorm == CTB_DENORM_CUDA && !(st.y - st.x > 0.0f)) ? 0.0f : st.x;
        }
        add[j] = a;
    }

    // Tiles entirely outside the reconstruction circle hold only the offset.
    {
        const int xe = min(x0 + TX - 1, n - 1), ye = min(y0 + TY - 1, n - 1);
        const double dx = fmax(0.0, fmax(x0 - ctr, ctr - xe));
        const double dy = fmax(0.0, fmax(y0 - ctr, ctr - ye));
        if (dx * dx + dy * dy > ctr * ctr) {
            const int y = y0 + ly;
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
                const int x = x0 + lx + XS * k;
                if (x >= n || y >= n) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int z = 4 * zg + j;
                    if (z < nz) J.out[(static_cast<long long>(z) * n + y) * n + x] = add[j];
                }
            }
            return true;
        }
    }

    const double dcd = J.dc;
    const float dcf = static_cast<float>(J.dc);
    const double ox = static_cast<double>(x0) - ctr, oy = static_cast<double>(y0) - ctr;
    const float4* plane = J.filt + static_cast<long long>(zg) * na * J.pitch;
    const int nch = (na + CA - 1) / CA;

    auto issue = [&](int c, int b) {
        const int a0 = c * CA;
        const int cnt = min(CA, na - a0);
        if (t < cnt) {
            const int a = a0 + t;
            const double2 tc = J.trig.cs[a];
            const float2 tf = J.trig.csf[a];
            const double uo = ox * tc.x - oy * tc.y + dcd;
            const double umin = uo + fmin(0.0, (TX - 1) * tc.x) + fmin(0.0, -(TY - 1) * tc.y);
            const double umax = uo + fmax(0.0, (TX - 1) * tc.x) + fmax(0.0, -(TY - 1) * tc.y);
            const int ws = static_cast<int>(floor(umin)) - 1;
            FewRec r;
            r.f0 = static_cast<float>(uo - ws);
            r.c = static_cast<float>(tc.x);
            r.s = static_cast<float>(tc.y);
            r.rc = tf.x;
            r.rs = tf.y;
            // taps near bin 0 or bin sq-1: the reference's float u decides them
            // (the CUDA backend's per-tap bounds need no rule: bins outside
            // [0, sq) are zeros of the guard)
            r.edge = (J.edge_rule && (umin < 2.0 || umax > sq - 3.0)) ? 1 : 0;
            r.pad[0] = r.pad[1] = 0;
            S.rec[b][t] = r;
            bulk_load(&S.win[b][t][0], plane + static_cast<long long>(a) * J.pitch + J.guard + ws,
                      WIN * sizeof(float4), &bar[b]);
        }
        if (t == 0) mbar_expect_tx(&bar[b], static_cast<unsigned>(cnt * WIN * sizeof(float4)));
    };

    float4 acc[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float fx = static_cast<float>(lx), fy = static_cast<float>(ly);
    // positions inside the reconstruction circle (SerialBackend.cpp:220-224);
    // the others are written as the offset only, so their taps are never loaded
    unsigned inside_mask = 0;
    {
        const float yy = static_cast<float>(y0 + ly) - radf;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const float xx = static_cast<float>(x0 + lx + XS * k) - radf;
            if (!(xx * xx + yy * yy > radf * radf)) inside_mask |= 1u << k;
        }
    }

    // all buffers are idle between items: chunk g of this CTA uses buffer g & 1
    issue(0, chunks & 1);
    __syncthreads();
    for (int c = 0; c < nch; ++c) {
        const unsigned g = chunks + c;
        const int b = g & 1;
        if (c + 1 < nch) issue(c + 1, (g + 1) & 1);
        // A failed wait leaves stale window data; the block then stops as a
        // whole at the barrier below (the decision is block-uniform).
        const bool landed = mbar_wait_bounded(&bar[b], (g >> 1) & 1, err);
        const int cnt = min(CA, na - c * CA);
        for (int j = 0; j < cnt; ++j) {
            const FewRec r = S.rec[b][j];
            const float4* w = S.win[b][j];
            const float ub = fmaf(fx, r.c, fmaf(-fy, r.s, r.f0));
            const float c8 = static_cast<float>(XS) * r.c;
            if (!r.edge) {
                // i = floor(u) by rounding u - 1/2 with the kRound addition (no
                // conversion-unit instructions); at an exact tie u = i + 1 the taps
                // shift to (i, i+1) with weights (0, 1), the same value
                const float ubh = ub - 0.5f;
#pragma unroll
                for (int k = 0; k < VPT; ++k) {
                    if (!(inside_mask & (1u << k))) continue;
                    const float uh = fmaf(static_cast<float>(k), c8, ubh);
                    const float tr = uh + kRound;
                    const int i = __float_as_int(tr) - kRoundBits;
                    const float d = uh - (tr - kRound);  // frac(u) - 1/2
                    const float w1 = d + 0.5f;
                    const float w0 = 0.5f - d;
                    const float4 lo = w[i], hi = w[i + 1];
                    acc[k].x = fmaf(w1, hi.x, fmaf(w0, lo.x, acc[k].x));
                    acc[k].y = fmaf(w1, hi.y, fmaf(w0, lo.y, acc[k].y));
                    acc[k].z = fmaf(w1, hi.z, fmaf(w0, lo.z, acc[k].z));
                    acc[k].w = fmaf(w1, hi.w, fmaf(w0, lo.w, acc[k].w));
                }
            } else {
                // SerialBackend.cpp:229-239 evaluates u = (xx cos - yy sin) + dc in
                // float without fused multiply-add and keeps the tap pair only when
                // 0 <= floor(u) and floor(u) + 1 < sq; that decision is reproduced
                // here exactly, the interpolation itself uses the accurate u.
#pragma unroll
                for (int k = 0; k < VPT; ++k) {
                    if (!(inside_mask & (1u << k))) continue;
                    const float u = fmaf(static_cast<float>(k), c8, ub);
                    const float fl = floorf(u);
                    const int i = static_cast<int>(fl);
                    const float xs = static_cast<float>(x0 + lx + XS * k) - radf;
                    const float ys = static_cast<float>(y0 + ly) - radf;
                    const float us = __fadd_rn(__fsub_rn(__fmul_rn(xs, r.rc), __fmul_rn(ys, r.rs)), dcf);
                    const int is = static_cast<int>(floorf(us));
                    const bool ok = (is >= 0) && (is + 1 < sq);
                    const float w1 = ok ? u - fl : 0.0f;
                    const float w0 = ok ? 1.0f - (u - fl) : 0.0f;
                    const float4 lo = w[i], hi = w[i + 1];
                    acc[k].x = fmaf(w1, hi.x, fmaf(w0, lo.x, acc[k].x));
                    acc[k].y = fmaf(w1, hi.y, fmaf(w0, lo.y, acc[k].y));
                    acc[k].z = fmaf(w1, hi.z, fmaf(w0, lo.z, acc[k].z));
                    acc[k].w = fmaf(w1, hi.w, fmaf(w0, lo.w, acc[k].w));
                }
            }
        }
        if (!__syncthreads_and(landed)) {
            if (t == 0) {
                mbar_wait_bounded(&bar[b], (g >> 1) & 1, err);
                if (c + 1 < nch) mbar_wait_bounded(&bar[b ^ 1], ((g + 1) >> 1) & 1, err);
            }
            __syncthreads();
            return false;
        }
    }
    chunks += nch;

    const int y = y0 + ly;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int x = x0 + lx + XS * k;
        if (x >= n || y >= n) continue;
        const bool inside = inside_mask & (1u << k);
        const float v[4] = {acc[k].x, acc[k].y, acc[k].z, acc[k].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int z = 4 * zg + j;
            if (z < nz) J.out[(static_cast<long long>(z) * n + y) * n + x] = (inside ? v[j] : 0.0f) + add[j];
        }
    }
    return true;
}

// One item: the tile (x0, y0) of slice groups zg J.zgs ... of job J (a pair, or
// one group where a pair would pass the last slice).
template <class C>
__device__ __forceinline__ bool bp_item(BpSmem<C>& S, const BpJob& J, int zi, int x0, int y0, unsigned& stages,
                                        unsigned* err) {
    const int zg = zi * J.zgs;
    if constexpr (C::PAIR)
        if (J.zgs == 2 && 4 * (zg + 1) < J.nz) return bp_tile<C, 2>(S, J, zg, x0, y0, stages, err);
    return bp_tile<C, 1>(S, J, zg, x0, y0, stages, err);
}

template <class C>
__device__ __forceinline__ void bp_init(BpSmem<C>& S) {
    if (threadIdx.x == 0) {
        for (int b = 0; b < C::NST; ++b) {
            mbar_init(&S.full[b], 1);
            mbar_init(&S.empty[b], THREADS / 32);
            S.sent[b] = 0;
        }
        S.dead = 0;
        mbar_fence_init();
    }
}

// MODE 0: one job, one CTA per item (job 0 indexed statically keeps its fields
// constant-bank operands). MODE 1: many jobs, one CTA per item, the job found
// from blockIdx.x. MODE 2: a persistent grid whose thread 0 draws items from
// *counter.
template <class C, int MODE>
__global__ void __launch_bounds__(THREADS, C::MINB) k_backproject(const __grid_constant__ BpBatch batch,
                                                                  unsigned* __restrict__ counter,
                                                                  unsigned* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_item;
    __shared__ unsigned long long few_bar[2];
    constexpr bool MIX = MODE != 0 && FewOf<C>::ANY;  // jobs of few angles among the others
    if constexpr (C::FEW || MIX) {
        if (threadIdx.x == 0)
            for (int b = 0; b < 2; ++b) mbar_init(&few_bar[b], 1);
    }
    if constexpr (!C::FEW) bp_init(*reinterpret_cast<BpSmem<C>*>(smem_raw));
    else if (threadIdx.x == 0) mbar_fence_init();
    chain_wait();  // lets the next call's first kernel start in this one's tail
    unsigned stages = 0, chunks = 0;
    // item `local` of job J
    auto run = [&](const BpJob& J, int local) {
        const int zi = local / J.tiles, tl = local - zi * J.tiles;
        const int x0 = (tl % J.tiles_x) * C::TX, y0 = (tl / J.tiles_x) * C::TY;
        if constexpr (C::FEW) {
            return few_tile<C>(*reinterpret_cast<FewSmem<C>*>(smem_raw), few_bar, J, zi, x0, y0, chunks, err);
        } else {
            if constexpr (MIX) {
                using F = typename FewOf<C>::type;
                if (J.few)
                    return few_tile<F>(*reinterpret_cast<FewSmem<F>*>(smem_raw), few_bar, J, zi, x0, y0, chunks, err);
            }
            return bp_item(*reinterpret_cast<BpSmem<C>*>(smem_raw), J, zi, x0, y0, stages, err);
        }
    };
    if constexpr (MODE == 0) {
        __syncthreads();
        run(batch.job[0], blockIdx.x);
    } else if constexpr (MODE == 1) {
        __syncthreads();
        const int item = blockIdx.x;
        int j = 0;
        while (j + 1 < batch.njobs && batch.job[j + 1].first <= item) ++j;
        run(batch.job[j], item - static_cast<int>(batch.job[j].first));
    } else {
        for (;;) {
            if (threadIdx.x == 0) s_item = static_cast<int>(atomicAdd(counter, 1u));
            __syncthreads();
            const int item = s_item;  // totals are below 2^31 (checked at launch)
            if (item >= batch.total) break;
            int j = 0;
            while (j + 1 < batch.njobs && batch.job[j + 1].first <= item) ++j;
            if (!run(batch.job[j], item - static_cast<int>(batch.job[j].first))) break;
            // shared state of this item is dead before the next item's staging, also
            // where one kind's copies land in the other's records
            if constexpr (MIX) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
}

// Self-test of a lost copy: one item of two slice groups, one of whose stages is
// never copied. Every warp's wait for it gives up after `limit_us` microseconds or
// as soon as another's did, and the block ends as it does after such a fault.
template <class C>
__global__ void __launch_bounds__(THREADS, C::MINB) k_bp_selftest(const __grid_constant__ BpBatch batch, int stage,
                                                                  unsigned limit_us, unsigned* err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    BpSmem<C>& S = *reinterpret_cast<BpSmem<C>*>(smem_raw);
    bp_init(S);
    __syncthreads();
    unsigned stages = 0;
    bp_tile<C, 2, true>(S, batch.job[0], 0, 0, 0, stages, err, BpLost{stage, 1000ull * limit_us});
}

// Launches with one CTA per item whose items with work need fewer CTAs per SM
// (b.per_sm) than fit: a CTA asks for so much shared memory that no more than those
// fit. Tiles outside the circle end at once, and CTAs are handed out before that is
// known: with 1.9 items of work per SM some SMs got three and others one; now the rest
// go to the SMs that come free. Measured, FBP: 330 -> 235 us at 387^2 x 16 x 580, 200
// -> 143 at 387^2 x 8, 50.4 -> 42.1 at 200^2 x 8 x 314 in 16x16 tiles.
// Where every CTA is resident anyhow (not b.spread) the bound only costs (27.8 -> 31.7
// us at 96^2 x 24 x 150), unless the launch is chained to the kernel before it: then
// its CTAs start in the filter's tail, and the bound keeps them from piling up on the
// SMs that are free first (194 against 162 us for a volume of 128^3 x 180 without it).
// Measured, FBP: 23.4 -> 21.4 us at 64^2 x 64 x 101, 43.8 -> 40.6 at 128^2 x 32 x 201,
// 41.8 -> 39.6 at 200^2 x 8 x 314. Only for a job by itself (b.alone): beside another
// stage's kernels the CTAs that wait take their room (256^3 x 360 in slabs 2437 ->
// 2447 us), and batches gain nothing.
constexpr int kSmemPerSm = 228 * 1024, kSmemPerCta = 1024;  // of an SM; what each CTA takes besides
constexpr size_t smem_for(size_t own, int per_sm) {
    const size_t floor = kSmemPerSm / (per_sm + 1) - kSmemPerCta + 128;  // per_sm + 1 CTAs do not fit
    return own > floor ? own : floor;
}

template <class C>
cudaError_t set_smem() {
    const int bytes = static_cast<int>(smem_for(sizeof(SmemOf<C>), 1));
    cudaError_t e = cudaFuncSetAttribute(k_backproject<C, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_backproject<C, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_backproject<C, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

template <class C, int MODE>
cudaError_t launch_items(const BpBatch& b, unsigned* d_err, cudaStream_t st) {
    const dim3 grid(static_cast<unsigned>(b.total));
    const bool few = b.per_sm >= 1 && b.per_sm < C::MINB;
    const size_t own = sizeof(SmemOf<C>), smem = few && (b.alone || b.spread) ? smem_for(own, b.per_sm) : own;
    unsigned* const no_counter = nullptr;
    if (few && b.alone) return launch_chained(k_backproject<C, MODE>, grid, dim3(THREADS), smem, st, b, no_counter, d_err);
    k_backproject<C, MODE><<<grid, THREADS, smem, st>>>(b, no_counter, d_err);
    return cudaGetLastError();
}

template <class C>
cudaError_t launch_one(const BpBatch& b, unsigned* d_err, cudaStream_t st) {
    cudaError_t e = set_smem<C>();
    if (e != cudaSuccess) return e;
    return launch_items<C, 0>(b, d_err, st);
}

template <class C>
cudaError_t launch_many(const BpBatch& b, bool persistent, unsigned* d_counter, unsigned* d_err, cudaStream_t st) {
    cudaError_t e = set_smem<C>();
    if (e != cudaSuccess) return e;
    if (!persistent) return launch_items<C, 1>(b, d_err, st);
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_backproject<C, 2>, THREADS, sizeof(SmemOf<C>));
    const long long grid = std::min<long long>(b.total, static_cast<long long>(sms) * (per_sm > 0 ? per_sm : 1));
    e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    k_backproject<C, 2><<<static_cast<unsigned>(grid), THREADS, sizeof(SmemOf<C>), st>>>(b, d_counter, d_err);
    return cudaGetLastError();
}

template <class C>
BpShape shape_of() {
    return BpShape{C::TX, C::TY, C::TX * C::TY / THREADS, C::CA, C::WIN};
}

}  // namespace

cudaError_t launch_wait_selftest(unsigned limit_us, unsigned* d_err, cudaStream_t st) {
    k_wait_selftest<<<1, 64, 0, st>>>(limit_us, d_err);
    return cudaGetLastError();
}

cudaError_t launch_bp_selftest(const float4* d_filt, int na, const FiltLayout& fl, int n_out, Trig trig, float* d_out,
                               unsigned limit_us, unsigned* d_err, cudaStream_t st) {
    BpBatch b;
    b.job[0] = make_bp_job(d_filt, 8, na, fl, n_out, trig, nullptr, CTB_DENORM_NONE, d_out, 0, kConvSerial);
    const int smem = static_cast<int>(sizeof(BpSmem<V0>));
    const cudaError_t e = cudaFuncSetAttribute(k_bp_selftest<V0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_bp_selftest<V0><<<1, THREADS, smem, st>>>(b, 3, limit_us, d_err);
    return cudaGetLastError();
}

BpShape bp_shape(int variant) {
    switch (variant) {
    case 1: return shape_of<V1>();
    case 2: return shape_of<V2>();
    case 3: return shape_of<V3>();
    case 4: return shape_of<V4>();
    case 5: return shape_of<V5>();
    case 6: return shape_of<F0>();
    case 7: return shape_of<F2>();
    case 8: return shape_of<F3>();
    default: return shape_of<V0>();
    }
}

namespace {

// Tiles of a shape that meet the reconstruction circle (the others are
// filled without a loop over the angles).
long long active_tiles(int n, const BpShape& sh, double ctr) {
    long long count = 0;
    for (int y0 = 0; y0 < n; y0 += sh.ty) {
        const int ye = std::min(y0 + sh.ty, n) - 1;
        const double dy = std::max(0.0, std::max(y0 - ctr, ctr - ye));
        if (dy > ctr) continue;
        const double half = std::sqrt(ctr * ctr - dy * dy);  // the circle's columns in these rows
        const int lo = std::max(0, static_cast<int>(std::ceil(ctr - half)));
        const int hi = std::min(n - 1, static_cast<int>(std::floor(ctr + half)));
        if (hi >= lo) count += hi / sh.tx - lo / sh.tx + 1;
    }
    return count;
}

// Relative time of a launch with `items` work items on `sms` SMs: the items of
// an SM times an item's cost. Three items fit an SM at once: up to that count
// the fullest SM decides, a lone item taking 1.4 times its share of a full SM
// (its 8 warps do not fill it); beyond it the SMs even out to half an item.
// Costs per item (one or two slice groups) relative to a 32x32 tile of one group,
// from the backprojector's time at 512^2 x 64 x 720 with stages of 16 windows: 32x32
// 1.658 and 1.462 ms, 32x16 1.822 and 1.640, 16x16 2.173 and 2.082. With the present
// stages an FBP takes 1.792 and 1.581, 1.933 and 1.714, 2.281 and 2.063 (0.18 of it
// the filter): 1.73 for a pair, 0.54 and 0.95, 0.33 and 0.58.
double launch_cost(int variant, int zgs, long long items, int sms) {
    const double pair = variant == 2 ? 0.99 : variant == 3 ? 0.63 : 1.76;
    const double one = variant == 2 ? 0.55 : variant == 3 ? 0.33 : 1.0;
    const double per_sm = static_cast<double>(items) / sms;
    const double rounds = per_sm <= 1.0 ? 1.4 : per_sm <= 3.0 ? std::ceil(per_sm) : per_sm + 0.5;
    return (zgs == 2 ? pair : one) * rounds;
}

// Items of a job that run the angle loop, with zgs slice groups per item.
long long active_items(const BpJob& J, int variant, int zgs) {
    return active_tiles(J.n, bp_shape(variant), J.ctr) * (((J.nz + 3) / 4 + zgs - 1) / zgs);
}

}  // namespace

int bp_default_variant(int n_out, int nz, int na, int sms) {
    // Few angles: the kernel without columns (few_tile), up to where the columns are
    // as fast, which for launches that do not fill the SMs is later, a call being mostly
    // one tile's serial chain there. us per FBP, columns / without, at 512^2 x 64: 116.5
    // / 115.9 with 24 angles, 129.8 / 144.0 with 32; 512^2 x 8: 38.7 / 32.1 with 32, 42.7
    // / 42.2 with 48; 512^2 x 4, which has no pairs: 33.9 / 31.8 with 48; 64^2 x 8: 16.9
    // / 14.6 with 64, 17.4 / 17.0 with 80.
    const long long ctas = static_cast<long long>((n_out + 31) / 32) * ((n_out + 31) / 32) * ((nz + 3) / 4);
    if (na <= (ctas <= sms || (ctas <= 4 * sms && nz <= 4) ? 64 : ctas <= 4 * sms ? 40 : 24)) {
        // 32x32 once its CTAs reach the SM count, 32x16 above a quarter of it (64^2 x 16
        // x 101: 16x16 25 us, 32x16 31, 32x32 44)
        return ctas >= sms ? 6 : 4 * ctas >= sms ? 7 : 8;
    }
    // The shape whose launch is estimated fastest for the job alone; a smaller
    // tile has to gain 15 % in the estimate, which leaves its own start-up cost
    // out. Measured on B200, us per FBP, 32x32 / 32x16 / 16x16: 27.8 / 21.7 / 19.7
    // at 64^2 x 16 x 101; 46.2 / 44.1 / 54.3 at 128^2 x 32 x 201; 142.6 / 141.0 /
    // 161.6 at 387^2 x 8 x 580; 1565 / 1714 / 1991 at 512^2 x 64 x 720. The 64x32
    // tile and the other rings are left to the autotuner.
    BpJob J;
    J.n = n_out;
    J.nz = nz;
    J.ctr = static_cast<double>(n_out / 2);
    int best = 0;
    double least = 0.0;
    for (const int v : {0, 2, 3}) {
        const double t = std::min(launch_cost(v, 1, active_items(J, v, 1), sms),
                                  launch_cost(v, 2, active_items(J, v, 2), sms));
        if (v == 0 || t < 0.85 * least) {
            best = v;
            least = t;
        }
    }
    return best;
}

void bp_number_items(BpBatch& b, int variant, int sms) {
    // Pairs of slice groups share every weight (FBP 1.58 against 1.79 ms at 512^2 x
    // 64 x 720) but make half as many items, which costs more than it gives
    // where the items do not fill the SMs (58.8 against 40.4 us at 128^2 x 32
    // x 201). A slice's result does not depend on the choice.
    long long one = 0, two = 0;
    for (int k = 0; k < b.njobs; ++k) {
        one += active_items(b.job[k], variant, 1);
        two += active_items(b.job[k], variant, b.job[k].few ? 1 : 2);
    }
    const bool pair = variant != 1 && launch_cost(variant, 2, two, sms) < launch_cost(variant, 1, one, sms);
    b.total = 0;
    for (int k = 0; k < b.njobs; ++k) {
        BpJob& J = b.job[k];
        J.zgs = pair && !J.few ? 2 : 1;
        J.first = b.total;
        b.total += static_cast<long long>(J.tiles) * (((J.nz + 3) / 4 + J.zgs - 1) / J.zgs);
    }
    const long long active = pair ? two : one, per_sm = (active + sms - 1) / sms;
    b.per_sm = static_cast<int>(std::min(per_sm, 1LL << 20));
    b.spread = b.total > per_sm * sms;
}

FiltLayout filt_layout(int sq, int n_out) {
    // Every position of every tile grid (n rounded up to whole tiles of any
    // shape, at most kBpTileMax) lies within m = max(r, n_pad - 1 - r) of the
    // centre along each axis, so |u - dc| <= m * sqrt(2); windows start one
    // bin below the tile's minimum and span at most kBpWindowMax bins.
    FiltLayout fl;
    fl.sq = sq;
    const int r = n_out / 2;
    const int n_pad = (n_out + kBpTileMax - 1) / kBpTileMax * kBpTileMax;
    const int m = r > n_pad - 1 - r ? r : n_pad - 1 - r;
    const double reach = m * std::sqrt(2.0) + 3.0;
    const double dc = sq / 2;
    const int left = static_cast<int>(std::ceil(reach + 2.0 - dc));
    const int right = static_cast<int>(std::ceil(dc + reach + kBpWindowMax + 2.0 - sq));
    fl.guard = left > 0 ? left : 0;
    fl.pitch = fl.guard + sq + (right > 0 ? right : 0);
    return fl;
}

BpJob make_bp_job(const float4* d_filt, int nz, int na, const FiltLayout& fl, int n_out, Trig trig,
                  const float4* d_stats, int denorm, float* d_out, int variant, int convention) {
    const BpShape sh = bp_shape(variant);
    BpJob J;
    J.filt = d_filt;
    J.out = d_out;
    J.stats = d_stats;
    J.trig = trig;
    J.nz = nz;
    J.na = na;
    J.sq = fl.sq;
    J.guard = fl.guard;
    J.pitch = fl.pitch;
    J.n = n_out;
    J.denorm = denorm;
    if (convention == kConvCuda) {  // CUDABackend.cu:205-224, 672
        J.ctr = 0.5 * (n_out - 1);
        J.dc = 0.5 * (fl.sq - 1);
        J.edge_rule = 0;
    } else {  // SerialBackend.cpp:205-224
        J.ctr = static_cast<double>(n_out / 2);
        J.dc = static_cast<double>(fl.sq / 2);
        J.edge_rule = 1;
    }
    J.tiles_x = (n_out + sh.tx - 1) / sh.tx;
    J.tiles = J.tiles_x * ((n_out + sh.ty - 1) / sh.ty);
    J.first = 0;
    J.zgs = 1;
    J.few = variant >= kBpVariants;
    return J;
}

cudaError_t launch_backproject_batch(const BpBatch& b, int variant, unsigned* d_counter, unsigned* d_err,
                                     cudaStream_t st, bool persistent) {
    if (b.total == 0) return cudaSuccess;
    if (b.total > 0x7fffffffLL) return cudaErrorInvalidValue;
    bool all_few = true;  // four CTAs per SM instead of the columns' three
    for (int k = 0; k < b.njobs; ++k) all_few = all_few && b.job[k].few;
    if (all_few) {
        if (variant == 0) return launch_many<F0>(b, persistent, d_counter, d_err, st);
        if (variant == 2) return launch_many<F2>(b, persistent, d_counter, d_err, st);
        return launch_many<F3>(b, persistent, d_counter, d_err, st);
    }
    switch (variant) {
    case 1: return launch_many<V1>(b, persistent, d_counter, d_err, st);
    case 2: return launch_many<V2>(b, persistent, d_counter, d_err, st);
    case 3: return launch_many<V3>(b, persistent, d_counter, d_err, st);
    case 4: return launch_many<V4>(b, persistent, d_counter, d_err, st);
    case 5: return launch_many<V5>(b, persistent, d_counter, d_err, st);
    default: return launch_many<V0>(b, persistent, d_counter, d_err, st);
    }
}

cudaError_t launch_backproject(const float4* d_filt, int nz, int na, const FiltLayout& fl,
                               int n_out, Trig trig, const float4* d_stats, int denorm,
                               float* d_out, unsigned* d_err, cudaStream_t st, int variant, int convention, bool alone) {
    BpBatch b;
    b.njobs = 1;
    b.job[0] = make_bp_job(d_filt, nz, na, fl, n_out, trig, d_stats, denorm, d_out, variant, convention);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    bp_number_items(b, variant, sms);
    b.alone = alone;
    if (b.total > 0x7fffffffLL) return cudaErrorInvalidValue;
    switch (variant) {
    case 1: return launch_one<V1>(b, d_err, st);
    case 2: return launch_one<V2>(b, d_err, st);
    case 3: return launch_one<V3>(b, d_err, st);
    case 4: return launch_one<V4>(b, d_err, st);
    case 5: return launch_one<V5>(b, d_err, st);
    case 6: return launch_one<F0>(b, d_err, st);
    case 7: return launch_one<F2>(b, d_err, st);
    case 8: return launch_one<F3>(b, d_err, st);
    default: return launch_one<V0>(b, d_err, st);
    }
}

}  // namespace ctb
