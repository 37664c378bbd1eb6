// dev_ilu_rows.cu -- the triangular sweeps of FP64 factors in row records.
//
// As the FP32 node-row sweep of dev_ilu.cu: one thread block per temporal
// block, each on an SM of its own and each the whole level chain, with the
// solution window in shared memory.
//
// What bounds it.  This part takes an FP64 instruction of one warp in 64 cycles
// whatever its live lanes and however independent, and one of any warp of the
// SM every 19 (measured), so a level costs the instructions of one warp times
// the larger of 64 and 19 times the warps.  The sweep it replaced ran all
// temporal blocks in one thread block (12,400 multiply-adds a level on the
// 80,703-row rod, on one SM).
//
// Layout.  Lane = (group of the warp's chunk, row r of the group, share h of
// the row's entries); G rows a group, H shares a row, 32 / (G H) groups a
// warp.  The groups of a level are sorted by their longest row and dealt to
// chunks; chunk c is taken by warp c mod ncw at its own slot of the level
// (a level of more chunks is split in consecutive sub-levels).  H is chosen
// per triangle by those cycles summed over the levels (rows_cost): one lane a
// row when levels are wide (the 40 groups a level of the 20 x 20 x 60 rod:
// four or five warps), two or four when they are narrow (a level's few rows
// then spread over several warps instead of one running whole rows).
//
// A slot holds per lane {row r of the inverted G x G diagonal block, window
// element | steps of the warp << 16 | 1 << 24 when the warp has a chunk,
// destination}, then per four steps four 16-bit window elements and four
// values (negated: the right-hand side is the accumulator's start).  Steps
// beyond the warp's longest row are skipped in pairs (the branch is the same
// for the whole warp); a lane's own padding reads an all-zero window element.
// The slots are filled on the device from the level-ordered rows.
//
// Flow.  One warp copies whole levels ahead into a ring in shared memory
// (cp.async.bulk, an mbarrier per level) and the others read the next level's
// entry into registers between the multiply-adds of the current one.  Waits
// are bounded; what follows one that gives up is as in ilu_ring.cuh.
//
// Measured (one apply through the C ABI with host vectors, GB300), before
// with the row records through the ring in one thread block: 20 x 20 x 60 rod
// (80,703 rows, q = 6), FP64: 10,262 -> 2,250 us, 2,700 cycles a level, five
// warps of 23 FP64 instructions at the SM's rate of 19 to 21 cycles each;
// 10 x 10 x 30 rod: 3,227 -> 787 us; 4 x 4 x 12 rod: 1,337 -> 320 us, 1,500
// cycles a level, 700 of them the 11 FP64 instructions of its one chunk.
// (With the copying warp off the level barrier, as in ilu_ring.cuh: 2,557 us.)
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>

#include "ilu_ring.cuh"
#include "ilu_sched.h"
#include "xt_device.h"

namespace xt {

namespace {

constexpr int kRowWarps = 7;  // computing warps of a sweep, at most (with the copying one: 255 registers a thread)
constexpr unsigned kNone = 0xffffu;

// Steps a lane's registers hold: rows of up to H * steps entries.
__host__ __device__ constexpr int row_steps(int H) { return H == 1 ? 20 : (H == 2 ? 12 : 8); }
// Bytes of a lane's record: G values, two words, to 16 bytes.
template <int G>
__host__ __device__ constexpr int rec_bytes()
{
    return (G * 8 + 8 + 15) / 16 * 16;
}
template <int G, int H>
__host__ __device__ constexpr int row_slot_bytes()
{
    return 32 * (rec_bytes<G>() + row_steps(H) * (2 + 8));
}

}  // namespace

// One triangle's slots.
struct RowTri {
    int nl = 0, ncw = 0, H = 0, zero = 0, win = 0;
    long long lanes = 0;
    DBuf<unsigned char> slots;
    std::vector<int> first, count, row_slot;  // per slot: its groups; per row: its lane
};

struct RowSweep {
    int g = 1;
    RowTri L, U;
    DBuf<int> src;                    // row of each forward lane (-1: none)
    DBuf<unsigned char> rhsL, rhsU;   // [q][lanes] of the value type
};

namespace {

// The cycles of a triangle's levels with H shares a row and at most kRowWarps
// warps: 64 cycles an instruction of one warp, 19 an instruction of any; about
// 350 a level for the rest (window reads, shuffles, barrier).
long long rows_cost(const TriHost& h, const std::vector<int>& longest, int H, bool& fits)
{
    const int g = h.g, per = 32 / (g * H);
    constexpr int one = 64, any = 19, fixed = 350;
    long long cost = 0;
    fits = true;
    for (int l = 0; l < h.nlevels && fits; ++l) {
        const int gb = h.level_ptr[l], ng = h.level_ptr[l + 1] - gb, nch = (ng + per - 1) / per;
        for (int c = 0; c < nch; c += kRowWarps) {  // the first chunk of a sub-level has its longest row
            const int steps = (longest[gb + c * per] + H - 1) / H;
            if (steps > row_steps(H)) fits = false;
            const int n = (steps + 1) / 2 * 2 + (H == 1 ? 0 : (H == 2 ? 1 : 2)) + g;
            cost += (long long)n * std::max(one, any * std::min(nch - c, kRowWarps)) + fixed;
        }
    }
    return cost;
}

// Chunks, slots and warps of one triangle; ord is its level order with each
// level sorted by longest row.
bool rows_plan(const TriHost& h, const std::vector<int>& ord, int H, int warps, RowTri& t)
{
    const int g = h.g, per = 32 / (g * H);
    std::vector<int> nch(h.nlevels);
    for (int l = 0; l < h.nlevels; ++l)
        nch[l] = (h.level_ptr[l + 1] - h.level_ptr[l] + per - 1) / per;
    std::vector<int> sorted(nch);
    std::sort(sorted.begin(), sorted.end());
    // enough warps for nine levels of ten; the wider ones take sub-levels
    const int p90 = sorted[(size_t)(0.9 * (sorted.size() - 1))];
    t.H = H;
    t.ncw = std::max(1, std::min(kRowWarps, warps > 0 ? warps : p90));
    t.nl = 0;
    for (int c : nch) t.nl += (c + t.ncw - 1) / t.ncw;
    const size_t nslot = (size_t)t.nl * t.ncw;
    if ((long long)nslot * 32 >= INT32_MAX) return false;
    t.lanes = (long long)nslot * 32;
    t.first.assign(nslot, 0);
    t.count.assign(nslot, 0);
    t.row_slot.assign((size_t)h.ngroups * g, -1);
    size_t sl = 0;
    for (int l = 0; l < h.nlevels; ++l) {
        const int gb = h.level_ptr[l], ng = h.level_ptr[l + 1] - gb;
        for (int c = 0; c < nch[l]; ++c) {
            t.first[sl + c] = gb + c * per;
            t.count[sl + c] = std::min(per, ng - c * per);
            for (int k = 0; k < t.count[sl + c]; ++k) {
                const int G = h.order[ord[gb + c * per + k]];
                for (int r = 0; r < g; ++r)
                    t.row_slot[(size_t)G * g + r] = (int)((sl + c) * 32 + (k * g + r) * H);
            }
        }
        sl += (size_t)((nch[l] + t.ncw - 1) / t.ncw) * t.ncw;
    }
    t.zero = h.nslots * g;
    t.win = (h.nslots + 1) * g;
    return t.win < (int)kNone;
}

// Level order of a triangle with each level's groups sorted by longest row,
// and the longest row of each entry of that order.
void rows_sort(const TriHost& h, std::vector<int>& ord, std::vector<int>& longest)
{
    const int g = h.g;
    std::vector<int> len(h.ngroups);
    for (int i = 0; i < h.ngroups; ++i) {
        int m = 0;
        for (int r = 0; r < g; ++r)
            m = std::max(m, h.ext_ptr[(size_t)i * g + r + 1] - h.ext_ptr[(size_t)i * g + r]);
        len[i] = m;
    }
    ord.resize(h.ngroups);
    for (int i = 0; i < h.ngroups; ++i) ord[i] = i;
    for (int l = 0; l < h.nlevels; ++l)
        std::stable_sort(ord.begin() + h.level_ptr[l], ord.begin() + h.level_ptr[l + 1],
                         [&](int a, int b) { return len[a] > len[b]; });
    longest.resize(h.ngroups);
    for (int i = 0; i < h.ngroups; ++i) longest[i] = len[ord[i]];
}

struct RowFill {
    const int *first, *count;      // per slot: its groups in ord
    const int* ord;                // sorted level order -> level order
    const int* row0;               // level order -> first row
    const int* ext_ptr;            // per (level-order group, row)
    const int* ext_col;
    const double* ext_v;
    const double* minv;            // level order, g x g
    const int* wslot;              // window slot of group id
    const int* dst;                // forward: the backward lane of each row; else null
    int* src;                      // forward: the row of each lane; else null
    unsigned char* slots;
    int nslots, zero, q;
};

// One warp per slot.
template <int G, int H>
__global__ void k_fill_rows(RowFill f)
{
    constexpr int S = row_steps(H), RB = rec_bytes<G>(), GS = G * H;
    const int lane = threadIdx.x & 31;
    const int sl = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (sl >= f.nslots) return;
    unsigned char* b = f.slots + (size_t)sl * row_slot_bytes<G, H>();
    const int gw = lane / GS, r = (lane % GS) / H, hh = lane % H;
    const bool on = gw < f.count[sl];
    int k0 = 0, n = 0, row = -1, i = 0;
    if (on) {
        i = f.ord[f.first[sl] + gw];
        row = f.row0[i] + r;
        k0 = f.ext_ptr[(size_t)i * G + r];
        n = f.ext_ptr[(size_t)i * G + r + 1] - k0;
    }
    int steps = (n + H - 1) / H;
    for (int off = 16; off > 0; off >>= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, off));
    double* m = reinterpret_cast<double*>(b + lane * RB);
    for (int k = 0; k < G; ++k) m[k] = on ? (double)f.minv[((size_t)i * G + r) * G + k] : 0.0;
    unsigned* w = reinterpret_cast<unsigned*>(b + lane * RB + G * 8);
    const bool own = on && hh == 0;
    w[0] = (own ? (unsigned)(f.wslot[f.row0[i] / G] * G + r) : kNone) | ((unsigned)steps << 16) |
           (f.count[sl] > 0 ? 1u << 24 : 0u);
    w[1] = own ? (unsigned)(f.dst ? f.dst[row] : row * f.q) : 0u;
    if (f.src) f.src[(size_t)sl * 32 + lane] = own ? row : -1;
    unsigned short* off16 = reinterpret_cast<unsigned short*>(b + 32 * RB);
    unsigned char* vals = b + 32 * RB + 32 * S * 2;
    for (int st = 0; st < S; ++st) {
        const int e = st * H + hh;
        unsigned short o = (unsigned short)f.zero;
        double v = 0.0;
        if (e < n) {
            const int c = f.ext_col[k0 + e];
            o = (unsigned short)(f.wslot[c / G] * G + c % G);
            v = (double)-f.ext_v[k0 + e];
        }
        off16[((st >> 2) * 32 + lane) * 4 + (st & 3)] = o;
        // two values of a lane together: a warp's 16-byte loads are consecutive
        reinterpret_cast<double*>(vals)[((size_t)(st >> 1) * 32 + lane) * 2 + (st & 1)] = v;
    }
}

// A slot in registers; loaded in steps between the multiply-adds of the
// level before it.
template <int G, int H>
struct RowRegs {
    static constexpr int S = row_steps(H), RB = rec_bytes<G>(), VQ = 4 * 8 / 16;
    uint4 rec[RB / 16];
    uint2 off[S / 4];
    uint4 val[S / 4 * VQ];
    double b;

    __device__ __forceinline__ void load_rec(unsigned p, unsigned rhs, int lane)
    {
#pragma unroll
        for (int k = 0; k < RB / 16; ++k) rec[k] = lds_v4(p + lane * RB + 16 * k);
        b = lds_d(rhs);
    }
    __device__ __forceinline__ void load_quad(unsigned p, int k, int lane)
    {
        off[k] = lds_v2(p + 32 * RB + k * 256 + lane * 8);
#pragma unroll
        for (int u = 0; u < VQ; ++u)
            val[k * VQ + u] = lds_v4(p + 32 * RB + 32 * S * 2 + (k * VQ + u) * 512 + lane * 16);
    }
    __device__ __forceinline__ unsigned word(int i) const  // word i of the record
    {
        const uint4 r = rec[i >> 2];
        return (i & 3) == 0 ? r.x : ((i & 3) == 1 ? r.y : ((i & 3) == 2 ? r.z : r.w));
    }
    __device__ __forceinline__ double m(int k) const
    {
        return __hiloint2double((int)word(2 * k + 1), (int)word(2 * k));
    }
    __device__ __forceinline__ unsigned wo() const { return word(G * 8 / 4); }
    __device__ __forceinline__ int dst() const { return (int)word(G * 8 / 4 + 1); }
    __device__ __forceinline__ unsigned o(int st) const
    {
        const unsigned w = (st & 2) ? off[st >> 2].y : off[st >> 2].x;
        return (st & 1) ? (w >> 16) : (w & 0xffffu);
    }
    __device__ __forceinline__ double v(int st) const
    {
        const uint4 r = val[st >> 1];
        return (st & 1) ? __hiloint2double((int)r.w, (int)r.z) : __hiloint2double((int)r.y, (int)r.x);
    }
};

struct RowArgs {
    const unsigned char* slots;
    const double* rhs;
    double* out;
    long long rstride, ostride;  // between temporal blocks
    int nl, ncw, zero, win;
    int* err;
    int polls;  // of a wait
};

// Levels in flight: a level takes 1,200 cycles and more, four cover a read
// from DRAM.
constexpr int kRingLevels = 4;
// Ring bytes a warp takes of one level: its slot and its 32 right-hand sides.
template <int G, int H>
__host__ __device__ constexpr int ring_bytes() { return row_slot_bytes<G, H>() + 32 * 8; }
__host__ __device__ constexpr unsigned window_bytes(int win) { return ((unsigned)win * 8u + 127u) / 128u * 128u; }

constexpr int kRowSpin = 1 << 20;  // polls of a wait for the copies in flight after one gave up

// Warps 0 .. ncw - 1 compute; the last warp copies levels into the ring and
// waits for them, one level barrier ahead of the warps that read them: a wait
// on an mbarrier takes 180 cycles even when its copy has long landed, and
// starting a copy 200, which the level chain does not see this way.
template <int G, int H, bool UPPER>
__global__ void __launch_bounds__((kRowWarps + 1) * 32, 1) k_tri_rows(RowArgs a)
{
    extern __shared__ __align__(128) unsigned char row_smem[];
    constexpr int S = row_steps(H), GS = G * H, SB = row_slot_bytes<G, H>();
    constexpr int NR = kRingLevels;
    __shared__ unsigned long long bars[NR];
    double* win = reinterpret_cast<double*>(row_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tb = blockIdx.x;
    const unsigned wbase = smem_addr(win);
    const unsigned ring = wbase + window_bytes(a.win);
    const unsigned lev_slots = (unsigned)a.ncw * SB, lev_rhs = (unsigned)a.ncw * 32 * 8;
    const unsigned lev = lev_slots + lev_rhs;
    if (threadIdx.x < G) win[a.zero + threadIdx.x] = 0.0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < NR; ++k) bar_init(smem_addr(bars + k));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == a.ncw) {  // copies
        const double* gb = a.rhs + (size_t)tb * a.rstride;
        auto copy = [&](int l) {
            const unsigned to = ring + (unsigned)(l % NR) * lev, bar = smem_addr(bars + l % NR);
            bar_expect(bar, lev);
            bulk_copy(to, a.slots + (size_t)l * lev_slots, lev_slots, bar);
            bulk_copy(to + lev_slots, gb + (size_t)l * a.ncw * 32, lev_rhs, bar);
        };
        auto landed = [&](int l, int polls) {
            return bar_wait(smem_addr(bars + l % NR), (unsigned)(l / NR) & 1u, polls);
        };
        bool ok = true;
        int issued = min(NR, a.nl);
        // level l is there, or, once a wait has given up, every level in
        // flight has landed or its place is zeroed (no chunk)
        auto wait = [&](int l) {
            ok = landed(l, a.polls);
            if (ok) return;
            for (int m = l; m < issued; ++m)
                if (!landed(m, kRowSpin))
                    for (unsigned o = 0; o < lev; o += 16u)
                        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(ring + (unsigned)(m % NR) * lev + o), "r"(0) : "memory");
        };
        if (lane == 0) {
            for (int l = 0; l < issued; ++l) copy(l);
            wait(0);
            if (ok && a.nl > 1) wait(1);
        }
        __syncwarp();
        asm volatile("bar.sync 0;" ::: "memory");  // levels 0 and 1 are there
        for (int l = 0; l < a.nl; ++l) {
            // level l's entry was read in the interval before, so its place is
            // free; level 0's is read in interval 0 itself, its place follows
            // one interval later
            if (lane == 0 && ok) {
                for (int m = l == 1 ? NR : l + NR; l > 0 && m <= l + NR && m < a.nl; ++m) {
                    copy(m);
                    issued = m + 1;
                }
                if (l + 2 < a.nl) wait(l + 2);
            }
            __syncwarp();
            asm volatile("bar.sync 0;" ::: "memory");
        }
        if (lane == 0 && !ok) *a.err = 1;
        return;
    }
    const int lane0 = (lane / GS) * GS;
    double* out = UPPER ? a.out + tb : a.out + (size_t)tb * a.ostride;
    const unsigned myslot = ring + (unsigned)warp * SB;
    const unsigned myrhs = ring + lev_slots + (unsigned)(warp * 32 + lane) * 8u;
    RowRegs<G, H> R[2];
    asm volatile("bar.sync 0;" ::: "memory");  // levels 0 and 1 are there
    R[0].load_rec(myslot, myrhs, lane);
#pragma unroll
    for (int k = 0; k < S / 4; ++k) R[0].load_quad(myslot, k, lane);
    unsigned at = NR > 1 ? lev : 0;  // the next level's place
    // one level: its sums with r, while the next level's entry goes into nx
    // (a place beyond the last level holds old data: read, not used)
    auto level = [&](RowRegs<G, H>& r, RowRegs<G, H>& nx) {
        const unsigned wo = r.wo();
        const int steps = (wo >> 24) ? (int)(wo >> 16) & 0xff : -1;  // -1: no chunk; the same for the whole warp
        double x[S];
#pragma unroll
        for (int st = 0; st < (S < 8 ? S : 8); ++st)
            if ((st & ~3) < steps) x[st] = lds_d(wbase + r.o(st) * 8u);
        double acc = r.b;
#pragma unroll
        for (int k = 0; k < S / 4; ++k) {
            if (4 * k < steps) {
                acc = fma(r.v(4 * k), x[4 * k], acc);
                acc = fma(r.v(4 * k + 1), x[4 * k + 1], acc);
            }
            if (k + 2 < S / 4 && 4 * k + 8 < steps)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (4 * k + 8 + u < S)
                        x[4 * k + 8 + u] = lds_d(wbase + r.o(4 * k + 8 + u) * 8u);
            nx.load_quad(myslot + at, k, lane);
            if (4 * k + 2 < steps) {
                acc = fma(r.v(4 * k + 2), x[4 * k + 2], acc);
                acc = fma(r.v(4 * k + 3), x[4 * k + 3], acc);
            }
        }
        nx.load_rec(myslot + at, myrhs + at, lane);
        if (steps >= 0) {
            double d = acc;
#pragma unroll
            for (int m = 1; m < H; m <<= 1) d += __shfl_xor_sync(0xffffffffu, d, m);
            double sol;
            if constexpr (G == 1) {
                sol = r.m(0) * d;
            } else {
                const double d0 = __shfl_sync(0xffffffffu, d, lane0);
                const double d1 = __shfl_sync(0xffffffffu, d, lane0 + H);
                const double d2 = __shfl_sync(0xffffffffu, d, lane0 + 2 * H);
                sol = fma(r.m(2), d2, fma(r.m(1), d1, r.m(0) * d0));
            }
            if ((wo & 0xffffu) != kNone) {
                win[wo & 0xffffu] = sol;
                out[r.dst()] = sol;
            }
        }
        at = at + lev == NR * lev ? 0 : at + lev;
        asm volatile("bar.sync 0;" ::: "memory");
    };
    for (int l = 0; l < a.nl; l += 2) {
        level(R[0], R[1]);
        if (l + 1 < a.nl) level(R[1], R[0]);
    }
}

// Forward right-hand sides in lane order: rhs[q][lane] = sum_j Ainv(q, j)
// v(row(lane), j).  Lanes without a row keep the zero they were built with.
template <int Q>
__global__ void k_rows_rhs(const int* __restrict__ src, long long lanes,
                           const double* __restrict__ dAinv, const double* __restrict__ v,
                           double* __restrict__ rhs)
{
    __shared__ double sA[Q * Q];
    for (int i = threadIdx.x; i < Q * Q; i += blockDim.x) sA[i] = (double)dAinv[i];
    __syncthreads();
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < lanes;
         t += (long long)gridDim.x * blockDim.x) {
        const int row = src[t];
        if (row < 0) continue;
        double vr[Q];
#pragma unroll
        for (int j = 0; j < Q; ++j) vr[j] = v[(size_t)row * Q + j];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            double b = 0.0;
#pragma unroll
            for (int j = 0; j < Q; ++j) b = fma(sA[j * Q + q], vr[j], b);
            rhs[(size_t)q * lanes + t] = b;
        }
    }
}

template <int G, int H>
int fill_tri(const DevTri& d, const TriHost& h, const std::vector<int>& ord, RowTri& t, int q,
             const int* dst, int* src, cudaStream_t s)
{
    DBuf<int> first, count, dord, row0, wslot;
    DBuf<double> minv;
    const size_t nslot = t.first.size();
    XT_TRY(first.upload(t.first.data(), nslot, s));
    XT_TRY(count.upload(t.count.data(), nslot, s));
    XT_TRY(dord.upload(ord.data(), ord.size(), s));
    XT_TRY(wslot.upload(h.slot.data(), h.slot.size(), s));
    XT_TRY(minv.upload(h.minv.data(), h.minv.size(), s));
    XT_TRY(t.slots.alloc(nslot * (size_t)row_slot_bytes<G, H>()));
    RowFill f{first.p, count.p, dord.p, d.group_row0.p, d.ext_ptr.p, d.ext_col.p, d.ext_v64.p,
              minv.p, wslot.p, dst, src, t.slots.p, (int)nslot, t.zero, q};
    k_fill_rows<G, H><<<(unsigned)((nslot + 7) / 8), 256, 0, s>>>(f);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    XT_CUDA(cudaStreamSynchronize(s));  // the staging buffers go out of scope
    return XT_OK;
}

template <int G>
int fill_any(const DevTri& d, const TriHost& h, const std::vector<int>& ord, RowTri& t, int q,
             const int* dst, int* src, cudaStream_t s)
{
    if (t.H == 1) return fill_tri<G, 1>(d, h, ord, t, q, dst, src, s);
    if (t.H == 2) return fill_tri<G, 2>(d, h, ord, t, q, dst, src, s);
    return fill_tri<G, 4>(d, h, ord, t, q, dst, src, s);
}

template <int G>
size_t row_smem_bytes(const RowTri& t)
{
    const size_t e = t.H == 1 ? ring_bytes<G, 1>() : (t.H == 2 ? ring_bytes<G, 2>() : ring_bytes<G, 4>());
    return window_bytes(t.win) + (size_t)t.ncw * kRingLevels * e;
}

template <int G>
int build(const DevIlu& F, int q, RowSweep& R, bool& ok, cudaStream_t s)
{
    ok = false;
    const TriHost* h[2] = {&F.sched->L, &F.sched->U};
    RowTri* t[2] = {&R.L, &R.U};
    std::vector<int> ord[2], longest[2];
    bool fit[2] = {false, false};
    // XTFEM_ILU_ROW_H forces the shares, XTFEM_ILU_WARPS the warps (tests)
    const int force = env_int("XTFEM_ILU_ROW_H", 0), warps = env_int("XTFEM_ILU_WARPS", 0);
    auto plan = [&](int k) {
        rows_sort(*h[k], ord[k], longest[k]);
        int best = 0;
        long long bc = 0;
        for (int H : {1, 2, 4}) {
            bool f = false;
            const long long c = rows_cost(*h[k], longest[k], H, f);
            if (f && (force == 0 || force == H) && (best == 0 || c < bc)) {
                best = H;
                bc = c;
            }
        }
        if (!best) return XT_OK;
        // fewer warps where window and ring would not fit in shared memory
        fit[k] = rows_plan(*h[k], ord[k], best, warps, *t[k]);
        while (fit[k] && row_smem_bytes<G>(*t[k]) + 4096 > (size_t)max_dyn_smem()) {
            if (t[k]->ncw == 1) fit[k] = false;
            else fit[k] = rows_plan(*h[k], ord[k], best, t[k]->ncw - 1, *t[k]);
        }
        return XT_OK;
    };
    XT_TRY(side_by_side([&] { return plan(1); }, [&] { return plan(0); }));
    if (!fit[0] || !fit[1] || (long long)F.n * q >= INT32_MAX) return XT_OK;
    DBuf<int> dst;
    XT_TRY(dst.upload(R.U.row_slot.data(), R.U.row_slot.size(), s));
    XT_TRY(R.src.alloc((size_t)R.L.lanes));
    XT_TRY((fill_any<G>(F.L, *h[0], ord[0], R.L, q, dst.p, R.src.p, s)));
    XT_TRY((fill_any<G>(F.U, *h[1], ord[1], R.U, q, nullptr, nullptr, s)));
    const size_t bl = (size_t)q * R.L.lanes * 8, bu = (size_t)q * R.U.lanes * 8;
    XT_TRY(R.rhsL.alloc(bl));
    XT_TRY(R.rhsU.alloc(bu));
    // lanes that own no row start their sums at zero
    XT_CUDA(cudaMemsetAsync(R.rhsL.p, 0, bl, s));
    XT_CUDA(cudaMemsetAsync(R.rhsU.p, 0, bu, s));
    XT_CUDA(cudaStreamSynchronize(s));
    if (trace_on())
        std::fprintf(stderr, "[xtfem] row sweep: shares %d/%d, warps %d/%d, levels %d/%d\n",
                     R.L.H, R.U.H, R.L.ncw, R.U.ncw, R.L.nl, R.U.nl);
    for (RowTri* x : t) {
        x->first = std::vector<int>();
        x->count = std::vector<int>();
        x->row_slot = std::vector<int>();
    }
    ok = true;
    return XT_OK;
}

template <int G, int H, bool UPPER>
int launch_tri_rows(const RowTri& t, const RowArgs& a, int q, cudaStream_t s)
{
    static std::atomic<bool> attr{false};
    if (!attr.load(std::memory_order_acquire)) {  // idempotent: concurrent first calls are harmless
        XT_CUDA(cudaFuncSetAttribute(k_tri_rows<G, H, UPPER>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem() - 4096));
        attr.store(true, std::memory_order_release);
    }
    k_tri_rows<G, H, UPPER><<<q, (t.ncw + 1) * 32, row_smem_bytes<G>(t), s>>>(a);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

template <int G, bool UPPER>
int launch_shares(const RowTri& t, const RowArgs& a, int q, cudaStream_t s)
{
    if (t.H == 1) return launch_tri_rows<G, 1, UPPER>(t, a, q, s);
    if (t.H == 2) return launch_tri_rows<G, 2, UPPER>(t, a, q, s);
    return launch_tri_rows<G, 4, UPPER>(t, a, q, s);
}

template <int G>
int launch_both(const RowSweep& R, int q, double* z, cudaStream_t s)
{
    int* err = nullptr;
    XT_TRY(ilu_error_word(&err));
    double *rl = reinterpret_cast<double*>(R.rhsL.p), *ru = reinterpret_cast<double*>(R.rhsU.p);
    XT_TRY((launch_shares<G, false>(
        R.L, RowArgs{R.L.slots.p, rl, ru, R.L.lanes, R.U.lanes, R.L.nl, R.L.ncw, R.L.zero, R.L.win, err,
                   ring_polls()}, q, s)));
    return launch_shares<G, true>(
        R.U, RowArgs{R.U.slots.p, ru, z, R.U.lanes, 0, R.U.nl, R.U.ncw, R.U.zero, R.U.win, err, ring_polls()},
        q, s);
}

template <int Q>
void launch_rhs(const RowSweep& R, const double* dAinv, const double* v, cudaStream_t s)
{
    const int nb = (int)std::max(1LL, std::min<long long>((R.L.lanes + 255) / 256, 152LL * 8));
    k_rows_rhs<Q><<<nb, 256, 0, s>>>(R.src.p, R.L.lanes, dAinv, v, reinterpret_cast<double*>(R.rhsL.p));
    note_launches(1);
}

}  // namespace

int get_rows(const DevIlu& F, int q, cudaStream_t s, RowSweep*& out)
{
    out = nullptr;
    if (!F.sched || q < 1 || q > 8) return XT_OK;
    const int g = F.L.g;
    if (g != 1 && g != 3) return XT_OK;
    const int key = (q * 8 + std::max(0, std::min(7, env_int("XTFEM_ILU_ROW_H", 0)))) * 32 +
                    std::max(0, std::min(31, env_int("XTFEM_ILU_WARPS", 0)));
    auto it = F.rows.find(key);
    if (it == F.rows.end()) {
        auto R = std::make_shared<RowSweep>();
        R->g = g;
        bool ok = false;
        if (g == 3) XT_TRY((build<3>(F, q, *R, ok, s)));
        else XT_TRY((build<1>(F, q, *R, ok, s)));
        it = F.rows.emplace(key, ok ? R : nullptr).first;
    }
    out = it->second.get();
    return XT_OK;
}

int run_rows(const RowSweep& R, int q, const double* dAinv, const double* v, double* z, cudaStream_t s)
{
    switch (q) {
    case 1: launch_rhs<1>(R, dAinv, v, s); break;
    case 2: launch_rhs<2>(R, dAinv, v, s); break;
    case 3: launch_rhs<3>(R, dAinv, v, s); break;
    case 4: launch_rhs<4>(R, dAinv, v, s); break;
    case 5: launch_rhs<5>(R, dAinv, v, s); break;
    case 6: launch_rhs<6>(R, dAinv, v, s); break;
    case 7: launch_rhs<7>(R, dAinv, v, s); break;
    default: launch_rhs<8>(R, dAinv, v, s); break;
    }
    return R.g == 3 ? launch_both<3>(R, q, z, s) : launch_both<1>(R, q, z, s);
}

}  // namespace xt
