// ilu_ring.cuh -- the shared-memory ring of the triangular sweeps that keep a
// level's data in registers ahead (dev_ilu.cu, dev_ilu_rows.cu).
//
// One warp of the thread block copies levels (the slots of all computing
// warps, then their right-hand sides) into a ring of kRingParts parts of B
// levels with cp.async.bulk, an mbarrier per part, waits for each part and
// announces it on a named barrier; the computing warps read their entries
// from it.  The copying warp takes no part in the levels: starting a copy
// takes it about 200 cycles and an mbarrier wait 180 however long ago the copy
// landed (joined to every level barrier it made a level of one warp 730 cycles
// long).  Its waits are bounded.  Once one has given up it starts no further
// copy, hands over the remaining parts as they are, by the same barriers, raises
// the error word that ilu_check reads and leaves once the copies in flight have
// landed.  The computing warps run on, over records of earlier parts or, for the
// first parts, whose places hold none yet, after ring_settle: wrong sums, but
// addresses within the buffers.
//
// Named barriers: 1 levels (the computing warps); 2, 3 a part has landed
// (even, odd parts); 4, 5 a part has been read.  Both sides take part in every
// part's barriers, so that no warp arrives twice in a phase.
#pragma once

namespace xt {

constexpr int kRingParts = 4;
constexpr int kRingSpin = 1 << 20;  // polls of a wait before it gives up

// Shared memory, mbarriers and bulk copies by shared-memory address.
__device__ __forceinline__ unsigned smem_addr(const void* p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ float lds_f(unsigned addr)
{
    float r;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ double lds_d(unsigned addr)
{
    double r;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ unsigned lds_u(unsigned addr)
{
    unsigned r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint2 lds_v2(unsigned addr)
{
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint4 lds_v4(unsigned addr)
{
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "r"(addr));
    return r;
}
__device__ __forceinline__ void bar_init(unsigned bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// The phase of the given parity is complete, within `polls` polls.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, int polls)
{
    for (int i = 0; i < polls; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void ring_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void ring_arrive(int id, int threads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// The level barrier of the computing warps.
__device__ __forceinline__ void ring_level(int threads)
{
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// Part m has landed, within `polls` polls of its mbarrier.
__device__ __forceinline__ bool ring_wait(unsigned bars, int m, int polls)
{
    return bar_wait(bars + 8u * (unsigned)(m % kRingParts), (unsigned)(m / kRingParts) & 1u, polls);
}
// One thread, after the wait for one of the first kRingParts parts has given up:
// parts m .. issued - 1 have landed, or, should one not within the full limit,
// its place is zeroed, for the computing warps take addresses from what they
// read.  A record of zeros reads and writes element 0 of its buffers.
inline __device__ __noinline__ void ring_settle(unsigned at, unsigned bars, unsigned part, int m, int issued)
{
    for (; m < issued; ++m) {
        if (ring_wait(bars, m, kRingSpin)) continue;
        const unsigned to = at + (unsigned)(m % kRingParts) * part;
        for (unsigned o = 0; o < part; o += 16u)
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(to + o), "r"(0) : "memory");
    }
}

struct SweepRing {
    unsigned at;                   // shared-memory address of the ring
    unsigned bars;                 // of the kRingParts mbarriers
    unsigned lev_slots, lev_rhs;   // bytes of a level
    int B, nl, nparts, ncw;
    unsigned part_slots, part;     // bytes of a part's slots, of a part

    __device__ __forceinline__ SweepRing(unsigned at_, unsigned bars_, int B_, int nl_, int ncw_,
                                         unsigned slot_bytes, unsigned rhs_bytes)
        : at(at_), bars(bars_), lev_slots((unsigned)ncw_ * slot_bytes),
          lev_rhs((unsigned)ncw_ * rhs_bytes), B(B_), nl(nl_), nparts((nl_ + B_ - 1) / B_), ncw(ncw_)
    {
        part_slots = (unsigned)B * lev_slots;
        part = part_slots + (unsigned)B * lev_rhs;
    }
    __device__ __forceinline__ int all() const { return (ncw + 1) * 32; }
    __device__ __forceinline__ int computing() const { return ncw * 32; }

    // one thread, before the block's first barrier
    __device__ __forceinline__ void init() const
    {
        for (int k = 0; k < kRingParts; ++k) bar_init(bars + 8u * (unsigned)k);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __device__ __forceinline__ void copy(int m, const unsigned char* slots, const unsigned char* rhs) const
    {
        const unsigned bar = bars + 8u * (unsigned)(m % kRingParts);
        const unsigned to = at + (unsigned)(m % kRingParts) * part;
        const unsigned n = (unsigned)min(B, nl - m * B);
        bar_expect(bar, n * (lev_slots + lev_rhs));
        bulk_copy(to, slots + (size_t)m * part_slots, n * lev_slots, bar);
        bulk_copy(to + part_slots, rhs + (size_t)m * B * lev_rhs, n * lev_rhs, bar);
    }
    // the copying warp's whole work; false in lane 0, which alone copies and
    // waits, when a wait gave up.  The waits for the first parts take at most
    // `polls` polls.  They have a loop of their own: one more test in the loop of
    // the others costs a part 130 cycles, and with four warps a level the copying
    // warp is what the others wait for (12 x 12 x 30 rod 177 -> 187 us an apply).
    __device__ __forceinline__ bool copies(const unsigned char* slots, const unsigned char* rhs, int lane,
                                           int polls) const
    {
        int issued = min(kRingParts, nparts);
        bool ok = true;
        if (lane == 0)
            for (int m = 0; m < issued; ++m) copy(m, slots, rhs);
        auto hand_over = [&](int m) {
            __syncwarp();
            ring_arrive(2 + (m & 1), all());
            // the part before has been read: its place takes the next copy
            if (m > 0) {
                ring_sync(4 + ((m - 1) & 1), all());
                if (lane == 0 && ok && m - 1 + kRingParts < nparts) {
                    copy(m - 1 + kRingParts, slots, rhs);
                    issued = m + kRingParts;
                }
            }
        };
        const int first = issued;
#pragma unroll 1
        for (int m = 0; m < first; ++m) {
            if (lane == 0 && ok) {
                ok = ring_wait(bars, m, polls);
                if (!ok) ring_settle(at, bars, part, m, issued);
            }
            hand_over(m);
        }
#pragma unroll 1
        for (int m = first; m < nparts; ++m) {
            if (lane == 0 && ok) ok = ring_wait(bars, m, kRingSpin);
            hand_over(m);
        }
        if (lane == 0 && !ok)  // leave with no copy in flight
            for (int m = max(0, issued - kRingParts); m < issued; ++m) (void)ring_wait(bars, m, kRingSpin);
        return ok;
    }
};

// A computing warp's way through the ring: where its next entry is.
struct RingReader {
    unsigned s, b;  // addresses of the next entry's slot and right-hand sides
    unsigned s0, b0, ep = 0;
    int ni = 0, left, ready = 2;       // the next entry: level in its part, parts not announced yet
    int ci = 0, after, done = 4;       // the level at hand: in its part, parts behind it

    __device__ __forceinline__ RingReader(const SweepRing& r, unsigned slot_off, unsigned rhs_off)
        : s0(r.at + slot_off), b0(r.at + r.part_slots + rhs_off), left(r.nparts), after(r.nparts - 1)
    {
        s = s0;
        b = b0;
    }
    // before the next entry is read (beyond the last one: old data)
    __device__ __forceinline__ void enter(const SweepRing& r)
    {
        if (ni == 0 && left > 0) {
            ring_sync(ready, r.all());
            ready ^= 1;  // 2, 3, 2, ...
            --left;
        }
    }
    // after it
    __device__ __forceinline__ void next(const SweepRing& r)
    {
        s += r.lev_slots;
        b += r.lev_rhs;
        if (++ni == r.B) {
            ni = 0;
            ep = ep == (kRingParts - 1) * r.part ? 0u : ep + r.part;
            s = s0 + ep;
            b = b0 + ep;
        }
    }
    // after the barrier of a level: its entry is in registers and used
    __device__ __forceinline__ void used(const SweepRing& r)
    {
        if (++ci == r.B) {
            ci = 0;
            if (after > 0) ring_arrive(done, r.all());
            done ^= 1;  // 4, 5, 4, ...
            --after;
        }
    }
};

// Levels of a part, for levels of `warps` warps: handing a part over (its wait,
// two barriers, the next copies) takes the copying warp 700 cycles or more, a
// level about 350 with one or two warps, 400 with three and 500 and more with
// wider ones: four, three and two levels.  Fewer where they do not fit in `room`
// bytes, 0 where one does not.  With three warps a fourth level would leave a
// batch one block an SM.  Measured, two levels (four up to 3 KB a level) before,
// both sweeps of one apply with its copies: plate of 32 x 64 x 2 elements 419
// and 374 us, panel of 96 x 24 x 1 450 and 398, 6 x 6 x 200 rod 792 and 691, 10
// x 10 x 30 rod 246 and 232; with three levels the 16 x 16 x 48 rod, six warps,
// takes 613 in place of 598.
inline int ring_levels(long long level_bytes, int warps, long long room)
{
    const long long n = room / (level_bytes * kRingParts);
    const long long want = warps <= 2 ? 4 : (warps == 3 ? 3 : 2);
    return (int)(n < want ? (n < 0 ? 0 : n) : want);
}

}  // namespace xt
