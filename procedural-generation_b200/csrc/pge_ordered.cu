// pge_ordered.cu -- the exact, droplet-ordered apply of one wave's change lists.
//
// The reference applies every particle's change list serially in particle
// order against the live terrain (bake/globe/erosion/particle.py:821-1042).
// Entry k of droplet p reads the live terrain of its own cell c_k, of the
// next entry's cell c_{k+1} (erosion floor, final-deposit ceiling) and of
// the previous step entry's cell c_{k-1} (step-deposit ceiling), and writes
// c_k.  So the apply of droplet p depends on earlier droplets only through
// the cells in its sliding window {c_{k-1}, c_k, c_{k+1}}.
//
// Here every droplet of a wave applies its own list on its own warp, and
// each cell is handed from droplet to droplet in droplet order:
//   * the entries of the wave are sorted by (cell, droplet, entry) and each
//     entry learns D = the number of distinct earlier droplets that visit
//     its cell, whether it is its droplet's first visit there, and whether
//     it is the last;
//   * a cell's live net change and its hand-off counter share one 16-byte
//     word: a droplet acquires a cell (the counter reads epoch + D; the net
//     change comes with it) one entry before it writes there (the erosion
//     floor and final-deposit ceiling read the next entry's cell), and hands
//     it on with one store of (net change, epoch + D + 1) right after its
//     last write there; the step-deposit ceiling of the following entry uses
//     the live surface snapshotted at that write -- exactly what the serial
//     order reads, since no other droplet runs between two entries of one
//     droplet.  The stockpile test (is the death cell submerged?) reads the
//     death cell as the droplet's own last write there left it, so it is
//     taken at that write and the death cell is handed on like any other;
//   * a droplet's path through the wave is mostly its own entries one after
//     another (on a wave's critical path 9 in 10 steps go from an entry to
//     its droplet's next one, 1 in 10 over a hand-off of ~350 ns), so what
//     one entry costs bounds the wave.  The rank kernel, which has every
//     entry in parallel, therefore writes all that an entry reads -- its
//     cell's terrain, whom to wait for, which neighbours in the list share
//     or read its cell -- into one 32-byte record in list order, and the
//     apply is left with two shared-memory reads, the arithmetic and the
//     hand-off store;
//   * the order-dependent float64 sums that nothing in the wave reads back
//     -- the discharge and momentum tracks and the stockpile -- are summed
//     after the apply, per cell, walking the sorted entries: (droplet,
//     entry) order within a cell is the serial order.  The packed samples of
//     the touched cells are refreshed in the same walk.
// Every read and write of a cell therefore happens in exactly the
// reference's serial order, and the float64 arithmetic is the reference's
// (this file is compiled without FMA contraction).  Waits are bounded: a
// wait that gives up sets an error flag the host reports.
#include <cub/cub.cuh>

#include "pge_internal.cuh"
#include "pge_ordered.cuh"

namespace pge {

namespace {
inline int grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    return (int)(b < 1 ? 1 : (b > 1048576 ? 1048576 : b));
}

constexpr int kSpinLimit = 1 << 24;  // ~ seconds of looks and sleeps: far beyond any real hand-off

// A cell's hand-off word: 16 bytes, two 8-byte halves (acc low 32 bits | count << 32) and (acc high 32 bits | count <<
// 32), where acc is the live net change and count the hand-off counter.  A reader that sees the same count in both
// halves holds one whole word as long as each half is one: PTX promises that of the relaxed loads and stores below
// (64-bit single-copy atomicity).  The copies ahead (`send`) are asynchronous, weak reads, of which it does not say so;
// they read 16 aligned bytes of one 32-byte sector, which this GPU moves as one.  A copy that is old, or torn between
// the halves, fails the test of the counts and is read again with a relaxed load.
__device__ __forceinline__ void hand_pack(double acc, uint32_t count, unsigned long long &w0, unsigned long long &w1)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(acc);
    w0 = ((unsigned long long)count << 32) | (bits & 0xffffffffull);
    w1 = ((unsigned long long)count << 32) | (bits >> 32);
}

__device__ __forceinline__ double hand_acc(unsigned long long w0, unsigned long long w1)
{
    return __longlong_as_double((long long)((w1 << 32) | (w0 & 0xffffffffull)));
}

__device__ __forceinline__ bool hand_ready(unsigned long long w0, unsigned long long w1, uint32_t want)
{
    return (uint32_t)(w0 >> 32) == want && (uint32_t)(w1 >> 32) == want;
}

__device__ __forceinline__ void hand_load(const double2 *p, unsigned long long &w0, unsigned long long &w1)
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "l"(p) : "memory");
}

__device__ __forceinline__ void hand_store(double2 *p, double acc, uint32_t count)
{
    unsigned long long w0, w1;
    hand_pack(acc, count, w0, w1);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" : : "l"(p), "l"(w0), "l"(w1));
}

// a cell this droplet holds and has written before: its own last write (coherent for the same thread)
__device__ __forceinline__ double own_value(const double2 *hand, long long c)
{
    unsigned long long w0, w1;
    hand_load(hand + c, w0, w1);
    return hand_acc(w0, w1);
}

// asynchronous copies into shared memory: the waits count copy groups, so waiting for an old
// entry's data never waits for the copies issued after it
__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// (the copies and the commit carry no memory clobber: a ring slot is only read after the group wait that
// covers its copy, and that wait is the compiler barrier; the compiler may then overlap a copy's issue
// with the arithmetic around it)
__device__ __forceinline__ void cp_ca8(void *d, const void *g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sm_addr(d)), "l"(__cvta_generic_to_global(g)));
}
__device__ __forceinline__ void cp_cg16(void *d, const void *g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm_addr(d)), "l"(__cvta_generic_to_global(g)));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace

// ---------------------------------------------------------------------------
// ranks
// ---------------------------------------------------------------------------
// key = the slot's cell (invalid past a list's end); the slots enter the stable sort in (droplet,
// entry) order, so equal cells keep the serial order
__global__ void ordered_keys_kernel(long long nslots, int cap, const int32_t *cell, const int64_t *count,
                                    SortKey invalid, SortKey *keys, int32_t *vals, uint32_t *tails, unsigned int *ticket)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < nslots; s += (long long)gridDim.x * blockDim.x) {
        const long long q = s / cap, k = s - q * cap;
        if ((s & 31) == 0) tails[s >> 5] = 0;
        keys[s] = k < count[q] ? (SortKey)cell[s] : invalid;
        vals[s] = (int32_t)s;
    }
}

// the entries of a wave's lists compacted in (droplet, entry) order: entry k of droplet q goes to offsets[q] + k
__global__ void ordered_compact_keys_kernel(long long nslots, int cap, const int32_t *cell, const int64_t *count,
                                            const long long *offsets, SortKey *keys, int32_t *vals, uint32_t *tails,
                                            unsigned int *ticket)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < nslots; s += (long long)gridDim.x * blockDim.x) {
        const long long q = s / cap, k = s - q * cap;
        if ((s & 31) == 0) tails[s >> 5] = 0;
        if (k < count[q]) {
            const long long e = offsets[q] + k;
            keys[e] = (SortKey)cell[s];
            vals[e] = (int32_t)s;
        }
    }
}

__global__ void entry_total_kernel(const int64_t *count, const long long *offsets, long long nw, long long *total)
{
    *total = nw > 0 ? offsets[nw - 1] + count[nw - 1] : 0;
}

// whether an entry reads the next one's cell live: an erosion (its floor) and a final deposit (its ceiling) do, a step
// deposit and a lake park do not
__device__ __forceinline__ bool reads_next(double delta, float vol) { return vol != -3.0f && (delta < 0.0 || vol < 0.0f); }

// One warp per 32 consecutive sorted slots.  An entry's rank is the number of droplets that start between its cell's
// first slot and it: counted in the bits of the warp's slots, after those of the slots before them where their first
// cell's run came in from there.  The 128 slots before are counted again; beyond them, warp by warp, what each warp left
// in `tails`: the droplets that start in its last cell's run, from the run's start (TAIL_RUN) or only in its own slots
// (TAIL_OWN).  Nobody waits: where a warp has left nothing yet, its slots are counted again too.
// (Flags, two library scans and a pass over them: 22 us a wave in six launches at N_c = 1024; as here 7.5 in one.
// The run's first warp walking all of it: 12.4, and 68 where runs reach thousands of entries.  Every warp counting back
// over the whole run, which grows with its square: 328 us for 835,000 entries on a few cells, 813 for 1.67 million, the
// scans 35 and 57, as here 49 and 95.)
enum : uint32_t { TAIL_OWN = 1, TAIL_RUN = 2 };
__global__ void __launch_bounds__(256) ordered_rank_kernel(long long nslots, const SortKey *keys, const int32_t *vals, int cap,
                                                           SortKey invalid, const double *delta, const float *vol,
                                                           const int64_t *count, const CellTerr *terr, uint32_t epoch,
                                                           uint32_t *tails, EntryRec *rec)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    // the record of sorted slot i: D distinct earlier droplets at its cell
    auto emit = [&](long long i, SortKey k, uint32_t D) {
        const int32_t s = vals[i], q = s / cap, e = s - q * cap;
        const CellTerr t = terr[k];
        const float v = vol[s];
        const double d = delta[s];
        EntryRec r;
        r.delta = d;
        r.hs = t.hs;
        r.base = t.base;
        r.cell = (int32_t)k;
        // the droplet's visits before and after this one are its neighbours in the sorted order
        const int32_t back = i > 0 && keys[i - 1] == k && vals[i - 1] / cap == q ? s - vals[i - 1] : 0;
        const int32_t fwd = i + 1 < nslots && keys[i + 1] == k && vals[i + 1] / cap == q ? vals[i + 1] - s : 0;
        const bool reads = e + 1 < count[q] && reads_next(d, v);
        uint32_t f = (uint32_t)(back < APPLY_HIST ? back : APPLY_HIST);
        if (fwd == 0) f |= ENTRY_LAST;
        if (back == 0) f |= ENTRY_FIRST;
        if (back != 0 || D == 0) f |= ENTRY_OPEN;
        if (v >= 0.0f) f |= ENTRY_STEP;
        if (t.active && v != -3.0f) f |= d < 0.0 ? ENTRY_ERO : ENTRY_DEP;
        if (reads) f |= ENTRY_READS;
        if (reads && fwd != 1) f |= ENTRY_NEEDS;
        if (fwd == 1) f |= ENTRY_SAME;
        if (e > 0 && (back == 1 || reads_next(delta[s - 1], vol[s - 1]))) f |= ENTRY_HELD;
        if (fwd >= APPLY_HIST) f |= ENTRY_FAR;
        r.flags = f;
        r.turn = epoch + D;
        rec[s] = r;
    };
    // whether slot i starts a droplet's visit to the cell of key k (the slot's own)
    auto visit = [&](long long i, SortKey k) { return i == 0 || keys[i - 1] != k || vals[i - 1] / cap != vals[i] / cap; };
    for (long long base = warp * 32; base < nslots; base += nwarps * 32) {
        const long long i = base + lane;
        const SortKey k = i < nslots ? keys[i] : invalid;
        const unsigned cells = __ballot_sync(full, k != invalid && (i == 0 || keys[i - 1] != k));
        const unsigned starts = __ballot_sync(full, k != invalid && visit(i, k));
        const SortKey k0 = __shfl_sync(full, k, 0);
        if (k0 == invalid) break;  // (the invalid slots come last)
        const long long w0 = base >> 5;  // these slots' place in `tails`
        const bool goes_on = __shfl_sync(full, k, 31) != invalid;
        if (lane == 0 && goes_on) {
            const unsigned own = cells ? starts & (full << (31 - __clz(cells))) : starts;
            *(volatile uint32_t *)(tails + w0) = (uint32_t)__popc(own) << 2 | (cells ? TAIL_RUN : TAIL_OWN);
        }
        uint32_t before = 0;  // droplets that start before this warp's slots at the cell whose run comes in
        if (!(cells & 1u)) {
            long long w = w0;  // counted back to this warp's slots
            auto count_128 = [&]() {
                bool whole = true;
                bool v[4], in[4];
                w -= 4;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const long long j = 32 * (w + q) + lane;
                    in[q] = j >= 0 && keys[j] == k0;
                    v[q] = in[q] && visit(j, k0);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    before += (uint32_t)__popc(__ballot_sync(full, v[q]));
                    whole = __all_sync(full, in[q]) && whole;
                }
                return whole;
            };
            bool whole = count_128();
            while (whole) {
                // the 32 warps before, the nearest first; one whose last slot is of another cell ends the run
                const long long t = w - 1 - lane;
                const bool in = t >= 0 && keys[32 * t + 31] == k0;
                const uint32_t tail = in ? *(volatile uint32_t *)(tails + t) : (uint32_t)TAIL_RUN;
                const unsigned run = __ballot_sync(full, (tail & 3u) == TAIL_RUN), none = __ballot_sync(full, (tail & 3u) == 0);
                const int to_run = run ? __ffs(run) - 1 : 32, to_none = none ? __ffs(none) - 1 : 32;
                const bool ends = to_run < to_none;
                before += __reduce_add_sync(full, lane < to_none && lane <= to_run ? tail >> 2 : 0u);
                if (ends) break;
                w -= to_none;
                if (to_none == 0) whole = count_128();
            }
            if (lane == 0 && goes_on && !cells)
                *(volatile uint32_t *)(tails + w0) = (before + (uint32_t)__popc(starts)) << 2 | TAIL_RUN;
        }
        if (k == invalid) continue;
        const unsigned upto = full >> (31 - lane);
        const unsigned own = cells & upto;  // the cells that start at or before this slot
        const unsigned from = own ? full << (31 - __clz(own)) : full;
        emit(i, k, (own ? 0u : before) + (uint32_t)__popc(starts & upto & from) - 1u);
    }
}

// the ordered apply's read-only terrain record of every cell
__global__ void ordered_terrain_kernel(long long ncell, const double2 *L, const float4 *B, const uint8_t *mask, CellTerr *terr)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        CellTerr t;
        t.hs = L[c].x;
        t.base = B[c].w;
        t.active = !mask || mask[c] == PGE_MASK_ACTIVE ? 1u : 0u;
        terr[c] = t;
    }
}

size_t ordered_temp_bytes(long long nslots, long long max_wave)
{
    size_t a = 0, d = 0, x = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, x, (int64_t *)nullptr, (long long *)nullptr, (int)max_wave);
    cub::DeviceRadixSort::SortPairs(nullptr, a, (SortKey *)nullptr, (SortKey *)nullptr, (int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)nslots);
    cub::DeviceRadixSort::SortPairs(nullptr, d, (uint32_t *)nullptr, (uint32_t *)nullptr, (int32_t *)nullptr, (int32_t *)nullptr,
                                    (int)(max_wave * LAKE_PARKS));
    const size_t m = a > d ? a : d;
    return m > x ? m : x;
}

// ---------------------------------------------------------------------------
// lake parks: each lake's room counted down in droplet order (particle.py:912-933)
// ---------------------------------------------------------------------------
// one item per (droplet, park slot): key = the lake of the park's cell (all ones: no lake, or past the
// droplet's parks); the items enter the stable sort in (droplet, park) order, which is the serial order
__global__ void park_keys_kernel(long long nitems, int cap, const int32_t *cell, const double *delta, const int32_t *park_n,
                                 const int32_t *park_k, const int32_t *lake_id, long long lakes, uint32_t *keys, int32_t *vals,
                                 double *rest)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nitems; i += (long long)gridDim.x * blockDim.x) {
        const long long q = i / LAKE_PARKS;
        const int j = (int)(i - q * LAKE_PARKS);
        uint32_t key = 0xffffffffu;
        double r = 0.0;
        if (j < park_n[q] && park_k[i] >= 0 && park_k[i] < cap) {  // (an entry past the list's room was not recorded)
            const long long s = q * cap + park_k[i];
            const int32_t lk = lake_id[cell[s]];
            if (lk >= 0 && lk < lakes)
                key = (uint32_t)lk;
            else
                r = delta[s];  // no lake to take it: all of it is refused
        }
        keys[i] = key;
        vals[i] = (int32_t)i;
        rest[i] = r;
    }
}

// A warp takes 32 sorted items and the lakes whose first park is among them; a lake takes what it still has room for,
// the rest is refused, and the room is counted down in the serial order.  The warp reads its items together; the lakes
// whose parks all lie within them are walked in shared memory by the lane of their first, all at once.  A lake with parks
// beyond them (at most the last) is walked by the whole warp, 32 parks at a time, their reads in flight together and only
// the room counted down one after another.  Parks on one cell add to its load in their order (no other lake touches the
// cell).
//
// Bound by the reads' latency and the longest lake's parks.  A wave of 2048 droplets, all the parks in lakes of one cell /
// of 37 / of 500 / in one lake, us: a thread walking its lake's, every read behind the one before 5.0 / 16 / 95 / 1460;
// the whole warp for each lake in turn 44 / 15 / 12 / 137; as here 5.3 / 5.9 / 12 / 132.
constexpr int PARK_THREADS = 64, PARK_WARPS = PARK_THREADS / 32;
struct ParkItems {
    double sent[32], taken[32], rest[32];
};
__global__ void __launch_bounds__(PARK_THREADS) park_walk_kernel(long long nitems, int cap, const uint32_t *keys, const int32_t *vals,
                                                                 const int32_t *cell, const double *delta, const int32_t *park_k,
                                                                 double *lake_room, double *lake_load, double *rest)
{
    __shared__ ParkItems items[PARK_WARPS];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    ParkItems &w = items[threadIdx.x >> 5];
    const long long nwarps = (long long)gridDim.x * PARK_WARPS;
    // the item at sorted place t (a park with a lake: its entry index was checked by park_keys_kernel): its load to
    // shared memory
    auto load_item = [&](long long t, int32_t &v, int32_t &c) {
        v = vals[t];
        const long long s = (long long)(v / LAKE_PARKS) * cap + park_k[v];
        c = cell[s];
        w.sent[lane] = delta[s];
    };
    // what the item at this lane was refused, and what its cell takes: the lanes of a cell, all in `mine`, in their order
    auto settle = [&](unsigned mine, int32_t v, int32_t c) {
        rest[v] = w.rest[lane];
        unsigned same = __match_any_sync(mine, c);
        if (lane == __ffs(same) - 1) {
            double load = lake_load[c];
            for (; same; same &= same - 1) {
                const double take = w.taken[__ffs(same) - 1];
                if (take > 0.0) load += take;
            }
            lake_load[c] = load;
        }
    };
    // one item counted down from its lake's room: what the lake takes of it
    auto count_down = [&](double &room, double sent, double &refused) {
        double take = sent;
        refused = 0.0;
        if (take > room) {
            refused = take - room;
            take = room;
        }
        if (take > 0.0) room -= take;
        return take;
    };
    for (long long base = ((long long)blockIdx.x * PARK_WARPS + (threadIdx.x >> 5)) * 32; base < nitems; base += nwarps * 32) {
        const long long i = base + lane;
        const uint32_t key = i < nitems ? keys[i] : 0xffffffffu;
        const bool head = key != 0xffffffffu && (i == 0 || keys[i - 1] != key);
        const unsigned heads = __ballot_sync(full, head), valid = __ballot_sync(full, key != 0xffffffffu);
        if (!heads) continue;
        // the last lake goes on beyond these items (no lake sorts last, so they are then all valid)
        const uint32_t key31 = __shfl_sync(full, key, 31);
        const bool open = valid == full && base + 32 < nitems && keys[base + 32] == key31;
        const int first = __ffs(heads) - 1, last = 31 - __clz(heads), end = open ? last : __popc(valid);
        // ---- the lakes within the items
        const bool in = lane >= first && lane < end;
        const unsigned mine = __ballot_sync(full, in);
        int32_t v = 0, c = 0;
        if (in) load_item(i, v, c);
        __syncwarp();
        if (in && head) {
            const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;
            const int to = later ? lane + __ffs(later) : end;
            double room = lake_room[key];
            for (int k = lane; k < to; k++) w.taken[k] = count_down(room, w.sent[k], w.rest[k]);
            lake_room[key] = room;
        }
        __syncwarp();
        if (in) settle(mine, v, c);
        __syncwarp();
        if (!open) continue;
        // ---- the lake that goes on
        double room = lake_room[key31];
        for (long long t0 = base + last;; t0 += 32) {
            const long long t = t0 + lane;
            const bool at = t < nitems && keys[t] == key31;
            const unsigned theirs = __ballot_sync(full, at);  // a prefix of the lanes (keys are sorted)
            const int n = __popc(theirs);
            if (at) load_item(t, v, c);
            __syncwarp();
            double my_take = 0.0, my_rest = 0.0;
            for (int k = 0; k < n; k++) {
                double refused;
                const double take = count_down(room, w.sent[k], refused);
                if (k == lane) {
                    my_take = take;
                    my_rest = refused;
                }
            }
            w.taken[lane] = my_take;
            w.rest[lane] = my_rest;
            __syncwarp();
            if (at) settle(theirs, v, c);
            __syncwarp();
            if (n < 32) break;
        }
        if (lane == 0) lake_room[key31] = room;
    }
}

cudaError_t park_wave(const ParkWave &pw, cudaStream_t st)
{
    const long long n = pw.nw * LAKE_PARKS;
    park_keys_kernel<<<grid_for(n), 256, 0, st>>>(n, pw.cap, pw.cell, pw.delta, pw.park_n, pw.park_k, pw.lake_id, pw.lakes, pw.keys_in,
                                                  pw.vals_in, pw.rest);
    size_t tb = pw.temp_bytes;
    // the digits a lake's number has; no lake (all ones) sorts last still
    int bits = 1;
    while ((1LL << bits) <= pw.lakes && bits < 32) bits++;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(pw.temp, tb, pw.keys_in, pw.keys_out, pw.vals_in, pw.vals_out, (int)n, 0, bits, st);
    if (e != cudaSuccess) return e;
    park_walk_kernel<<<grid_for(n, PARK_THREADS), PARK_THREADS, 0, st>>>(n, pw.cap, pw.keys_out, pw.vals_out, pw.cell, pw.delta, pw.park_k, pw.lake_room,
                                                  pw.lake_load, pw.rest);
    return cudaPeekAtLastError();
}

// ---------------------------------------------------------------------------
// the ordered apply
// ---------------------------------------------------------------------------
namespace {
constexpr unsigned FULL = 0xffffffffu;
// records of a droplet's list on chip: the chunk being applied, the next two and the one before (a power of two)
constexpr int REC_RING = 128;
// a waiting warp whose turn is n droplets away sleeps n - 1 times BACK_NS (at most BACK_MAX of them; a hand-off takes
// several) between its looks.  A wave whose droplets all cross one cell, us a pass at 2048 / 4096 / 8192 / 32,768
// droplets: at most 16 of them 3290 / 9406 / 22,843 / 103,940 (the looks then hold up the hand-offs), 256 of them
// 3040 / 5710 / 11,110 / 43,510; waves spread over the terrain are the same with either (2048 droplets: 832, 825).
constexpr uint32_t BACK_NS = 64, BACK_MAX = 256;
constexpr int LONGEST = 4 + (int)BACK_MAX / 8;  // what four looks and the longest sleep count

template <int N>
struct Int {
    static constexpr int value = N;
};

// per droplet state carried from entry to entry
struct Walk {
    double deficit, surplus, prev_live;
    int clamped;
    int32_t death;
    bool sub_death;
};

}  // namespace

// One change-list entry against the live terrain (particle.py:934-1002): the erosion floor (the
// base level or the cell itself, the next path cell's live surface nlive), the deposit ceilings (the
// previous step's live surface, or for a final deposit the next, older path cell), the deficit and
// surplus carried along the droplet's list.  acc is the cell's live net change; returns the new one
// and the amount actually moved (negative: eroded).
template <bool ECAP, bool LAKE>
__device__ __forceinline__ double entry_arith(const PgeParams &p, Walk &w, const EntryRec &r, double acc, double nlive, double capv,
                                              float2 route, double &amount)
{
    const uint32_t f = r.flags;
    const double s_c = r.hs + acc, b_c = (double)r.base;
    double acc_new = acc;
    amount = 0.0;
    if (f & ENTRY_ERO) {
        const double ew = -r.delta;
        double room = p.iter_erode + acc;
        if (ECAP) {
            const double r2 = capv + acc;
            room = r2 < room ? r2 : room;
        }
        double e_act = ew > room ? room : ew;
        double floor_ = s_c >= b_c ? b_c : s_c;
        // a lake bed is never eroded below its water level (particle.py:952-956)
        if (LAKE) floor_ = route.y >= 1.5f && (double)route.x > floor_ ? (double)route.x : floor_;
        floor_ = (f & ENTRY_READS) && nlive > floor_ ? nlive : floor_;
        const double lim = s_c - floor_;
        e_act = e_act > lim ? lim : e_act;
        e_act = e_act < 0.0 ? 0.0 : e_act;
        acc_new = acc - e_act;
        amount = -e_act;
        const bool less = e_act < ew;
        w.clamped += less;
        const double deficit = w.deficit + (ew - e_act);
        w.deficit = less ? deficit : w.deficit;
        const double live = r.hs + acc_new;
        w.prev_live = (f & ENTRY_STEP) ? live : w.prev_live;  // (a bank cut is no step)
    } else if (f & ENTRY_DEP) {
        const bool below = s_c < b_c, is_step = (f & ENTRY_STEP) != 0;
        const double got = r.delta + w.surplus;
        double t = got < w.deficit ? got : w.deficit;
        t = w.deficit > 0.0 ? t : 0.0;
        const double want = got - t;
        w.deficit -= t;
        const double room = p.iter_deposit - acc;
        double d_act = want > room ? room : want;
        // the ceiling: the last step's live surface (none yet: infinite), for a final deposit the next, older path cell's
        double ceil_ = (is_step ? w.prev_live : nlive) + p.dep_floor;
        const double ceil_b = ceil_ - (p.dep_floor + p.fan_slope);
        ceil_ = below && is_step ? ceil_b : ceil_;
        const double lim1 = ceil_ - s_c;
        d_act = (f & (ENTRY_STEP | ENTRY_READS)) && d_act > lim1 ? lim1 : d_act;
        const double lim2 = b_c - p.dep_floor - s_c;
        d_act = below && d_act > lim2 ? lim2 : d_act;
        d_act = d_act < 0.0 ? 0.0 : d_act;
        acc_new = acc + d_act;
        amount = d_act;
        w.clamped += d_act < want;
        w.surplus = want - d_act;
        const double live = r.hs + acc_new;
        w.prev_live = is_step ? live : w.prev_live;
        if (!is_step) {  // the final deposits end the list: the first one's cell takes the stockpile
            w.death = w.death < 0 ? r.cell : w.death;
            w.sub_death = r.cell == w.death ? live < b_c : w.sub_death;
        }
    }
    return acc_new;
}

// a droplet's stockpile (particle.py:1019-1041) and its statistics, once its list is applied
__device__ __forceinline__ void droplet_end(const OrderedArgs &a, const Walk &w, long long q, long long eroded, long long deposited)
{
    const PgeParams &p = a.p;
    long long topend = 0, lostoff = 0;
    int32_t dth = -1;
    double add = 0.0;
    double surplus = w.surplus;
    if (a.park_n) {  // the loads its lakes had no room for join what it could not place (particle.py:1019)
        double refused = 0.0;
        const int np = a.park_n[q];
        for (int j = 0; j < np; j++) refused += a.park_rest[q * LAKE_PARKS + j];
        surplus += refused;
    }
    if (w.death >= 0 && surplus > 0.0) {
        if (w.sub_death) {
            double keep = surplus * (1.0 - p.offshore_writeoff);
            if (keep < 1e-4) keep = 0.0;
            add = keep;
            topend = fx_mass(keep);
            lostoff = fx_mass(surplus) - topend;
        } else {
            add = surplus;
            topend = fx_mass(surplus);
        }
        dth = w.death;
    }
    a.dth[q] = dth;
    a.keep[q] = add;
    PgeStats *st = a.stats;
    auto total = [](int64_t *dst, long long v) {
        if (v) red_add(reinterpret_cast<long long *>(dst), v);
    };
    total(&st->clamped, w.clamped);
    total(&st->to_pending_fx, topend);
    if (w.deficit > 0.0) total(&st->deficit_out_fx, fx_mass(w.deficit));
    total(&st->lost_offshore_fx, lostoff);
    total(&st->eroded_fx, eroded);
    total(&st->deposited_fx, deposited);
}

// One warp a droplet: every lane runs the droplet's entries (the same values in all lanes), the lanes share the
// copies of its records and the statistics of 32 entries at a time.
//
// A block takes the next droplet by a ticket, so the droplets it can wait for -- the earlier ones -- have all started,
// in whatever order the GPU starts a wave's blocks and however few of them it holds at once (20 a multiprocessor, by their
// registers and shared memory): the earliest droplet that has not ended waits for nobody.
//
// Bound by the instructions of one entry on one warp (~110, 215-235 ns; 2048 droplets at work at once: 405), not
// by memory.  What each choice measured, ns an entry without a wait: hand-off words read into registers ahead of
// their use 430 (the compiler's wait for any shared-memory read then waits for them too), by asynchronous copies
// 320, those two entries deep instead of one 223; flags precomputed by the rank kernel and the entries unrolled by
// four (no register moves) 410 -> 320; rare paths (a revisit, a wait) in one branch each 237 -> 226.  Passes, first
// build -> this one: 815 -> 467 us a wave (N_c = 1024), 3620 -> 1843 (N_c = 128, 65,536 droplets), 7007 -> 3697
// (a window of 389^2).
template <bool ECAP, bool LAKE>
__global__ void __launch_bounds__(32) ordered_apply_kernel(const OrderedArgs a)
{
    __shared__ EntryRec rec[REC_RING];
    __shared__ alignas(16) ulonglong2 land[2][4];
    __shared__ double hist[APPLY_HIST];  // the net change each of the last entries left at its cell
    __shared__ double amt[32];           // what each entry of the chunk moved
    __shared__ double capv[ECAP ? REC_RING : 1];
    __shared__ float2 route[LAKE ? REC_RING : 1];
    const PgeParams &p = a.p;
    const int lane = threadIdx.x;
    unsigned int mine = 0;
    if (lane == 0) mine = atomicAdd(a.ticket, 1u);
    const long long q = __shfl_sync(FULL, mine, 0);
    const int K = (int)a.count[q];
    if (K <= 0) {
        if (lane == 0) a.dth[q] = -1;
        return;
    }
    const EntryRec *list = a.rec + q * a.cap;
    auto stage_rec = [&](int e) {
        EntryRec *r = &rec[e & (REC_RING - 1)];
        if (e < K) {
            cp_cg16(r, list + e);
            cp_cg16(reinterpret_cast<char *>(r) + 16, reinterpret_cast<const char *>(list + e) + 16);
        } else {  // past the list's end: an entry that does nothing
            r->flags = ENTRY_OPEN | ENTRY_FIRST | ENTRY_HELD;
            r->cell = 0;
        }
    };
    auto stage_ext = [&](int e) {  // an entry whose record has landed
        if ((ECAP || LAKE) && e < K) {
            const int32_t c = rec[e & (REC_RING - 1)].cell;
            if (ECAP) cp_ca8(&capv[e & (REC_RING - 1)], a.ecap + c);
            if (LAKE) cp_ca8(&route[e & (REC_RING - 1)], a.R + c);
        }
    };
    stage_rec(lane);
    stage_rec(32 + lane);
    cp_commit();
    cp_wait<0>();
    __syncwarp();
    stage_ext(lane);
    EntryRec e0 = rec[0], e1 = rec[1], e2 = rec[2], e3 = rec[3];
    // The hand-off words of the cells ahead: every entry sends for the words of the three after it, which land two
    // entries on (a read of L2 takes as long as an entry); entry e's at e % 4, the sends of even and odd entries apart.
    auto send = [&](int half, int at, int32_t c0, int32_t c1, int32_t c2) {
        const int32_t c = lane == 0 ? c0 : lane == 1 ? c1 : c2;
        __syncwarp();  // every lane has read what the words before these left there
        if (lane < 3) cp_cg16(&land[half][(at + lane) & 3], a.hand + c);
        cp_commit();
    };
    send(1, 0, e0.cell, e1.cell, e2.cell);
    stage_rec(64 + lane);
    cp_commit();
    cp_wait<0>();
    __syncwarp();
    stage_ext(32 + lane);
    ulonglong2 wa = land[1][0], wb = land[1][1];  // this entry's word and the next one's, as last read

    Walk w;
    w.deficit = w.surplus = 0.0;
    w.prev_live = __longlong_as_double(0x7ff0000000000000ll);
    w.clamped = 0;
    w.death = -1;
    w.sub_death = false;
    long long eroded = 0, deposited = 0;
    double held = 0.0;  // the net change of the current entry's cell, where the entry before it read it (ENTRY_HELD)
    int k = 0;

    // entry k + J (A) and the three after it; the record of entry k + J + 4 takes A's place
    auto entry = [&](auto J_, EntryRec &A, const EntryRec &B, const EntryRec &C, const EntryRec &D) -> bool {
        constexpr int J = decltype(J_)::value;
        const uint32_t f = A.flags;
        // the cell's net change, and where this entry needs the next one's cell that one's: a revisit takes what this
        // droplet's own last visit left, else the earlier droplets have to have handed the cell on
        const bool need_a = !(f & (ENTRY_HELD | ENTRY_OPEN)), need_b = (f & ENTRY_NEEDS) && !(B.flags & ENTRY_OPEN);
        bool ok = (!need_a || hand_ready(wa.x, wa.y, A.turn)) && (!need_b || hand_ready(wb.x, wb.y, B.turn));
        ulonglong2 wc;
        const bool late = !ok;
        if (late) {
            for (int i = 0; !ok; i++) {  // (i: the looks, and the sleeps at eight BACK_NS a look)
                if (need_a && !hand_ready(wa.x, wa.y, A.turn)) hand_load(a.hand + A.cell, wa.x, wa.y);
                hand_load(a.hand + B.cell, wb.x, wb.y);
                hand_load(a.hand + C.cell, wc.x, wc.y);
                const bool ok_a = !need_a || hand_ready(wa.x, wa.y, A.turn);
                ok = ok_a && (!need_b || hand_ready(wb.x, wb.y, B.turn));
                if ((i & 3) == 3 && !ok) {
                    // droplets still to come before the one that hands the cell to this one: sleep the least time they
                    // take, so that the looks of all who wait for one cell do not hold up the hand-offs on it
                    const uint32_t at = (uint32_t)((ok_a ? wb.x : wa.x) >> 32), want = ok_a ? B.turn : A.turn;
                    const uint32_t away = want - ((int32_t)(at - a.epoch) < 0 ? a.epoch : at);
                    if (away > 1) {
                        const uint32_t n = away < BACK_MAX ? away - 1 : BACK_MAX;
                        __nanosleep(n * BACK_NS);
                        i += (int)(n >> 3 & ~3u);
                    }
                    if (i >= kSpinLimit || ((i & 255) >= 256 - LONGEST && *(volatile int *)a.error)) {
                        if (i >= kSpinLimit) atomicExch(a.error, 1);
                        return false;  // this wait, or another one, gave up
                    }
                }
            }
        }
        send(J & 1, J + 1, B.cell, C.cell, D.cell);
        double acc = (f & ENTRY_HELD) ? held : hand_acc(wa.x, wa.y), acc_n = hand_acc(wb.x, wb.y);
        const bool again_a = !(f & (ENTRY_HELD | ENTRY_FIRST)), again_b = (f & ENTRY_NEEDS) && !(B.flags & ENTRY_FIRST);
        if (again_a || again_b) {
            auto own = [&](const EntryRec &r, int e) {
                const int back = (int)(r.flags & ENTRY_BACK_MASK);
                return back < APPLY_HIST ? hist[(e - back) & (APPLY_HIST - 1)] : own_value(a.hand, r.cell);
            };
            if (again_a) acc = own(A, k + J);
            if (again_b) acc_n = own(B, k + J + 1);
        }
        acc_n = (f & ENTRY_SAME) ? acc : acc_n;
        double moved;
        const double acc_new = entry_arith<ECAP, LAKE>(p, w, A, acc, B.hs + acc_n, ECAP ? capv[(k & (REC_RING - 1)) + J] : 0.0,
                                                       LAKE ? route[(k & (REC_RING - 1)) + J] : make_float2(0.f, 0.f), moved);
        // a droplet's last write at a cell hands the cell on; before a revisit too far back for `hist` the net change is
        // only left in the word
        if ((f & (ENTRY_LAST | ENTRY_FAR)) && lane == 0) hand_store(a.hand + A.cell, acc_new, A.turn + ((f & ENTRY_LAST) ? 1u : 0u));
        hist[(k & (APPLY_HIST - 1)) + J] = acc_new;
        amt[(k & 31) + J] = moved;
        held = (f & ENTRY_SAME) ? acc_new : acc_n;
        A = rec[((k + 4) & (REC_RING - 1)) + J];
        cp_wait<1>();
        __syncwarp();
        wa = land[(J + 1) & 1][(J + 1) & 3];
        wb = late ? wc : land[(J + 1) & 1][(J + 2) & 3];
        return true;
    };
    bool ok = true;
    while (k < K) {
        const int c0 = k, end = k + 32 < K ? k + 32 : K;
        // (entries past the list's end do nothing)
        for (; k < end; k += 4)
            if (!(ok = entry(Int<0>{}, e0, e1, e2, e3) && entry(Int<1>{}, e1, e2, e3, e0) && entry(Int<2>{}, e2, e3, e0, e1) &&
                       entry(Int<3>{}, e3, e0, e1, e2)))
                break;
        if (!ok) break;
        // the chunk's statistics, and the records of the chunk two on (the next one's have landed)
        __syncwarp();
        if (c0 + lane < end) {
            const double x = amt[lane];
            if (signbit(x))
                eroded += fx_mass(-x);
            else
                deposited += fx_mass(x);
        }
        cp_wait<0>();
        __syncwarp();
        stage_rec(k + 64 + lane);
        stage_ext(k + 32 + lane);
        cp_commit();
    }
    cp_wait<0>();
    for (int o = 16; o > 0; o >>= 1) {
        eroded += __shfl_xor_sync(FULL, eroded, o);
        deposited += __shfl_xor_sync(FULL, deposited, o);
    }
    if (ok && lane == 0) droplet_end(a, w, q, eroded, deposited);
}

// ---------------------------------------------------------------------------
// after the apply: per touched cell, in the serial (droplet, entry) order, the discharge and
// momentum tracks (particle.py:1013-1018) and the stockpile (:1019-1041); then the cell's net
// change to the accumulators and its packed samples (:1005-1009).  First every sorted slot gathers
// what its entry adds into arrays in sorted order (one thread a slot, all loads in flight at once);
// then each cell's run of those arrays is summed in order, by a lane where it ends within 64 slots,
// else by a whole warp.
// ---------------------------------------------------------------------------
__global__ void ordered_gather_kernel(const OrderedArgs a, long long nslots, const SortKey *keys, const int32_t *vals,
                                      SortKey invalid, FinishRows g)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nslots; i += (long long)gridDim.x * blockDim.x) {
        const SortKey key = keys[i];
        if (key == invalid) continue;
        const int32_t s = vals[i], q = s / a.cap;
        const bool active = !a.mask || a.mask[key] == PGE_MASK_ACTIVE;
        const float v = a.vol[s];
        const bool track = active && v > 0.0f;
        g.v[i] = track ? v : 0.0f;
        g.m0[i] = track ? a.mom[2 * (long long)s] : 0.0f;
        g.m1[i] = track ? a.mom[2 * (long long)s + 1] : 0.0f;
        g.kp[i] = (a.rec[s].flags & ENTRY_LAST) && a.dth[q] == (int32_t)key ? a.keep[q] : -1.0;  // keep >= 0
    }
}

// One warp per 32 consecutive sorted slots, for the cell runs that start there.  The rows of 64 slots are laid out as
// float64 in shared memory; a run that ends within them is added by the lane of its first slot, all of a warp's runs at
// once.  A longer one is walked by the whole warp, 32 entries at a time (the next window's rows read while this one is
// added), four lanes adding one sum each -- the discharge, the two momentum tracks and the stockpile.  Either way a sum
// is added in slot order, the serial order.  (An entry that adds nothing to a sum adds 0, which leaves it as it is: the
// sums start at +0 and so are never -0.)
//
// Bound by the latency of a run's reads and the float64 adds of the longest.  Every run walked by the warp, one after
// another: 36.6 us a wave at N_c = 1024, 81-104 at N_c = 128 where hundreds of a wave's droplets cross a cell; 8.1 and 30.
constexpr int FINISH_THREADS = 256, FINISH_WARPS = FINISH_THREADS / 32, FINISH_PITCH = 68;  // (no two sums' reads share a bank)

struct FinishRow {
    float v, m0, m1;
    double kp;
};

__global__ void __launch_bounds__(FINISH_THREADS) ordered_finish_kernel(const OrderedArgs a, long long nslots, const SortKey *keys,
                                                                        SortKey invalid, FinishRows g)
{
    __shared__ double win[FINISH_WARPS][4][FINISH_PITCH];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double(*w)[FINISH_PITCH] = win[threadIdx.x >> 5];
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    auto row = [&](long long j) { return FinishRow{g.v[j], g.m0[j], g.m1[j], g.kp[j]}; };
    auto lay = [&](int at, const FinishRow &r) {
        const bool step = r.v > 0.0f;  // a step of volume > 0 on an active cell (gathered as 0 otherwise)
        w[0][at] = step ? (double)r.v : 0.0;
        w[1][at] = step ? (double)r.m0 : 0.0;
        w[2][at] = step ? (double)r.m1 : 0.0;
        w[3][at] = r.kp >= 0.0 ? r.kp : 0.0;
    };
    const FinishRow none{0.0f, 0.0f, 0.0f, -1.0};
    // a touched cell's net change to the accumulators and its packed samples (particle.py:1005-1009)
    auto settle = [&](long long c) {
        const unsigned long long *hw = reinterpret_cast<const unsigned long long *>(a.hand + c);
        const double acc = hand_acc(hw[0], hw[1]);
        a.acc4[4 * c] = acc;
        if (!a.mask || a.mask[c] == PGE_MASK_ACTIVE) {
            const float surf = (float)(a.L[c].x + acc);
            a.A[c].x = surf;
            const double sd = a.sediment[c] + acc;
            a.B[c].z = (float)(sd > 0.0 ? sd : 0.0);
            // the route flag follows the live surface; a lake cell stays a lake cell (particle.py:1010-1012)
            if (a.R && a.R[c].y < 1.5f) a.R[c].y = a.R[c].x != surf ? 1.0f : 0.0f;
        }
    };
    for (long long base = warp * 32; base < nslots; base += nwarps * 32) {
        const long long i = base + lane, i2 = i + 32;
        const SortKey k0 = i < nslots ? keys[i] : invalid, k1 = i2 < nslots ? keys[i2] : invalid;
        SortKey before = __shfl_up_sync(full, k0, 1);
        if (lane == 0) before = base > 0 ? keys[base - 1] : ~k0;
        SortKey mid = __shfl_up_sync(full, k1, 1);
        const SortKey last0 = __shfl_sync(full, k0, 31);
        if (lane == 0) mid = last0;
        const bool head = k0 != invalid && before != k0;
        const unsigned heads = __ballot_sync(full, head);
        if (!heads) continue;
        // bit b: slot base + b does not go on with the run of the slot before it
        const unsigned long long ends = (unsigned long long)__ballot_sync(full, before != k0) | ((unsigned long long)__ballot_sync(full, mid != k1) << 32);
        const unsigned long long rest = lane < 63 ? ends >> (lane + 1) : 0ull;
        const int len = rest ? __ffsll((long long)rest) : 0;  // 0: the run goes on past the window
        lay(lane, k0 != invalid ? row(i) : none);
        lay(32 + lane, k1 != invalid ? row(i2) : none);
        __syncwarp();
        if (head && len) {
            const long long c = (long long)k0;
            double *accp = a.acc4 + 4 * c;
            double tq = accp[1], ta = accp[2], tb = accp[3], pd = a.pend[c];
            for (int t = lane; t < lane + len; t++) {
                tq += w[0][t];
                ta += w[1][t];
                tb += w[2][t];
                pd += w[3][t];
            }
            accp[1] = tq;
            accp[2] = ta;
            accp[3] = tb;
            a.pend[c] = pd;
            settle(c);
        }
        __syncwarp();
        unsigned longer = __ballot_sync(full, head && !len);  // (at most the last run)
        while (longer) {
            const int hl = __ffs(longer) - 1;
            longer &= longer - 1;
            const SortKey key = __shfl_sync(full, k0, hl);
            const long long c = (long long)key;
            double *mine = lane < 3 ? a.acc4 + 4 * c + 1 + lane : a.pend + c;  // this lane's sum (the first four lanes)
            double sum = lane < 4 ? *mine : 0.0;
            long long j = base + hl + lane;
            bool in = j < nslots && keys[j] == key;
            FinishRow r = in ? row(j) : none;
            while (true) {
                const int n = __popc(__ballot_sync(full, in));  // the run covers a prefix of the lanes (keys are sorted)
                lay(lane, r);
                if (n == 32) {
                    j += 32;
                    in = j < nslots && keys[j] == key;
                    r = in ? row(j) : none;
                }
                __syncwarp();
                const double *mw = w[lane & 3];
                if (n == 32) {
#pragma unroll 8
                    for (int t = 0; t < 32; t++) sum += mw[t];
                } else {
                    for (int t = 0; t < n; t++) sum += mw[t];
                }
                __syncwarp();  // every lane has read the window before the next one is written
                if (n < 32) break;
            }
            if (lane < 4) *mine = sum;
            if (lane == 0) settle(c);
        }
    }
}

// zero the hand-off counters (the live net changes stay), so the 32-bit epochs can start over
__global__ void hand_reset_kernel(long long ncell, double2 *hand)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        unsigned long long *hw = reinterpret_cast<unsigned long long *>(hand + c);
        hw[0] &= 0xffffffffull;
        hw[1] &= 0xffffffffull;
    }
}

cudaError_t hand_reset(long long ncell, double2 *hand, cudaStream_t st)
{
    hand_reset_kernel<<<grid_for(ncell), 256, 0, st>>>(ncell, hand);
    return cudaPeekAtLastError();
}

cudaError_t ordered_terrain(long long ncell, const double2 *L, const float4 *B, const uint8_t *mask, CellTerr *terr, cudaStream_t st)
{
    ordered_terrain_kernel<<<grid_for(ncell), 256, 0, st>>>(ncell, L, B, mask, terr);
    return cudaPeekAtLastError();
}

cudaError_t ordered_wave(const OrderedWave &w, cudaStream_t st)
{
    long long nslots = w.nw * w.cap;
    size_t tb = w.temp_bytes;
    cudaError_t e;
    if (w.offsets) {
        // long lists (a lifetime of thousands of steps, most of it unused): only the recorded entries go through
        // the ranks, in (droplet, entry) order; their count comes back to the host for the library sorts
        if ((e = cub::DeviceScan::ExclusiveSum(w.temp, tb, w.a.count, w.offsets, (int)w.nw, st)) != cudaSuccess) return e;
        entry_total_kernel<<<1, 1, 0, st>>>(w.a.count, w.offsets, w.nw, w.offsets + w.nw);
        long long total = 0;
        if ((e = cudaMemcpyAsync(&total, w.offsets + w.nw, sizeof(long long), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
        ordered_compact_keys_kernel<<<grid_for(nslots), 256, 0, st>>>(nslots, w.cap, w.a.cell, w.a.count, w.offsets, w.keys_in,
                                                                      w.vals_in, w.tails, w.a.ticket);
        nslots = total;
    } else {
        ordered_keys_kernel<<<grid_for(nslots), 256, 0, st>>>(nslots, w.cap, w.a.cell, w.a.count, w.invalid, w.keys_in, w.vals_in,
                                                              w.tails, w.a.ticket);
    }
    tb = w.temp_bytes;
    e = cub::DeviceRadixSort::SortPairs(w.temp, tb, w.keys_in, w.keys_out, w.vals_in, w.vals_out, (int)nslots, 0, w.end_bit, st);
    if (e != cudaSuccess) return e;
    ordered_rank_kernel<<<grid_for(nslots), 256, 0, st>>>(nslots, w.keys_out, w.vals_out, w.cap, w.invalid, w.a.delta, w.a.vol, w.a.count,
                                                          w.a.terr, w.a.epoch, w.tails, const_cast<EntryRec *>(w.a.rec));
    const bool lake = w.a.lakes && w.a.R;
    const int blocks = (int)w.nw;  // a warp per droplet
    if (w.a.ecap && lake)
        ordered_apply_kernel<true, true><<<blocks, 32, 0, st>>>(w.a);
    else if (w.a.ecap)
        ordered_apply_kernel<true, false><<<blocks, 32, 0, st>>>(w.a);
    else if (lake)
        ordered_apply_kernel<false, true><<<blocks, 32, 0, st>>>(w.a);
    else
        ordered_apply_kernel<false, false><<<blocks, 32, 0, st>>>(w.a);
    FinishRows g;
    g.v = w.fin[0];
    g.m0 = w.fin[1];
    g.m1 = w.fin[2];
    g.kp = reinterpret_cast<double *>(w.keys_in);  // (the sort's input keys are free again)
    ordered_gather_kernel<<<grid_for(nslots), 256, 0, st>>>(w.a, nslots, w.keys_out, w.vals_out, w.invalid, g);
    ordered_finish_kernel<<<grid_for(nslots, FINISH_THREADS), FINISH_THREADS, 0, st>>>(w.a, nslots, w.keys_out, w.invalid, g);
    return cudaPeekAtLastError();
}

}  // namespace pge
