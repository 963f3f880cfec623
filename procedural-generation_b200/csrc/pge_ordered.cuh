// pge_ordered.cuh -- the droplet-ordered apply of one wave (pge_ordered.cu).
#pragma once
#include "pge_internal.cuh"

namespace pge {

// one entry of a wave's change lists as the ordered apply reads it (built by the rank kernel): the entry, its
// cell's read-only terrain and where its droplet was there before, so that the apply reads nothing else but the
// hand-off words
struct alignas(16) EntryRec {
    double delta;
    double hs;       // height + sediment at the start of the pass
    float base;
    uint32_t flags;  // ENTRY_* | entries since its droplet's previous visit to the cell (0: none; APPLY_HIST: that or more)
    int32_t cell;
    uint32_t turn;   // the cell's hand-off counter once the earlier droplets of the wave have handed it on
};
static_assert(sizeof(EntryRec) == 32, "two 16-byte reads an entry");
// entries whose net change the apply keeps on chip for its droplet's own revisits
constexpr int APPLY_HIST = 128;
constexpr uint32_t ENTRY_BACK_MASK = 0xffu;
constexpr uint32_t ENTRY_LAST = 1u << 8;    // its droplet's last visit to the cell
constexpr uint32_t ENTRY_FIRST = 1u << 9;   // its droplet's first visit to the cell
constexpr uint32_t ENTRY_OPEN = 1u << 10;   // no earlier droplet to wait for: a revisit, or the wave's first visitor
constexpr uint32_t ENTRY_STEP = 1u << 11;   // a step entry (vol >= 0), not a bank cut, a park or a final deposit
constexpr uint32_t ENTRY_DEP = 1u << 12;    // deposits (delta >= 0) on an active cell
constexpr uint32_t ENTRY_ERO = 1u << 13;    // erodes (delta < 0) an active cell; neither: changes nothing (a lake park among them)
constexpr uint32_t ENTRY_READS = 1u << 14;  // reads the next entry's cell: an erosion's floor, a final deposit's ceiling
constexpr uint32_t ENTRY_NEEDS = 1u << 15;  // reads it, and it is another cell
constexpr uint32_t ENTRY_SAME = 1u << 16;   // the next entry is at the same cell
constexpr uint32_t ENTRY_HELD = 1u << 17;   // the entry before it read this cell, or is at it: its net change is at hand
constexpr uint32_t ENTRY_FAR = 1u << 18;    // its droplet comes back only after APPLY_HIST entries or more

// a cell's read-only terrain for the ordered apply (built once per pass)
struct alignas(16) CellTerr {
    double hs;        // height + sediment at the start of the pass
    float base;
    uint32_t active;  // 1: the cell's mask is PGE_MASK_ACTIVE
};

struct OrderedArgs {
    // the wave's change lists, `cap` slots per droplet
    const int32_t *cell;
    const double *delta;
    const float *vol;
    const float *mom;
    const int64_t *count;
    int cap;
    long long nw;
    const EntryRec *rec;
    const CellTerr *terr;
    // terrain
    const double2 *L;  // x: height + sediment
    const double *sediment;
    float4 *A;
    float4 *B;
    float2 *R;  // packed routing surface (route, flag) or nullptr: flags follow the live surface
    int lakes;  // R's flags mark overflowing lakes: a lake bed is not eroded below its routing surface
    const uint8_t *mask;
    const double *ecap;
    // per cell: the live net change and the hand-off counter, one 16-byte word
    double2 *hand;
    uint32_t epoch;  // this wave's: a cell with D earlier visitors is free once its counter reads epoch + D
    // per droplet: the stockpile cell (-1: none) and the amount it adds there
    int32_t *dth;
    double *keep;
    // float64 accumulators in serial order: (net change, discharge, momentum a, b) and the stockpile
    double *acc4;
    double *pend;
    PgeParams p;
    PgeStats *stats;
    int *error;
    unsigned int *ticket;  // droplets of the wave taken so far (zeroed by the keys kernel)
    // lake parks (nullptr: off): per droplet its park count, per park (LAKE_PARKS a droplet) the rest its lake
    // had no room for, added to the droplet's leftover load in list order
    const int32_t *park_n;
    const double *park_rest;
};

// the lake parks of one wave (erosion.lake_fill): each lake's room counted down in droplet order
struct ParkWave {
    long long nw;  // droplets of the wave
    int cap;
    const int32_t *cell;
    const double *delta;
    const int32_t *park_n, *park_k;  // per droplet its parks and their entry indices
    const int32_t *lake_id;          // per cell
    double *lake_room;               // per lake, counted down in place
    long long lakes;
    double *lake_load;               // per cell, the loads the lakes took
    double *rest;                    // out: per park the rest refused
    uint32_t *keys_in, *keys_out;
    int32_t *vals_in, *vals_out;
    void *temp;
    size_t temp_bytes;
};

// what each sorted slot adds to its cell, gathered in sorted order for the finish
struct FinishRows {
    float *v, *m0, *m1;  // step volume and momentum (0 unless a step of volume > 0 on an active cell)
    double *kp;          // the droplet's stockpile where this is its last visit to its stockpile cell, else -1
};

// the ranks' sort key, an entry's cell: 64 bits wide, since the library's tile for 32-bit keys leaves a wave's ~260,000
// slots on too few blocks (10.9 us a digit against 9.9)
typedef unsigned long long SortKey;

struct OrderedWave {
    OrderedArgs a;
    long long nw;
    int cap, end_bit;
    SortKey invalid;
    SortKey *keys_in, *keys_out;
    int32_t *vals_in, *vals_out;
    float *fin[3];  // the finish's gathered rows, a float a slot each
    uint32_t *tails;  // the ranks' count of each 32 sorted slots' last run (the finish's rows are free until the finish)
    void *temp;
    size_t temp_bytes;
    // long lists: the recorded entries compacted before the ranks (nullptr: every slot goes through them);
    // max_wave + 1 int64: each droplet's first entry, then the wave's total
    long long *offsets;
};

// the list length above which a wave's entries are compacted before their ranks (a host read a wave)
#ifndef PGE_COMPACT_CAP
#define PGE_COMPACT_CAP 512
#endif
constexpr int COMPACT_CAP = PGE_COMPACT_CAP;

size_t ordered_temp_bytes(long long nslots, long long max_wave);
cudaError_t park_wave(const ParkWave &pw, cudaStream_t st);
cudaError_t ordered_wave(const OrderedWave &w, cudaStream_t st);
cudaError_t hand_reset(long long ncell, double2 *hand, cudaStream_t st);
cudaError_t ordered_terrain(long long ncell, const double2 *L, const float4 *B, const uint8_t *mask, CellTerr *terr, cudaStream_t st);

}  // namespace pge
