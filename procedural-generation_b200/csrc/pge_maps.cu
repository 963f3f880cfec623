// pge_maps.cu -- the per-iteration map passes around the droplet pass.
//
// Compiled with -fmad=false like the float64 droplet trace, so the float64
// stencils round like the reference's numba / numpy code.
//
//   pack / refresh / fold+EMA   particle.py:164-191, 1005-1012, 1079-1101, 1230-1242
//   thermal passes a / r / b    particle.py:1107-1227, maps.py:1050-1085
//   uplift                      maps.py:1088-1147
//   datum order statistic       maps.py:1446-1508 (radix select instead of np.partition)
//   halo gather                 field.py:104-125
//   spawn weights / inverse CDF maps.py:793-833, particle.py:1245-1260
#include <cstring>

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "pge_internal.cuh"
#include "pge_maps.cuh"

namespace pge {

namespace {
__device__ __forceinline__ bool interior(long long c, int NE, int H, int N)
{
    const unsigned u = (unsigned)c, row = u / (unsigned)NE;  // (a cell index fits 31 bits)
    const int j = (int)(u - row * (unsigned)NE), i = (int)(row % (unsigned)NE);
    return i >= H && i < H + N && j >= H && j < H + N;
}

inline int grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    return (int)(b < 1 ? 1 : (b > 1048576 ? 1048576 : b));
}
// a grid-stride launch for kernels that end in a few global atomics a block: 8 blocks a multiprocessor
inline int grid_reduce(long long n, int threads = 256)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 148;
    }
    const int b = grid_for(n, threads);
    return b < 8 * sms ? b : 8 * sms;
}
}  // namespace

// ---------------------------------------------------------------------------
// pack / refresh / fold + EMA
// ---------------------------------------------------------------------------
__global__ void pack_kernel(long long ncell, const double *__restrict__ h, const double *__restrict__ s,
                            const double *__restrict__ q, const double *__restrict__ mom, const float *__restrict__ evap,
                            const float *__restrict__ hard, const double *__restrict__ base, float4 *A, float4 *B, double2 *L)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const double sd = s[c];
        const double hs = h[c] + sd;
        A[c] = make_float4((float)hs, (float)q[c], (float)mom[2 * c], (float)mom[2 * c + 1]);
        B[c] = make_float4(evap[c], hard[c], (float)sd, (float)base[c]);
        L[c] = make_double2(hs, 0.0);
    }
}

__global__ void pack_metric_kernel(long long n, const float *__restrict__ g, const float *__restrict__ gi, float4 *G)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        G[2 * c] = make_float4(g[3 * c], g[3 * c + 1], g[3 * c + 2], gi[3 * c]);
        G[2 * c + 1] = make_float4(gi[3 * c + 1], gi[3 * c + 2], 0.f, 0.f);
    }
}

// between waves: the packed surface / sediment and the ledger's wave-start
// change follow the net change so far (apply_changes' samp sync, particle.py:1005-1009)
__global__ void refresh_kernel(long long ncell, const double *__restrict__ s, const long long *__restrict__ acc4, float4 *A,
                               float4 *B, double2 *L, float2 *R)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const double a = (double)acc4[4 * c] * INV_FX_MASS;
        double2 l = L[c];
        if (l.y == a) continue;  // unchanged since the last refresh
        l.y = a;
        L[c] = l;
        const float surf = (float)(l.x + a);
        A[c].x = surf;
        const double sd = s[c] + a;
        B[c].z = (float)(sd > 0.0 ? sd : 0.0);
        // the route flag follows the live surface; a lake cell stays a lake cell (particle.py:1010-1012)
        if (R && R[c].y < 1.5f) R[c].y = R[c].x != surf ? 1.0f : 0.0f;
    }
}

// the routing surface and its flag, beside the packed surface (particle.py:165-190): 2 on an
// overflowing lake, 3 on one with room for its rivers' load, else 1 where the route is not the surface
__global__ void pack_route_kernel(long long ncell, const double *__restrict__ h, const double *__restrict__ s,
                                  const double *__restrict__ route, const uint8_t *__restrict__ lake, float2 *R)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const float r = (float)route[c], surf = (float)(h[c] + s[c]);
        const uint8_t lk = lake ? lake[c] : (uint8_t)0;
        R[c] = make_float2(r, lk > 0 ? (lk > 1 ? 3.0f : 2.0f) : (r != surf ? 1.0f : 0.0f));
    }
}

// the lakes of a window (maps.py:662-672): interior active cells the routing surface covers more
// than min_depth deep
__global__ void window_lakes_kernel(long long ncell, int N, int H, const double *__restrict__ h, const double *__restrict__ s,
                                    const double *__restrict__ route, const uint8_t *__restrict__ mask, double min_depth,
                                    uint8_t *flag, unsigned long long *count)
{
    const int NE = N + 2 * H;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(c % NE), i = (int)((c / NE) % NE);
        const bool inner = i >= H && i < H + N && j >= H && j < H + N;
        const bool lake = inner && (!mask || mask[c] == PGE_MASK_ACTIVE) && route[c] - (h[c] + s[c]) > min_depth;
        flag[c] = lake ? 1 : 0;
        const unsigned ballot = __ballot_sync(__activemask(), lake);
        if (count && ballot && (threadIdx.x & 31) == __ffs(ballot) - 1) atomicAdd(count, (unsigned long long)__popc(ballot));
    }
}

// the accumulators as float64: fixed point (wave apply) or plain float64 (ordered apply)
__device__ __forceinline__ void acc_values(const long long *acc4, const long long *pend, long long c, int exact, double &a,
                                           double &q, double &ma, double &mb, double &pd)
{
    if (exact) {
        const double *d4 = reinterpret_cast<const double *>(acc4);
        a = d4[4 * c];
        q = d4[4 * c + 1];
        ma = d4[4 * c + 2];
        mb = d4[4 * c + 3];
        pd = reinterpret_cast<const double *>(pend)[c];
    } else {
        a = (double)acc4[4 * c] * INV_FX_MASS;
        q = (double)acc4[4 * c + 1] * INV_FX_TRACK;
        ma = (double)acc4[4 * c + 2] * INV_FX_TRACK;
        mb = (double)acc4[4 * c + 3] * INV_FX_TRACK;
        pd = (double)pend[c] * INV_FX_MASS;
    }
}

__global__ void fold_ema_kernel(long long ncell, double *h, double *s, double *q, double *mom, double *pending,
                                const uint8_t *__restrict__ mask, const long long *__restrict__ acc4,
                                const long long *__restrict__ pend, double ema, int exact)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const bool act = mask ? mask[c] == PGE_MASK_ACTIVE : true;
        double a, tq, tma, tmb, pd;
        acc_values(acc4, pend, c, exact, a, tq, tma, tmb, pd);
        if (a != 0.0 && act) {
            if (a > 0.0) {
                s[c] += a;
            } else {
                const double take = -a, sd = s[c];
                if (sd >= take) {
                    s[c] = sd - take;
                } else {
                    h[c] -= take - sd;
                    s[c] = 0.0;
                }
            }
        }
        if (act) {
            q[c] = (1.0 - ema) * q[c] + ema * tq;
            mom[2 * c] = (1.0 - ema) * mom[2 * c] + ema * tma;
            mom[2 * c + 1] = (1.0 - ema) * mom[2 * c + 1] + ema * tmb;
        }
        if (pd != 0.0) pending[c] += pd;
    }
}

__global__ void read_acc_kernel(long long ncell, const long long *__restrict__ acc4, const long long *__restrict__ pend,
                                const unsigned long long *mode, double *acc, double *dtr, double *mtr, double *pending)
{
    const int exact = (int)*mode;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        double a, q, ma, mb, pd;
        acc_values(acc4, pend, c, exact, a, q, ma, mb, pd);
        if (acc) acc[c] = a;
        if (dtr) dtr[c] = q;
        if (mtr) {
            mtr[2 * c] = ma;
            mtr[2 * c + 1] = mb;
        }
        if (pending) pending[c] = pd;
    }
}

void pack(const PgeGrid &g, const PgeState &s, const Layout &lay, void *ws, cudaStream_t st)
{
    const long long n = lay.ncell;
    pack_kernel<<<grid_for(n), 256, 0, st>>>(n, s.height, s.sediment, s.discharge, s.momentum, s.evap, s.hardness, s.base,
                                             ws_ptr<float4>(ws, lay.cellA), ws_ptr<float4>(ws, lay.cellB),
                                             ws_ptr<double2>(ws, lay.live));
    pack_metric_kernel<<<grid_for(lay.nmetric), 256, 0, st>>>(lay.nmetric, s.metric, s.metric_inv, ws_ptr<float4>(ws, lay.metric8));
    if (s.route)
        pack_route_kernel<<<grid_for(n), 256, 0, st>>>(n, s.height, s.sediment, s.route, s.lake_flag, ws_ptr<float2>(ws, lay.route2));
}

void refresh(const PgeState &s, const Layout &lay, void *ws, cudaStream_t st)
{
    refresh_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, s.sediment, ws_ptr<long long>(ws, lay.acc4),
                                                       ws_ptr<float4>(ws, lay.cellA), ws_ptr<float4>(ws, lay.cellB),
                                                       ws_ptr<double2>(ws, lay.live), s.route ? ws_ptr<float2>(ws, lay.route2) : nullptr);
}

void fold_ema(PgeState &s, const Layout &lay, void *ws, double ema, int exact, cudaStream_t st)
{
    fold_ema_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, s.height, s.sediment, s.discharge, s.momentum, s.pending,
                                                        s.mask, ws_ptr<long long>(ws, lay.acc4), ws_ptr<long long>(ws, lay.pend),
                                                        ema, exact);
}

void read_accumulators(const Layout &lay, void *ws, double *acc, double *dtr, double *mtr, double *pending, cudaStream_t st)
{
    read_acc_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, ws_ptr<long long>(ws, lay.acc4),
                                                        ws_ptr<long long>(ws, lay.pend),
                                                        ws_ptr<unsigned long long>(ws, lay.counters) + 4, acc, dtr, mtr, pending);
}

// ---------------------------------------------------------------------------
// the erode / deposit brush: the change each cell received since the last spread (the wave apply adds
// every entry's applied change to its own cell) is shared out over the active cells of its face within
// distance < r + 1 (the interior ones on the sphere), weights r + 1 - distance in integers of
// 1/PGE_BRUSH_SCALE renormalised over the footprint; each share is truncated toward zero and the rest
// stays on the cell, so the total is kept exactly.  A gather: each cell adds the shares its neighbours
// send it, computed by the same expression the sender uses for its rest, so no atomics are needed and the
// result is the same whatever the order.
// ---------------------------------------------------------------------------
struct BrushGeo {
    int NE, lo, hi, r;
    const uint8_t *mask;
};

__device__ __forceinline__ int brush_weight(int r, int di, int dj)
{
    const double v = (double)(r + 1) - sqrt((double)(di * di + dj * dj));
    return v > 0.0 ? (int)llround(PGE_BRUSH_SCALE * v) : 0;
}

__device__ __forceinline__ bool brush_valid(const BrushGeo &g, long long fb, int i, int j)
{
    if (i < g.lo || i >= g.hi || j < g.lo || j >= g.hi) return false;
    return !g.mask || g.mask[fb + (long long)i * g.NE + j] == PGE_MASK_ACTIVE;
}

__device__ __forceinline__ long long brush_share(long long d, int q, int Q) { return (long long)((double)d * (double)q / (double)Q); }

// pass 1: each cell's change since the last spread and, where it has one, its footprint's total weight
__global__ void brush_delta_kernel(long long ncell, BrushGeo g, const long long *acc4, const long long *prev, long long *delta, int *Q)
{
    const long long plane = (long long)g.NE * g.NE;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const long long d = acc4[4 * c] - prev[c];
        delta[c] = d;
        int q = 0;
        if (d != 0) {
            const long long fb = c / plane * plane;
            const int ei = (int)((c - fb) / g.NE), ej = (int)((c - fb) % g.NE);
            for (int di = -g.r; di <= g.r; di++)
                for (int dj = -g.r; dj <= g.r; dj++) {
                    const int w = brush_weight(g.r, di, dj);
                    if (w && ((di == 0 && dj == 0) || brush_valid(g, fb, ei + di, ej + dj))) q += w;
                }
        }
        Q[c] = q;
    }
}

// pass 2: the shares the footprint sends each cell, plus the rest of its own change; net change = the last spread + that
__global__ void brush_gather_kernel(long long ncell, BrushGeo g, const long long *delta, const int *Q, long long *acc4, long long *prev)
{
    const long long plane = (long long)g.NE * g.NE;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const long long fb = c / plane * plane;
        const int ei = (int)((c - fb) / g.NE), ej = (int)((c - fb) % g.NE);
        long long sum = 0;
        if (brush_valid(g, fb, ei, ej))
            for (int di = -g.r; di <= g.r; di++) {
                const int i = ei + di;
                if (i < 0 || i >= g.NE) continue;
                for (int dj = -g.r; dj <= g.r; dj++) {
                    const int j = ej + dj;
                    const int w = brush_weight(g.r, di, dj);
                    if (!w || (di == 0 && dj == 0) || j < 0 || j >= g.NE) continue;
                    const long long s = fb + (long long)i * g.NE + j;
                    const long long d = delta[s];
                    if (d != 0) sum += brush_share(d, w, Q[s]);
                }
            }
        const long long d = delta[c];
        if (d != 0) {
            long long kept = d;
            for (int di = -g.r; di <= g.r; di++)
                for (int dj = -g.r; dj <= g.r; dj++) {
                    const int w = brush_weight(g.r, di, dj);
                    if (!w || (di == 0 && dj == 0) || !brush_valid(g, fb, ei + di, ej + dj)) continue;
                    kept -= brush_share(d, w, Q[c]);
                }
            sum += kept;
        }
        if (sum != 0 || d != 0) {
            const long long v = prev[c] + sum;
            acc4[4 * c] = v;
            prev[c] = v;
        }
    }
}

void brush_spread(const PgeGrid &g, const PgeState &s, const Layout &lay, void *ws, int r, cudaStream_t st)
{
    const int NE = g.N + 2 * g.H;
    BrushGeo bg{NE, g.spherical ? g.H : 0, g.spherical ? g.H + g.N : NE, r, s.mask};
    long long *acc4 = ws_ptr<long long>(ws, lay.acc4);
    long long *prev = ws_ptr<long long>(ws, lay.spread);
    long long *delta = ws_ptr<long long>(ws, lay.pwv);
    int *Q = ws_ptr<int>(ws, lay.flags);
    brush_delta_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, bg, acc4, prev, delta, Q);
    brush_gather_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, bg, delta, Q, acc4, prev);
}

// ---------------------------------------------------------------------------
// thermal erosion (talus / creep mass wasting)
// ---------------------------------------------------------------------------
struct ThermalArgs {
    int NE;
    const double *h, *s;
    const float *metric;  // (NE,NE,3) shared or (F,NE,NE,3)
    int metric_shared;
    const float *hard;    // talus = soft + (hard - soft) * hardness, in float32; nullptr: talus 0
    float talus_soft, talus_diff;
    const uint8_t *mask;  // nullptr: all active
    const double *base;   // creep: submerged cells (h + s < base) are frozen
    int creep;
    double rate, cap, dep_floor;
    double *new_h, *new_s;
};

// One pass, a tile a block: the tile's surface and three cells around it in shared memory, then in turn every cell's
// flows to its neighbours and their scale (two cells around), the share of its inflow a submerged cell has room for
// (one cell around), and the cells' new height and sediment -- the reference's three sweeps (particle.py:1107-1227) in
// its order of additions.  A flow and the one back share a distance, so a cell keeps four.
//
// Bound by shared-memory reads and float64 arithmetic, not by memory.  N_c = 1024, talus and creep: 1050 us as three
// sweeps of HBM and a copy (every neighbour's mask, surface and metric read and its distance's root taken 24 times a
// cell); as tiles of 16 x 32 464 with each flow computed again wherever it is used, 462 with the flows in shared memory,
// 427 with a thread's own flows in registers and its neighbours' already at their scale; tiles of 16 x 16 400, of
// 8 x 32 or 8 x 16 417.  The tile stays below the 48 KB a block may have without a function attribute: setting one
// waits until no other thread of the process is in a launch, and a thread that runs a pass of many waves is in one
// nearly all the time (64 worlds together, six iterations each: 3.0 to 4.2 s with the attribute set a call, 2.25).
//
// The metric is the six faces' alike, so a block takes its tile of every face in turn where one face's tiles fill the
// GPU (TH_FILL: four blocks on each of 148 multiprocessors), us, a face a block / in turn: N_c = 256 (289 tiles a face)
// 58 / 64, 320 (441) 75 / 71, 512 (1089) 144 / 127, 1024 (4225) 500 / 400.
constexpr int TH_I = 16, TH_J = 16, TH_THREADS = TH_I * TH_J, TH_FILL = 592;
constexpr int TH_RING = (TH_I + 4) * (TH_J + 4) - TH_THREADS;  // the two cells around the tile
struct ThermalTile {
    double sent[8][TH_I + 4][TH_J + 4];  // a cell's flow to each neighbour at its scale
    double dist[4][TH_I + 4][TH_J + 4];
    double surf[TH_I + 6][TH_J + 6];
    double rscale[TH_I + 2][TH_J + 2];
    uint8_t m[TH_I + 6][TH_J + 6];
};

// MASKED: some cells may be frozen or outside (a mask, or the creep pass's submerged cells)
template <bool MASKED>
__global__ void __launch_bounds__(TH_THREADS, 4) thermal_tile_kernel(const ThermalArgs t, int faces)
{
    __shared__ ThermalTile T;
    const int NE = t.NE, i0 = blockIdx.y * TH_I, j0 = blockIdx.x * TH_J;
    constexpr int DI[8] = {1, 1, 0, -1, -1, -1, 0, 1}, DJ[8] = {0, 1, 1, 1, 0, -1, -1, -1};  // k + 4 is opposite k
    const double half_rate = 0.5 * t.rate;
    // this thread's cell of the tile, and (the first TH_RING threads) one of the cells around it
    const int ta = threadIdx.x / TH_J, tb = threadIdx.x - ta * TH_J;
    int ra = 0, rb = 0;
    {
        const int q = threadIdx.x, w = TH_J + 4;
        if (q < 4 * w) {  // two rows above, two below
            const int r = q / w;
            ra = r < 2 ? r : TH_I + r;
            rb = q - r * w;
        } else {  // two columns on either side
            const int r = (q - 4 * w) / 4, c = (q - 4 * w) & 3;
            ra = 2 + r;
            rb = c < 2 ? c : TH_J + c;
        }
    }
    auto inner = [&](int i, int j) { return i >= 1 && i < NE - 1 && j >= 1 && j < NE - 1; };
    auto distances = [&](int a, int b, long long fb) {
        const int i = i0 + a - 2, j = j0 + b - 2;
        if (!inner(i, j)) return;
        const long long mc = (t.metric_shared ? 0 : fb) + (long long)i * NE + j;
        const double g0 = t.metric[3 * mc], g1 = t.metric[3 * mc + 1], g2 = t.metric[3 * mc + 2];
#pragma unroll
        for (int k = 0; k < 4; k++) T.dist[k][a][b] = sqrt(g0 * DI[k] * DI[k] + 2.0 * g1 * DI[k] * DJ[k] + g2 * DJ[k] * DJ[k]);
    };
    for (int f = blockIdx.z * faces; f < (int)(blockIdx.z + 1) * faces; f++) {
        const long long fb = (long long)f * NE * NE;
        for (int q = threadIdx.x; q < (TH_I + 6) * (TH_J + 6); q += TH_THREADS) {
            const int a = q / (TH_J + 6), b = q - a * (TH_J + 6), i = i0 + a - 3, j = j0 + b - 3;
            double v = 0.0;
            int m = PGE_MASK_OUTSIDE;
            if (i >= 0 && i < NE && j >= 0 && j < NE) {
                const long long c = fb + (long long)i * NE + j;
                v = t.h[c] + t.s[c];
                m = t.mask ? t.mask[c] : PGE_MASK_ACTIVE;
                if (t.creep && v < t.base[c]) m = PGE_MASK_FROZEN;
            }
            T.surf[a][b] = v;
            if (MASKED) T.m[a][b] = (uint8_t)m;
        }
        if (!t.metric_shared || f == (int)blockIdx.z * faces) {
            distances(ta + 2, tb + 2, fb);
            if (threadIdx.x < TH_RING) distances(ra, rb, fb);
        }
        __syncthreads();
        // the flows of cell (a, b) to its neighbours, their scale (0: nothing moves) and which neighbours are active
        auto flows = [&](int a, int b, double (&o)[8], unsigned &act) {
            const int i = i0 + a - 2, j = j0 + b - 2;
            double sc = 0.0;
            act = 0;
            if (inner(i, j) && (!MASKED || T.m[a + 1][b + 1] == PGE_MASK_ACTIVE)) {
                const double talus =
                    t.hard ? (double)__fadd_rn(t.talus_soft, __fmul_rn(t.talus_diff, t.hard[fb + (long long)i * NE + j])) : 0.0;
                const double surf = T.surf[a + 1][b + 1];
                double S = 0.0, mx = 0.0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const double d = surf - T.surf[a + 1 + DI[k]][b + 1 + DJ[k]];
                    const double ex = d - talus * T.dist[k & 3][a][b];
                    o[k] = d <= 0.0 || ex <= 0.0 ? 0.0 : half_rate * ex;
                    if (MASKED && T.m[a + 1 + DI[k]][b + 1 + DJ[k]] != PGE_MASK_ACTIVE) continue;
                    act |= 1u << k;
                    S += o[k];
                    if (o[k] > mx) mx = o[k];
                }
                if (S > 0.0) {
                    sc = 1.0;
                    if (S > 2.0 * mx) sc = 2.0 * mx / S;
                    if (t.cap > 0.0 && S * sc > t.cap) sc = t.cap / S;
                }
            }
#pragma unroll
            for (int k = 0; k < 8; k++) T.sent[k][a][b] = sc > 0.0 ? sc * o[k] : 0.0;
            return sc;
        };
        double o[8];
        unsigned act;
        if (threadIdx.x < TH_RING) flows(ra, rb, o, act);
        const double sc_self = flows(ta + 2, tb + 2, o, act);
        __syncthreads();
        // what flows into cell (a, b) (in the frame of the flows)
        auto inflow_of = [&](int a, int b) {
            double inflow = 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++) inflow += T.sent[(k + 4) & 7][a + DI[k]][b + DJ[k]];
            return inflow;
        };
        for (int q = threadIdx.x; q < (TH_I + 2) * (TH_J + 2); q += TH_THREADS) {
            const int a = q / (TH_J + 2), b = q - a * (TH_J + 2);
            double rs = 1.0;
            if (inner(i0 + a - 1, j0 + b - 1)) {
                const double surf = T.surf[a + 2][b + 2];
                if (!(surf >= 0.0 || (MASKED && T.m[a + 2][b + 2] != PGE_MASK_ACTIVE))) {
                    const double inflow = inflow_of(a + 1, b + 1);
                    double room = -t.dep_floor - surf;
                    if (room < 0.0) room = 0.0;
                    if (inflow > room) rs = room / inflow;
                }
            }
            T.rscale[a][b] = rs;
        }
        __syncthreads();
        const int i = i0 + ta, j = j0 + tb;
        if (i < NE && j < NE) {
            const long long c = fb + (long long)i * NE + j;
            double h = t.h[c], s = t.s[c];
            if (inner(i, j) && (!MASKED || T.m[ta + 3][tb + 3] == PGE_MASK_ACTIVE)) {
                double out = 0.0;
                if (sc_self > 0.0) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        if (!MASKED || (act >> k & 1u)) out += sc_self * T.rscale[ta + 1 + DI[k]][tb + 1 + DJ[k]] * o[k];
                }
                const double inflow = inflow_of(ta + 2, tb + 2) * T.rscale[ta + 1][tb + 1];
                if (out > 0.0) {
                    if (s >= out) {
                        s -= out;
                    } else {
                        h -= out - s;
                        s = 0.0;
                    }
                }
                s = s + inflow;
            }
            t.new_h[c] = h;
            t.new_s[c] = s;
        }
        __syncthreads();  // the next face's surface goes where this one's was read
    }
}

__global__ void copy2_kernel(long long n, const double *a, const double *b, double *da, double *db)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        da[c] = a[c];
        db[c] = b[c];
    }
}

// the talus pass from the state into the scratch (2 * n doubles) and the creep pass back into the state
void thermal_on_scratch(const PgeGrid &g, PgeState &s, double *tb, long long n, double rate, double creep_rate, double cap,
                        float soft, float diff, double dep_floor, cudaStream_t st)
{
    ThermalArgs t;
    t.NE = g.N + 2 * g.H;
    t.metric = s.metric;
    t.metric_shared = g.metric_shared;
    t.talus_soft = soft;
    t.talus_diff = diff;
    t.mask = s.mask;
    t.base = s.base;
    t.dep_floor = dep_floor;
    t.cap = cap;
    t.h = s.height;
    t.s = s.sediment;
    t.hard = s.hardness;
    t.creep = 0;
    t.rate = rate;
    t.new_h = tb;
    t.new_s = tb + n;
    dim3 grid((t.NE + TH_J - 1) / TH_J, (t.NE + TH_I - 1) / TH_I, g.F);
    int faces = 1;
    if (grid.x * grid.y >= TH_FILL) {
        faces = g.F;
        grid.z = 1;
    }
    if (t.mask)
        thermal_tile_kernel<true><<<grid, TH_THREADS, 0, st>>>(t, faces);
    else
        thermal_tile_kernel<false><<<grid, TH_THREADS, 0, st>>>(t, faces);
    if (!(creep_rate > 0.0)) {
        copy2_kernel<<<grid_for(n), 256, 0, st>>>(n, tb, tb + n, s.height, s.sediment);
        return;
    }
    t.h = tb;
    t.s = tb + n;
    t.hard = nullptr;
    t.creep = 1;
    t.rate = creep_rate;
    t.new_h = s.height;
    t.new_s = s.sediment;
    thermal_tile_kernel<true><<<grid, TH_THREADS, 0, st>>>(t, faces);
}

void thermal(const PgeGrid &g, PgeState &s, const Layout &lay, void *ws, double rate, double creep_rate, double cap, float soft,
             float diff, double dep_floor, cudaStream_t st)
{
    thermal_on_scratch(g, s, ws_ptr<double>(ws, lay.thermal), lay.ncell, rate, creep_rate, cap, soft, diff, dep_floor, st);
}

struct UpliftValue {
    const double *u;
    double cap;
    int use_cap;
    __device__ __forceinline__ double operator()(const long long c) const
    {
        const double v = u[c];
        return use_cap && v > cap ? cap : v;
    }
};

struct InteriorActive {
    int NE, H, N;
    const uint8_t *mask;
    __device__ __forceinline__ bool operator()(const long long c) const
    {
        return interior(c, NE, H, N) && (!mask || mask[c] == PGE_MASK_ACTIVE);
    }
};

struct Positive {
    __device__ __forceinline__ bool operator()(const double x) const { return x > 0.0; }
};

// ---------------------------------------------------------------------------
// numpy's pairwise summation, so that a float64 sum the reference takes with
// numpy (ndarray.sum / mean of a contiguous float64 array) is reproduced bit for
// bit: n < 8 values are added one by one to 0; up to 128 values are added as
// eight running sums over the leading multiple of 8, combined as
// ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)), and the rest added one by
// one; a longer range is split at n2 = n/2 rounded down to a multiple of 8 and
// the two halves' sums added.  (numpy's pairwise_sum, the reduction loop of
// np.add; checked against np.sum on ranges of 1..5000 values of mixed
// magnitudes.)  The split depends on the count alone, so a node finds its own
// range by walking down from the root: nothing is planned or stored.  Eight
// lanes sum a leaf, a block folds its PW_BLOCK_NODES consecutive nodes, and one
// block folds the blocks.
// ---------------------------------------------------------------------------
constexpr int PW_LEAF = 128;
constexpr int PW_MAX_DEPTH = 20;  // nodes at most 2^20: a longer array's leaves are summed by one lane each
constexpr int PW_BLOCK_LOG = 7, PW_BLOCK_NODES = 1 << PW_BLOCK_LOG;
constexpr int PW_THREADS = 1024;

__device__ double pw_leaf(const double *a, long long n)
{
    if (n < 8) {
        double res = 0.0;
        for (long long i = 0; i < n; i++) res += a[i];
        return res;
    }
    double r0 = a[0], r1 = a[1], r2 = a[2], r3 = a[3], r4 = a[4], r5 = a[5], r6 = a[6], r7 = a[7];
    long long i = 8;
    for (; i < n - (n % 8); i += 8) {
        r0 += a[i];
        r1 += a[i + 1];
        r2 += a[i + 2];
        r3 += a[i + 3];
        r4 += a[i + 4];
        r5 += a[i + 5];
        r6 += a[i + 6];
        r7 += a[i + 7];
    }
    double res = ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7));
    for (; i < n; i++) res += a[i];
    return res;
}

__device__ __forceinline__ long long pw_split(long long n)
{
    const long long n2 = n / 2;
    return n2 - n2 % 8;
}

// the pairwise sum of a[0, n) by an explicit post-order walk (depth <= 40 for any n < 2^40)
__device__ double pw_sum(const double *a, long long n)
{
    if (n <= PW_LEAF) return pw_leaf(a, n);
    long long lo[40], len[40];
    double left[40];
    int stage[40];
    int sp = 0;
    lo[0] = 0;
    len[0] = n;
    stage[0] = 0;
    double v = 0.0;
    while (true) {
        const int t = sp;
        if (len[t] <= PW_LEAF || stage[t] == 2) {
            // a finished node: a leaf, or both halves done (v holds the right half)
            v = len[t] <= PW_LEAF ? pw_leaf(a + lo[t], len[t]) : left[t] + v;
            if (sp == 0) return v;
            sp--;
            if (stage[sp] == 1) {  // the left half just finished: keep it, descend into the right half
                left[sp] = v;
                const long long n2 = pw_split(len[sp]);
                stage[sp] = 2;
                sp++;
                lo[sp] = lo[sp - 1] + n2;
                len[sp] = len[sp - 1] - n2;
                stage[sp] = 0;
            }
            continue;
        }
        stage[t] = 1;  // descend into the left half
        sp++;
        lo[sp] = lo[t];
        len[sp] = pw_split(len[t]);
        stage[sp] = 0;
    }
}

// a node's sum, or that it lies below a leaf (there is nothing in it: the leaf stands at its first descendant)
struct PwSum {
    double sum;
    int there;
};
__device__ __forceinline__ PwSum pw_add(const PwSum &l, const PwSum &r) { return r.there ? PwSum{l.sum + r.sum, 1} : l; }

__global__ void __launch_bounds__(256) pw_leaf_kernel(const double *a, const long long *count, int depth, PwSum *part)
{
    __shared__ PwSum node[PW_BLOCK_NODES];
    const int lane8 = threadIdx.x & 7, group = threadIdx.x >> 3;
    const unsigned eight = 0xffu << (threadIdx.x & 24);
    const long long M = *count;
    for (int t = group; t < PW_BLOCK_NODES; t += 32) {
        const unsigned k = blockIdx.x * PW_BLOCK_NODES + t;
        long long lo = 0, n = M;
        bool there = k < 1u << depth;
        for (int l = depth - 1; l >= 0 && there; l--) {
            const unsigned right = k >> l & 1u;
            if (n <= PW_LEAF) {  // a leaf above: it stands at its first descendant
                there = (k & ((1u << (l + 1)) - 1u)) == 0;
                break;
            }
            const long long n2 = pw_split(n);
            lo += right ? n2 : 0;
            n = right ? n - n2 : n2;
        }
        double sum = 0.0;
        if (there && n > PW_LEAF) {
            if (lane8 == 0) sum = pw_sum(a + lo, n);
        } else if (there && n < 8) {
            if (lane8 == 0) sum = pw_leaf(a + lo, n);
        } else if (there) {
            const double *p = a + lo;
            const int m = (int)n - (int)n % 8;
            double r = p[lane8];
            for (int i = 8; i < m; i += 8) r += p[i + lane8];
            r += __shfl_xor_sync(eight, r, 1);  // (commutative: every lane has r0 + r1, then (r0 + r1) + (r2 + r3), ..)
            r += __shfl_xor_sync(eight, r, 2);
            r += __shfl_xor_sync(eight, r, 4);
            for (int i = m; i < (int)n; i++) r += p[i];
            sum = r;
        }
        if (lane8 == 0) node[t] = PwSum{sum, there};
    }
    __syncthreads();
    for (int w = PW_BLOCK_NODES / 2; w > 0; w >>= 1) {
        PwSum s;
        if ((int)threadIdx.x < w) s = pw_add(node[2 * threadIdx.x], node[2 * threadIdx.x + 1]);
        __syncthreads();
        if ((int)threadIdx.x < w) node[threadIdx.x] = s;
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = node[0];
}

// folds the blocks' sums (a power of two of them); out = the sum, or with mean_out the sum / count
__global__ void __launch_bounds__(PW_THREADS) pw_fold_kernel(PwSum *part, int n, const long long *count, double *out, int mean_out)
{
    for (int w = n / 2; w > 0; w >>= 1) {
        // (each round reads the places 2k, 2k + 1 and writes the place k: the rounds of one width go in order)
        for (int k0 = 0; k0 < w; k0 += blockDim.x) {
            const int k = k0 + threadIdx.x;
            PwSum s{0.0, 0};
            if (k < w) s = pw_add(part[2 * k], part[2 * k + 1]);
            __syncthreads();
            if (k < w) part[k] = s;
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        const long long M = *count;
        *out = mean_out ? (M > 0 ? part[0].sum / (double)M : 0.0) : part[0].sum;
    }
}

size_t pairwise_scratch_bytes() { return sizeof(PwSum) << (PW_MAX_DEPTH - PW_BLOCK_LOG); }

// sum (or mean) of a[0, *count), at most n_max values, in numpy's pairwise order, written to *out on the stream
void pairwise_sum(const double *a, const long long *count, long long n_max, void *scratch, double *out, int mean, cudaStream_t st)
{
    PwSum *part = static_cast<PwSum *>(scratch);
    // a range at depth l is at most n / 2^l + 16 long: deep enough that every node fits a leaf
    int depth = PW_BLOCK_LOG;
    while (depth < PW_MAX_DEPTH && (n_max >> depth) > PW_LEAF - 32) depth++;
    const int blocks = 1 << (depth - PW_BLOCK_LOG);
    pw_leaf_kernel<<<blocks, 256, 0, st>>>(a, count, depth, part);
    pw_fold_kernel<<<1, PW_THREADS, 0, st>>>(part, blocks, count, out, mean);
}

// ---------------------------------------------------------------------------
// uplift and the datum's order statistic
// ---------------------------------------------------------------------------
constexpr int RED_BLOCKS = 1024;  // the partial-result area of the workspace: scalars of the uplift and the select

__global__ void uplift_add_kernel(long long ncell, double *h, const double *u, const uint8_t *mask, double cap, int use_cap,
                                  const double *mean, double scale)
{
    const double m = mean ? *mean : 0.0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        if (mask && mask[c] != PGE_MASK_ACTIVE) continue;
        double v = u[c];
        if (use_cap && v > cap) v = cap;
        h[c] += scale * (v - m);
    }
}

void uplift(const PgeGrid &g, PgeState &s, const Layout &lay, void *ws, double cap, double scale, cudaStream_t st)
{
    // maps._applied_uplift (maps.py:1136-1147): the mean of the (capped) field over the interior active
    // cells, u[interior][active].mean() -- their values in cell order, summed in numpy's pairwise order
    const int NE = g.N + 2 * g.H;
    const int use_cap = cap >= 0.0;
    double *partial = ws_ptr<double>(ws, lay.partial);
    long long *pcount = reinterpret_cast<long long *>(partial + RED_BLOCKS);
    double *mean = partial + 2 * RED_BLOCKS;
    if (g.spherical) {
        double *vals = ws_ptr<double>(ws, lay.pwv);
        size_t tb = lay.cubtmp_bytes;
        const thrust::counting_iterator<long long> c0(0);
        cub::DeviceSelect::Flagged(ws_ptr<void>(ws, lay.cubtmp), tb,
                                   thrust::make_transform_iterator(c0, UpliftValue{s.uplift, cap, use_cap}),
                                   thrust::make_transform_iterator(c0, InteriorActive{NE, g.H, g.N, s.mask}), vals, pcount,
                                   (int)lay.ncell, st);
        pairwise_sum(vals, pcount, lay.ncell, ws_ptr<void>(ws, lay.pwnode), mean, 1, st);
    }
    uplift_add_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, s.height, s.uplift, s.mask, cap, use_cap,
                                                           g.spherical ? mean : nullptr, scale);
}

// ---------------------------------------------------------------------------
// datum: k-th smallest interior surface by a 6-pass radix select on the
// order-preserving 64-bit image of the float64 keys
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long okey(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double unokey(unsigned long long k)
{
    const unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)b);
}

// digits of 11 bits, the last of 9: six passes
constexpr int SEL_BITS = 11, SEL_BINS = 1 << SEL_BITS, SEL_THREADS = 512;
struct SelectState {
    unsigned long long prefix;  // digits found so far (high bits)
    long long k;                // rank still sought inside the prefix
    unsigned int done;          // blocks that have added their histogram
    unsigned int hist[SEL_BINS];
};

// one digit: every block adds its histogram of the keys inside the prefix, the last one finds the digit of the rank
// sought and clears the histogram for the next
__global__ void __launch_bounds__(SEL_THREADS) select_digit_kernel(long long ncell, int NE, int H, int N, const double *__restrict__ h,
                                                                   const double *__restrict__ s, SelectState *ss, int shift, int bits)
{
    __shared__ unsigned int sh[SEL_BINS];
    __shared__ bool last;
    for (int i = threadIdx.x; i < SEL_BINS; i += SEL_THREADS) sh[i] = 0;
    __syncthreads();
    const unsigned long long prefix = ss->prefix;
    const unsigned long long hmask = shift + bits >= 64 ? 0ull : (~0ull << (shift + bits));
    const unsigned digit = (1u << bits) - 1u;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        if (!interior(c, NE, H, N)) continue;
        const unsigned long long k = okey(h[c] + s[c]);
        if ((k & hmask) != (prefix & hmask)) continue;
        atomicAdd(&sh[(unsigned)(k >> shift) & digit], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < SEL_BINS; i += SEL_THREADS)
        if (sh[i]) atomicAdd(&ss->hist[i], sh[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&ss->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the digit: the first bin whose running count passes the rank
    typedef cub::BlockScan<long long, SEL_THREADS> Scan;
    __shared__ typename Scan::TempStorage tmp;
    constexpr int PER = SEL_BINS / SEL_THREADS;
    unsigned int n[PER];
    long long mine = 0;
    for (int q = 0; q < PER; q++) {
        n[q] = ((volatile unsigned int *)ss->hist)[threadIdx.x * PER + q];
        mine += n[q];
    }
    long long before;
    Scan(tmp).ExclusiveSum(mine, before);
    const long long k = ss->k;
    __syncthreads();  // every thread has read the rank
    long long at = before;
    for (int q = 0; q < PER; q++) {
        const int bin = threadIdx.x * PER + q;
        // (a rank beyond the keys takes the last digit)
        if ((k >= at && k < at + (long long)n[q]) || (bin == (int)digit && k >= at + (long long)n[q])) {
            ss->k = k - at;
            ss->prefix = prefix | (unsigned long long)bin << shift;
        }
        at += n[q];
        ss->hist[bin] = 0;
    }
    if (threadIdx.x == 0) ss->done = 0;
}

__global__ void select_init_kernel(SelectState *ss, long long k)
{
    for (int i = threadIdx.x; i < SEL_BINS; i += blockDim.x) ss->hist[i] = 0;
    if (threadIdx.x == 0) {
        ss->prefix = 0;
        ss->k = k;
        ss->done = 0;
    }
}

__global__ void datum_shift_kernel(long long ncell, double *h, double *base, const SelectState *ss, double level, int plus_one,
                                   double *shift_out)
{
    double q = unokey(ss->prefix);
    if (plus_one) q += 1.0;
    q -= level;
    if (blockIdx.x == 0 && threadIdx.x == 0) *shift_out = q;
    if (q == 0.0) return;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        h[c] -= q;
        if (base[c] < 0.0) base[c] -= q;
    }
}

void hold_datum(const PgeGrid &g, PgeState &s, const Layout &lay, void *ws, double land_fraction, double level,
                double *shift_dev, cudaStream_t st)
{
    const int NE = g.N + 2 * g.H;
    const long long M = (long long)g.F * g.N * g.N;
    long long n_land = (long long)llrint(land_fraction * (double)M);  // numpy round: half to even
    if (n_land < 0) n_land = 0;
    if (n_land > M) n_land = M;
    long long k;
    int plus_one = 0;
    if (n_land == 0) {
        k = M - 1;
        plus_one = 1;
    } else {
        k = M - n_land;
    }
    SelectState *ss = ws_ptr<SelectState>(ws, lay.partial + 4 * RED_BLOCKS * sizeof(double));
    select_init_kernel<<<1, 256, 0, st>>>(ss, k);
    for (int top = 64; top > 0;) {
        const int bits = top < SEL_BITS ? top : SEL_BITS;
        top -= bits;
        select_digit_kernel<<<grid_reduce(lay.ncell, SEL_THREADS), SEL_THREADS, 0, st>>>(lay.ncell, NE, g.H, g.N, s.height, s.sediment, ss,
                                                                                         top, bits);
    }
    datum_shift_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, s.height, s.base, ss, level, plus_one, shift_dev);
}

// ---------------------------------------------------------------------------
// halo gather
// ---------------------------------------------------------------------------
__global__ void halo_scalar_kernel(long long K, const int32_t *dst, const int32_t *src, const double *w, double *f)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K; k += (long long)gridDim.x * blockDim.x) {
        double acc = 0.0;
#pragma unroll
        for (int q = 0; q < 16; q++) acc += w[16 * k + q] * f[src[16 * k + q]];
        f[dst[k]] = acc;
    }
}

__global__ void halo_vector_kernel(long long K, const int32_t *dst, const int32_t *src, const double *w, const double *rot,
                                   double *f)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K; k += (long long)gridDim.x * blockDim.x) {
        double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
        for (int q = 0; q < 16; q++) {
            const long long sidx = src[16 * k + q];
            const double va = f[2 * sidx], vb = f[2 * sidx + 1];
            const double *R = rot + 4 * (16 * k + q);
            const double wq = w[16 * k + q];
            a0 += wq * (R[0] * va + R[1] * vb);
            a1 += wq * (R[2] * va + R[3] * vb);
        }
        f[2 * (long long)dst[k]] = a0;
        f[2 * (long long)dst[k] + 1] = a1;
    }
}

void halo_gather(const PgeHalo &h, double *field, int vector, cudaStream_t st)
{
    if (h.K <= 0) return;
    if (vector)
        halo_vector_kernel<<<grid_for(h.K), 256, 0, st>>>(h.K, h.dst, h.src, h.w, h.rot, field);
    else
        halo_scalar_kernel<<<grid_for(h.K), 256, 0, st>>>(h.K, h.dst, h.src, h.w, field);
}

// ---------------------------------------------------------------------------
// spawns
// ---------------------------------------------------------------------------
// a float32 x > 0 is m * 2^(e - 150) with m a 24-bit integer (e the biased exponent, 1 for subnormals)
__device__ __forceinline__ void f32_parts(float x, long long &m, int &e)
{
    const unsigned b = __float_as_uint(x);
    const unsigned E = (b >> 23) & 0xffu;
    m = (long long)((b & 0x7fffffu) | (E ? 0x800000u : 0u));
    e = E ? (int)E : 1;
}

__global__ void spawn_weight_kernel(long long ncell, int NE, int H, int N, const double *h, const double *s, const double *base,
                                    const uint8_t *mask, const float *precip, double *w, long long *lastc, long long *erange)
{
    long long last = -1;
    int emin = 1 << 20, emax = -1;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        const bool ok = interior(c, NE, H, N) && (!mask || mask[c] == PGE_MASK_ACTIVE) && (h[c] + s[c] >= base[c]) && precip[c] > 0.0f;
        w[c] = ok ? (double)precip[c] : 0.0;
        if (ok) {
            if (c > last) last = c;
            long long m;
            int e;
            f32_parts(precip[c], m, e);
            emin = e < emin ? e : emin;
            emax = e > emax ? e : emax;
        }
    }
    // the block's extremes first, then one atomic each a block
    typedef cub::BlockReduce<long long, 256> BR;
    typedef cub::BlockReduce<int, 256> BRi;
    __shared__ typename BR::TempStorage t0;
    __shared__ typename BRi::TempStorage t1, t2;
    last = BR(t0).Reduce(last, cub::Max());
    emin = BRi(t1).Reduce(emin, cub::Min());
    emax = BRi(t2).Reduce(emax, cub::Max());
    if (threadIdx.x == 0) {
        if (last >= 0) atomicMax(reinterpret_cast<unsigned long long *>(lastc), (unsigned long long)last);
        if (emax >= 0) {
            atomicMin(erange, (long long)emin);
            atomicMax(erange + 1, (long long)emax);
        }
    }
}

// The fixed-point unit of the weights' integer scan: 2^(base - 150), the smallest weight's
// last bit (so every weight is an integer of it and every prefix sum exact) unless the spread
// of exponents would overflow 62 bits over ncell weights.
__device__ __forceinline__ int spawn_fx_base(const long long *erange, long long ncell)
{
    int lg = 0;
    while ((1LL << lg) < ncell) lg++;
    const int emin = (int)erange[0], emax = (int)erange[1];
    const int need = emax + 24 + lg - 62;
    return emin > need ? emin : need;
}

__global__ void spawn_quant_kernel(long long ncell, const double *w, const long long *erange, long long *wq)
{
    const int base = spawn_fx_base(erange, ncell);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x) {
        long long q = 0;
        if (w[c] > 0.0) {
            long long m;
            int e;
            f32_parts((float)w[c], m, e);
            const int sh = e - base;
            q = sh >= 0 ? m << sh : (sh > -40 ? (m + (1LL << (-sh - 1))) >> (-sh) : 0);
        }
        wq[c] = q;
    }
}

// the integer prefix sums back to float64, in place
__global__ void spawn_cdf_kernel(long long ncell, const long long *erange, double *cdf)
{
    const int base = spawn_fx_base(erange, ncell);
    long long *S = reinterpret_cast<long long *>(cdf);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x)
        cdf[c] = ldexp((double)S[c], base - 150);
}

__global__ void spawn_count_kernel(long long ncell, const double *w, long long *count)
{
    long long n = 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x)
        n += w[c] > 0.0;
    typedef cub::BlockReduce<long long, 256> BR;
    __shared__ typename BR::TempStorage tmp;
    n = BR(tmp).Sum(n);
    if (threadIdx.x == 0 && n) atomicAdd(reinterpret_cast<unsigned long long *>(count), (unsigned long long)n);
}

__global__ void spawn_search_kernel(long long ncell, int NE, int H, const double *cdf, const long long *lastc, const double *u,
                                    const double *off, long long P, int32_t *face, double *x, double *y, double *sed, double *dir)
{
    const double total = cdf[ncell - 1];
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
        const double target = u[p] * total;
        // first index with cdf > target (the reference walks its compacted cdf the same way)
        long long lo = 0, hi = ncell;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (cdf[mid] <= target) lo = mid + 1;
            else hi = mid;
        }
        long long c = lo < ncell ? lo : *lastc;
        const long long fa = c / ((long long)NE * NE);
        const long long rem = c - fa * NE * NE;
        const long long ei = rem / NE, ej = rem - ei * NE;
        face[p] = (int32_t)fa;
        x[p] = (double)(ei - H) + off[2 * p];
        y[p] = (double)(ej - H) + off[2 * p + 1];
        sed[p] = 0.0;
        dir[p] = 0.0;
    }
}

struct PendFlag {
    const double *pending;
    __device__ __forceinline__ bool operator()(const long long c) const { return pending[c] > 0.0; }
};

__global__ void pending_emit_kernel(const long long *idx, const long long *count, int NE, int H, double *pending, int32_t *face,
                                    double *x, double *y, double *sed, long long *released_fx)
{
    const long long n = *count;
    long long rel = 0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long c = idx[k];
        const long long fa = c / ((long long)NE * NE);
        const long long rem = c - fa * NE * NE;
        const long long ei = rem / NE, ej = rem - ei * NE;
        face[k] = (int32_t)fa;
        x[k] = (double)(ei - H) + 0.5;
        y[k] = (double)(ej - H) + 0.5;
        sed[k] = pending[c];
        rel += __double2ll_rn(pending[c] * FX_MASS);
        pending[c] = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) rel += __shfl_down_sync(0xffffffffu, rel, o);
    if ((threadIdx.x & 31) == 0 && rel) atomicAdd(reinterpret_cast<unsigned long long *>(released_fx), (unsigned long long)rel);
}

size_t cub_temp_bytes(int64_t ncell, int64_t max_droplets)
{
    size_t a = 0, b = 0, c = 0;
    cub::DeviceScan::InclusiveSum(nullptr, a, (double *)nullptr, (double *)nullptr, (int)ncell);
    cub::DeviceRadixSort::SortKeys(nullptr, b, (double *)nullptr, (double *)nullptr, (int)(max_droplets > 0 ? max_droplets : 1));
    cub::DeviceSelect::If(nullptr, c, thrust::counting_iterator<long long>(0), (long long *)nullptr, (long long *)nullptr,
                          (int)ncell, PendFlag{nullptr});
    size_t d = 0, f = 0, h = 0;
    cub::DeviceScan::InclusiveSum(nullptr, d, (long long *)nullptr, (long long *)nullptr, (int)ncell);
    cub::DeviceSelect::If(nullptr, f, (double *)nullptr, (double *)nullptr, (long long *)nullptr, (int)ncell, Positive{});
    cub::DeviceSelect::Flagged(nullptr, h, thrust::make_transform_iterator(thrust::counting_iterator<long long>(0), UpliftValue{}),
                               thrust::make_transform_iterator(thrust::counting_iterator<long long>(0), InteriorActive{}),
                               (double *)nullptr, (long long *)nullptr, (int)ncell);
    size_t m = a > b ? a : b;
    m = m > c ? m : c;
    m = m > d ? m : d;
    m = m > f ? m : f;
    return m > h ? m : h;
}

cudaError_t spawn_rain(const PgeGrid &g, const PgeState &s, const Layout &lay, void *ws, const double *u, const double *off,
                       long long P, PgeSpawns &sp, double *total_dev, long long *nspawn_dev, cudaStream_t st)
{
    // maps.spawn_weights / spawn_particles (maps.py:793-833): w = precip on spawnable cells, their
    // cumulative sum (np.cumsum: sequential), total = w.sum() (numpy's pairwise order) and the inverse
    // CDF of the sorted uniforms (particle.spawn_cells).  The cumulative sum is an integer scan of the
    // weights in fixed point (their float32 bits), so it is order-free and equals the sequential float64
    // sum bit for bit whenever that sum is exact -- every prefix below 2^53 units of the smallest
    // weight's last bit (any float32 precip of 0.1 .. 3 over 6.3 M cells, or uniform rain).
    const int NE = g.N + 2 * g.H;
    double *w = ws_ptr<double>(ws, lay.cdf);
    double *cdf = w + lay.ncell;
    double *keys = ws_ptr<double>(ws, lay.sortkeys);
    long long *ctr = ws_ptr<long long>(ws, lay.counters);
    long long *lastc = ctr + 2, *erange = ctr + 24, *nsel = ctr + 26;  // slots 4 (the pass mode), 8, 12.. are taken
    long long *wq = ws_ptr<long long>(ws, lay.pwv);
    cudaError_t e = cudaMemsetAsync(lastc, 0, sizeof(long long), st);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(erange, 0x7f, sizeof(long long), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(erange + 1, 0, sizeof(long long), st)) != cudaSuccess) return e;
    if (nspawn_dev && (e = cudaMemsetAsync(nspawn_dev, 0, sizeof(long long), st)) != cudaSuccess) return e;
    spawn_weight_kernel<<<grid_reduce(lay.ncell), 256, 0, st>>>(lay.ncell, NE, g.H, g.N, s.height, s.sediment, s.base, s.mask,
                                                             s.precip, w, lastc, erange);
    if (nspawn_dev) spawn_count_kernel<<<grid_reduce(lay.ncell), 256, 0, st>>>(lay.ncell, w, nspawn_dev);
    spawn_quant_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, w, erange, wq);
    size_t tb = lay.cubtmp_bytes;
    e = cub::DeviceScan::InclusiveSum(ws_ptr<void>(ws, lay.cubtmp), tb, wq, reinterpret_cast<long long *>(cdf), (int)lay.ncell, st);
    if (e != cudaSuccess) return e;
    spawn_cdf_kernel<<<grid_for(lay.ncell), 256, 0, st>>>(lay.ncell, erange, cdf);
    // the total weight in numpy's order: the spawnable weights compacted in cell order, summed pairwise
    double *wc = ws_ptr<double>(ws, lay.pwv);
    tb = lay.cubtmp_bytes;
    e = cub::DeviceSelect::If(ws_ptr<void>(ws, lay.cubtmp), tb, w, wc, nsel, (int)lay.ncell, Positive{}, st);
    if (e != cudaSuccess) return e;
    if (total_dev) pairwise_sum(wc, nsel, lay.ncell, ws_ptr<void>(ws, lay.pwnode), total_dev, 0, st);
    tb = lay.cubtmp_bytes;
    e = cub::DeviceRadixSort::SortKeys(ws_ptr<void>(ws, lay.cubtmp), tb, u, keys, (int)P, 0, 64, st);
    if (e != cudaSuccess) return e;
    spawn_search_kernel<<<grid_for(P), 256, 0, st>>>(lay.ncell, NE, g.H, cdf, lastc, keys, off, P, sp.face, sp.x, sp.y, sp.sed,
                                                     sp.dir);
    return cudaPeekAtLastError();
}

cudaError_t count_pending(const PgeGrid &g, const PgeState &s, const Layout &lay, void *ws, long long *count_dev, cudaStream_t st)
{
    long long *idx = ws_ptr<long long>(ws, lay.flags);
    long long *cnt = ws_ptr<long long>(ws, lay.counters) + 3;
    size_t tb = lay.cubtmp_bytes;
    cudaError_t e = cub::DeviceSelect::If(ws_ptr<void>(ws, lay.cubtmp), tb, thrust::counting_iterator<long long>(0), idx, cnt,
                                          (int)lay.ncell, PendFlag{s.pending}, st);
    if (e != cudaSuccess) return e;
    if (count_dev) e = cudaMemcpyAsync(count_dev, cnt, sizeof(long long), cudaMemcpyDeviceToDevice, st);
    return e;
}

cudaError_t collect_pending(const PgeGrid &g, PgeState &s, const Layout &lay, void *ws, PgeSpawns &sp, long long offset,
                            PgeStats *stats, cudaStream_t st)
{
    const int NE = g.N + 2 * g.H;
    long long *idx = ws_ptr<long long>(ws, lay.flags);
    const long long *count_dev = ws_ptr<long long>(ws, lay.counters) + 3;
    pending_emit_kernel<<<grid_for(lay.ncell / 64 + 1), 256, 0, st>>>(idx, count_dev, NE, g.H, s.pending, sp.face + offset,
                                                                     sp.x + offset, sp.y + offset, sp.sed + offset,
                                                                     reinterpret_cast<long long *>(&stats->released_fx));
    return cudaPeekAtLastError();
}

// ---------------------------------------------------------------------------
// soillib's pit-free erosion cap (particle.py:1046-1076): per active cell, k * |Godunov downhill
// gradient| of the surface, each axis the steeper of its two one-sided downhill differences
// (exit_slope off the array); float64 in the reference's operation order (no FMA in this file)
// ---------------------------------------------------------------------------
__global__ void slope_erode_cap_kernel(int F, int NE, const double *__restrict__ height, const double *__restrict__ sediment,
                                       const uint8_t *__restrict__ mask, double k, double exit_slope, double *__restrict__ out)
{
    const long long n = (long long)F * NE * NE;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        if (mask && mask[c] != PGE_MASK_ACTIVE) {
            out[c] = 0.0;
            continue;
        }
        const long long r = c % ((long long)NE * NE);
        const int i = (int)(r / NE), j = (int)(r - (long long)i * NE);
        const double h = height[c] + sediment[c];
        const double gxn = i == 0 ? exit_slope : h - (height[c - NE] + sediment[c - NE]);
        const double gxp = i == NE - 1 ? exit_slope : h - (height[c + NE] + sediment[c + NE]);
        const double gyn = j == 0 ? exit_slope : h - (height[c - 1] + sediment[c - 1]);
        const double gyp = j == NE - 1 ? exit_slope : h - (height[c + 1] + sediment[c + 1]);
        double gx = gxn > gxp ? gxn : gxp;
        double gy = gyn > gyp ? gyn : gyp;
        if (gx < 0.0) gx = 0.0;
        if (gy < 0.0) gy = 0.0;
        out[c] = k * sqrt(gx * gx + gy * gy);
    }
}

void slope_erode_cap(const PgeGrid &g, const PgeState &s, double k, double exit_slope, double *out, cudaStream_t st)
{
    const int NE = g.N + 2 * g.H;
    slope_erode_cap_kernel<<<grid_for((long long)g.F * NE * NE), 256, 0, st>>>(g.F, NE, s.height, s.sediment, s.mask, k, exit_slope,
                                                                             out);
}

// ---------------------------------------------------------------------------
// the isostasy smoother (maps.py:1331-1410): one explicit step of the metric-aware
// Laplace-Beltrami diffusion, FaceField.laplacian (field.py:179-188, 372-404) in flux form,
// (1/sqrt g) d_a(sqrt g g^ab d_b f), at extended indices 1..NE-2 of every face (0 on the outer
// ring), per m^2 and rounded to float32 as the reference's field is; then
//   out = a * in + (kappa * lap) * cell^2       (a = 1: a smoothing step; a = 0, kappa = 1: the
//                                                  Laplacian in cell units, for the step bound)
// float64 in the reference's operation order (no FMA in this file)
// ---------------------------------------------------------------------------
// A thread takes SM_ROWS cells of its column on SM_FACES faces: the metric is the same on every face, so the edges'
// coefficients (four means of strided float32 tables, half the reads) are made once for all of them.  Bound by the
// latency of its loads at the occupancy its registers leave (ncu: float64 pipe 34 %, L1 30 %).  N_c = 725, one step:
// a cell a thread 46.4 us; rows x faces 1 x 1 43, 1 x 3 33, 1 x 6 29.0, 2 x 6 34, 4 x 2 59; the next face's cells read
// ahead 29.3.
constexpr int SM_X = 32, SM_Y = 8, SM_ROWS = 1, SM_FACES = 6;
struct SmoothEdge {
    double sv, g, x;  // mean sqrt(g), mean metric across the edge, half the mean mixed metric
};
__global__ void __launch_bounds__(SM_X *SM_Y) smooth_step_kernel(int F, int NE, const double *__restrict__ d, const float *__restrict__ ginv,
                                                                 const float *__restrict__ sq, double c2, double kappa, int keep,
                                                                 double *__restrict__ out)
{
    const int j = blockIdx.x * SM_X + threadIdx.x, i0 = (blockIdx.y * SM_Y + threadIdx.y) * SM_ROWS;
    if (j >= NE || i0 >= NE) return;
    const int f0 = blockIdx.z * SM_FACES;
    const long long plane = (long long)NE * NE;
    const bool inner_j = j >= 1 && j <= NE - 2;
    SmoothEdge ei[SM_ROWS + 1], ep[SM_ROWS], em[SM_ROWS];  // to the row above each row (and below the last), to j + 1, to j - 1
    double s_c[SM_ROWS];
    if (inner_j) {
        auto edge = [&](int a, int b, int k) {  // between the cells at flat places a and b, along axis k / 2
            return SmoothEdge{0.5 * ((double)sq[a] + (double)sq[b]), 0.5 * ((double)ginv[3 * a + k] + (double)ginv[3 * b + k]),
                              0.5 * ((double)ginv[3 * a + 1] + (double)ginv[3 * b + 1]) * 0.5};
        };
#pragma unroll
        for (int r = 0; r <= SM_ROWS; r++) {
            const int i = i0 + r, at = i * NE + j;
            if (i >= 1 && i <= NE - 1) ei[r] = edge(at, at - NE, 0);
            if (r < SM_ROWS && i >= 1 && i <= NE - 2) {
                s_c[r] = (double)sq[at];
                ep[r] = edge(at, at + 1, 2);
                em[r] = edge(at, at - 1, 2);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < SM_FACES; q++) {
        if (f0 + q >= F) break;
        const double *df = d + (f0 + q) * plane;
        double *of = out + (f0 + q) * plane;
        double v[SM_ROWS + 2][3];
#pragma unroll
        for (int r = 0; r < SM_ROWS + 2; r++) {
            const int i = i0 + r - 1;
            const bool in = i >= 0 && i < NE;
            const double *p = df + (long long)i * NE + j;
            v[r][0] = in && inner_j ? p[-1] : 0.0;
            v[r][1] = in ? p[0] : 0.0;
            v[r][2] = in && inner_j ? p[1] : 0.0;
        }
        // the flux between rows r - 1 and r of v
        auto flux_i = [&](const SmoothEdge &e, int r) {
            const double fl = 0.5 * (v[r - 1][2] - v[r - 1][0]), fh = 0.5 * (v[r][2] - v[r][0]);
            return e.sv * (e.g * (v[r][1] - v[r - 1][1]) + e.x * (fl + fh));
        };
#pragma unroll
        for (int r = 0; r < SM_ROWS; r++) {
            const int i = i0 + r;
            if (i >= NE) break;
            double lap64 = 0.0;  // (0 on the outer ring)
            if (inner_j && i >= 1 && i <= NE - 2) {
                const double Fi_m = flux_i(ei[r], r + 1), Fi_p = flux_i(ei[r + 1], r + 2);
                const double fi_m = 0.5 * (v[r + 2][0] - v[r][0]), fi_c = 0.5 * (v[r + 2][1] - v[r][1]), fi_p = 0.5 * (v[r + 2][2] - v[r][2]);
                const double Fj_p = ep[r].sv * (ep[r].g * (v[r + 1][2] - v[r + 1][1]) + ep[r].x * (fi_c + fi_p));
                const double Fj_m = em[r].sv * (em[r].g * (v[r + 1][1] - v[r + 1][0]) + em[r].x * (fi_c + fi_m));
                const double lap = (Fi_p - Fi_m + Fj_p - Fj_m) / s_c[r];
                lap64 = (double)(float)(lap / c2);  // per m^2, a float32 field
            }
            const double upd = kappa * lap64 * c2;
            of[(long long)i * NE + j] = keep ? v[r + 1][1] + upd : upd;
        }
    }
}

void smooth_step(const PgeGrid &g, const double *in, const float *metric_inv, const float *sqrt_det, double kappa, int keep,
                 double cell_m, double *out, cudaStream_t st)
{
    const int NE = g.N + 2 * g.H;
    const double c2 = cell_m * cell_m;
    const dim3 grid((NE + SM_X - 1) / SM_X, (NE + SM_Y * SM_ROWS - 1) / (SM_Y * SM_ROWS), (g.F + SM_FACES - 1) / SM_FACES);
    smooth_step_kernel<<<grid, dim3(SM_X, SM_Y), 0, st>>>(g.F, NE, in, metric_inv, sqrt_det, c2, kappa, keep, out);
}

}  // namespace pge

namespace pge {

// ---------------------------------------------------------------------------
// routing surface: the epsilon-filled surface of a priority flood
// (globe/erosion/route.py:31-125), as the fixed point of a relaxation.  A cell
// reached from the seeds takes max(its surface, lowest reaching neighbour + eps);
// a heap flood reaches every cell first from its lowest reaching neighbour, so
// the fixed point is the heap flood's result value for value.  Neighbours are
// pushed to along the owner table (the reference's direction: from a popped cell
// to owner[its D8 neighbour]); values live as the datum select's order-preserving
// uint64 keys (okey) so a plain atomicMin keeps the lowest.
// ---------------------------------------------------------------------------
namespace {
enum : unsigned char { RF_EXCLUDED = 0, RF_FREE = 1, RF_SEED = 2 };
constexpr unsigned long long RF_UNREACHED = 0xFFFFFFFFFFFFFFFFull;
__constant__ int kRouteD8[8][2] = {{1, 0}, {1, 1}, {0, 1}, {-1, 1}, {-1, 0}, {-1, -1}, {0, -1}, {1, -1}};

}  // namespace

__global__ void route_init_kernel(int F, int NE, int H, int N, const double *__restrict__ h, const double *__restrict__ s,
                                  const double *__restrict__ base, const uint8_t *__restrict__ mask, const int32_t *__restrict__ owner,
                                  unsigned long long *key, unsigned char *state)
{
    const unsigned total = (unsigned)F * NE * NE;
    for (unsigned u = blockIdx.x * blockDim.x + threadIdx.x; u < total; u += gridDim.x * blockDim.x) {
        const int c = (int)u, r = c / NE, ej = c - r * NE, ei = r % NE;
        const double sv = h[c] + s[c];
        const bool outside = mask && mask[c] == PGE_MASK_OUTSIDE;
        if (outside || ei == 0 || ej == 0 || ei == NE - 1 || ej == NE - 1) {
            state[c] = RF_EXCLUDED;
            key[c] = okey(sv);
            continue;
        }
        bool seed = false;
        if (ei >= H && ei < H + N && ej >= H && ej < H + N) {
            seed = sv < 0.0 && sv <= base[c];
            // a neighbour outside the mask, or none that is real (a window's edge): only beside the halo without a mask
            const bool rim = mask || ei == H || ei == H + N - 1 || ej == H || ej == H + N - 1;
            for (int k = 0; k < 8 && rim && !seed; k++) {
                const int n = owner[c + kRouteD8[k][0] * NE + kRouteD8[k][1]];
                if (mask && mask[n] == PGE_MASK_OUTSIDE) {
                    seed = true;
                    break;
                }
                const int nr = n / NE, nej = n - nr * NE, nei = nr % NE;
                if (nei < H || nei >= H + N || nej < H || nej >= H + N) seed = true;
            }
        }
        state[c] = seed ? RF_SEED : RF_FREE;
        key[c] = seed ? okey(sv) : RF_UNREACHED;
    }
}

// One sweep of the relaxation, a tile a block: every active tile is relaxed to its own fixed point in shared memory
// (a cell takes what its lowest neighbour gives it), written back, and the tiles that its changed cells can lower
// are made active for the next sweep.  Within a face a cell's neighbours push to it what it pulls here; across a
// cube edge (the neighbour is a halo cell, owned by an interior cell of another face) the push goes to the owner.
// The values only ever fall, to the one fixed point, so neither the order nor a stale neighbour changes the result.
//
// Bound by the relaxations inside the tiles.  N_c = 1024, evolved world: sweeps of every cell from HBM, one cell
// further a sweep, 384 x 112 us; tiles, 16 sweeps of what is active, 66 us each.
constexpr int RT = 32;         // tile edge
constexpr int RT_STRIP = 4;    // cells a thread, one above the other
constexpr int RT_ROUNDS = 2;   // relaxations between two looks at whether the tile still changes
__global__ void __launch_bounds__(RT *RT / RT_STRIP) route_tile_kernel(int NE, int H, int tiles, const double *__restrict__ h,
                                                                       const double *__restrict__ s, const int32_t *__restrict__ owner,
                                                                       double eps, unsigned long long *key,
                                                                       const unsigned char *__restrict__ state, int first, int *active,
                                                                       int *next, unsigned long long *changed)
{
    __shared__ unsigned long long sk[RT + 2][RT + 2];
    const int tile = blockIdx.x;
    if (!__syncthreads_or(first || active[tile])) return;  // (one look for the whole block: the flag is cleared below)
    const int f = tile / (tiles * tiles), tr = tile - f * tiles * tiles, ti = tr / tiles, tj = tr - ti * tiles;
    const int fb = f * NE * NE, i0 = ti * RT, j0 = tj * RT;
    const int tx = threadIdx.x % RT, ty = threadIdx.x / RT;
    const volatile unsigned long long *vkey = key;
    // a cell that takes part: not excluded, and its own owner (a halo cell of the sphere only stands for another)
    for (int q = threadIdx.x; q < (RT + 2) * (RT + 2); q += blockDim.x) {
        const int a = q / (RT + 2), b = q - a * (RT + 2), i = i0 + a - 1, j = j0 + b - 1;
        unsigned long long k = RF_UNREACHED;
        if (i >= 0 && i < NE && j >= 0 && j < NE) {
            const int c = fb + i * NE + j;
            if (state[c] != RF_EXCLUDED && owner[c] == c) k = vkey[c];
        }
        sk[a][b] = k;
    }
    if (threadIdx.x == 0 && !first) active[tile] = 0;
    double surf[RT_STRIP];
    unsigned long long was[RT_STRIP];
    bool free_[RT_STRIP], in[RT_STRIP];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RT_STRIP; r++) {
        const int i = i0 + ty * RT_STRIP + r, j = j0 + tx;
        in[r] = i < NE && j < NE;
        free_[r] = false;
        surf[r] = 0.0;
        was[r] = sk[ty * RT_STRIP + r + 1][tx + 1];
        if (in[r]) {
            const int c = fb + i * NE + j;
            in[r] = owner[c] == c && state[c] != RF_EXCLUDED;
            free_[r] = in[r] && state[c] == RF_FREE;
            surf[r] = h[c] + s[c];
        }
    }
    volatile unsigned long long(*vk)[RT + 2] = sk;
    bool any = true;
    while (any) {
        bool mine = false;
#pragma unroll
        for (int t = 0; t < 2 * RT_ROUNDS; t++) {
#pragma unroll
            for (int q = 0; q < RT_STRIP; q++) {
                const int r = t & 1 ? RT_STRIP - 1 - q : q;  // down the strip, then up
                if (!free_[r]) continue;
                const int a = ty * RT_STRIP + r + 1, b = tx + 1;
                unsigned long long m = vk[a - 1][b - 1];
                m = min(m, vk[a - 1][b]);
                m = min(m, vk[a - 1][b + 1]);
                m = min(m, vk[a][b - 1]);
                m = min(m, vk[a][b + 1]);
                m = min(m, vk[a + 1][b - 1]);
                m = min(m, vk[a + 1][b]);
                m = min(m, vk[a + 1][b + 1]);
                if (m == RF_UNREACHED) continue;
                const double v = unokey(m) + eps;
                const unsigned long long kn = okey(surf[r] > v ? surf[r] : v);
                if (kn < vk[a][b]) {
                    vk[a][b] = kn;
                    mine = true;
                }
            }
        }
        any = __syncthreads_or(mine);
    }
    // write back, push across the cube edges, and wake the tiles whose cells this tile's rim can still lower (whoever
    // lowered the rim: this tile, or a push from another face since it last ran)
    bool woke = false;
#pragma unroll
    for (int r = 0; r < RT_STRIP; r++) {
        if (!in[r]) continue;
        const int a = ty * RT_STRIP + r, b = tx, i = i0 + a, j = j0 + b, c = fb + i * NE + j;
        const unsigned long long k = sk[a + 1][b + 1];
        if (k == RF_UNREACHED) continue;
        if (k < was[r]) atomicMin(key + c, k);
        const bool rim = a == 0 || a == RT - 1 || b == 0 || b == RT - 1 || i == H || i == NE - H - 1 || j == H || j == NE - H - 1;
        if (!rim) continue;
        const double v = unokey(k) + eps;
        for (int d = 0; d < 8; d++) {
            const int di = kRouteD8[d][0], dj = kRouteD8[d][1], nc = c + di * NE + dj;  // (excluded cells ring the array)
            const int n = owner[nc];
            int nt;  // the neighbour's tile
            if (n == nc) {
                nt = (f * tiles + (i + di) / RT) * tiles + (j + dj) / RT;
                if (nt == tile) continue;
            } else {
                const int nf = n / (NE * NE), nr = n - nf * NE * NE;
                nt = (nf * tiles + nr / NE / RT) * tiles + nr % NE / RT;
            }
            if (state[n] != RF_FREE) continue;
            const double sn = h[n] + s[n];
            const unsigned long long kn = okey(sn > v ? sn : v);
            if (kn < vkey[n] && (n == nc || atomicMin(key + n, kn) > kn)) {
                next[nt] = 1;
                woke = true;
            }
        }
    }
    if (__syncthreads_or(woke) && threadIdx.x == 0) *changed = 1ull;
}

__global__ void route_final_kernel(long long total, const double *__restrict__ h, const double *__restrict__ s,
                                   const unsigned long long *__restrict__ key, const unsigned char *__restrict__ state, double *route)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < total; c += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = key[c];
        route[c] = (state[c] == RF_EXCLUDED || k == RF_UNREACHED) ? h[c] + s[c] : unokey(k);
    }
}

cudaError_t route_flood(const PgeGrid &g, const PgeState &st, const int32_t *owner, double eps, double *route, const Layout &lay,
                        void *ws, long long max_sweeps, long long *sweeps_out, cudaStream_t s)
{
    const int NE = g.N + 2 * g.H;
    const long long n = lay.ncell;
    unsigned long long *key = ws_ptr<unsigned long long>(ws, lay.cdf);
    unsigned char *state = ws_ptr<unsigned char>(ws, lay.flags);
    unsigned long long *changed = ws_ptr<unsigned long long>(ws, lay.counters) + 8;
    const int tiles = (NE + RT - 1) / RT, nt = g.F * tiles * tiles;
    int *active = reinterpret_cast<int *>(state + (n + 7) / 8 * 8);  // two flags a tile, in the 7 bytes a cell left here
    route_init_kernel<<<grid_for(n), 256, 0, s>>>(g.F, NE, g.H, g.N, st.height, st.sediment, st.base, st.mask, owner, key, state);
    cudaError_t e = cudaMemsetAsync(active, 0, 2 * sizeof(int) * nt, s);
    if (e != cudaSuccess) return e;
    unsigned long long host_changed = 1;
    long long sweeps = 0;
    const int batch = 8;  // sweeps between convergence checks (the check synchronises the stream)
    while (host_changed && sweeps < max_sweeps) {
        for (int k = 0; k < batch; k++) {
            // (the last sweep of the batch says whether any tile is left to relax)
            if ((e = cudaMemsetAsync(changed, 0, 8, s)) != cudaSuccess) return e;
            const long long w = sweeps + k;
            route_tile_kernel<<<nt, RT * RT / RT_STRIP, 0, s>>>(NE, g.H, tiles, st.height, st.sediment, owner, eps, key, state, w == 0,
                                                                active + (w & 1) * nt, active + ((w + 1) & 1) * nt, changed);
        }
        sweeps += batch;
        if ((e = cudaMemcpyAsync(&host_changed, changed, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    }
    if (sweeps_out) *sweeps_out = host_changed ? -sweeps : sweeps;
    route_final_kernel<<<grid_for(n), 256, 0, s>>>(n, st.height, st.sediment, key, state, route);
    return cudaPeekAtLastError();
}

// ---------------------------------------------------------------------------
// sea mask: the base level (maps.py:360-420, hydro/run.py:64-83).  Interior
// cells under the waterline (float32 surface < 0) are joined into
// 8-connected components along the owner table (labels: the component's
// lowest cell id, by one pass of unions; propagating labels cell by cell took
// 256 sweeps of 194 us for the oceans of N_c = 1024); a component
// is open ocean when its area reaches min_area, and the largest always is;
// the others are closed basins, whose cells take the basin's lowest surface.
// ---------------------------------------------------------------------------
namespace {
// the interior cell that owns neighbour k of interior cell c, or -1 where the owner table names a halo cell (a grid
// too small for its halo's sources)
__device__ __forceinline__ int sea_nb(const int32_t *owner, int c, int k, int N, int H, int NE)
{
    const int row = c / N, j = c - row * N, f = row / N, i = row - f * N;
    const int o = owner[(f * NE + i + H + kRouteD8[k][0]) * NE + j + H + kRouteD8[k][1]];
    const int orow = o / NE, oj = o - orow * NE - H, of = orow / NE, oi = orow - of * NE - H;
    return oi < 0 || oi >= N || oj < 0 || oj >= N ? -1 : (of * N + oi) * N + oj;
}
}  // namespace

// Components by union-find (N_c = 1024: 0.45 ms for the three passes): a label is the parent cell, a root its own, and unions point the larger root at the
// smaller, so a component's root ends as its lowest cell id.  Each run of 32 cells of a row starts joined to its first.
__device__ __forceinline__ int sea_find(int32_t *label, int c)
{
    volatile int32_t *l = label;
    int p = l[c];
    while (p != c) {  // halving the path: any ancestor is a valid parent
        const int g = l[p];
        if (g != p) l[c] = g;
        c = p;
        p = g;
    }
    return c;
}

__device__ __forceinline__ void sea_unite(int32_t *label, int a, int b)
{
    while (true) {
        a = sea_find(label, a);
        b = sea_find(label, b);
        if (a == b) return;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicMin(label + a, b);
        if (old == a) return;
        a = old;  // another union moved that root: join what it joined
    }
}

__global__ void sea_init_kernel(int M, int N, int H, int NE, const double *__restrict__ h, const double *__restrict__ s,
                                int32_t *label, double *per, unsigned long long *floorkey)
{
    const int lane = threadIdx.x & 31;
    for (unsigned c0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; c0 < (unsigned)M; c0 += gridDim.x * blockDim.x) {
        const int c = (int)c0 + lane;
        const int row = c / N, j = c - row * N, f = row / N, i = row - f * N;
        bool below = false;
        if (c < M) {
            const int e = (f * NE + i + H) * NE + j + H;
            below = (float)(h[e] + s[e]) < 0.0f;
        }
        const unsigned land = ~__ballot_sync(0xffffffffu, below) & ((1u << lane) - 1u);
        int start = land ? 32 - __clz(land) : 0;  // the run's first lane: after the last land cell, in this row
        start = max(start, lane - j);
        if (c < M) {
            label[c] = below ? c - (lane - start) : -1;
            per[c] = 0.0;
            floorkey[c] = okey(0.0);  // the basin floor starts at 0 (maps.py: np.zeros, then np.minimum.at)
        }
    }
}

__global__ void sea_join_kernel(int M, int N, int H, int NE, const int32_t *__restrict__ owner, int32_t *label)
{
    for (unsigned u = blockIdx.x * blockDim.x + threadIdx.x; u < (unsigned)M; u += gridDim.x * blockDim.x) {
        const int c = (int)u;
        if (((volatile int32_t *)label)[c] < 0) continue;
        const int row = c / N, j = c - row * N, i = row % N;
        auto below = [&](int q) { return ((volatile int32_t *)label)[q] >= 0; };
        if (i == 0 || i == N - 1 || j == 0 || j == N - 1) {  // beside the halo: along the owner table
            for (int k = 0; k < 8; k++) {
                const int q = sea_nb(owner, c, k, N, H, NE);
                if (q >= 0 && below(q)) sea_unite(label, c, q);
            }
        } else {
            // the row above joins itself, so one of its cells that touch is enough; a run joins the one left of it
            if (below(c - N)) {
                sea_unite(label, c, c - N);
            } else {
                if (below(c - N - 1)) sea_unite(label, c, c - N - 1);
                if (below(c - N + 1)) sea_unite(label, c, c - N + 1);
            }
            if ((c & 31) == 0 && below(c - 1)) sea_unite(label, c, c - 1);
        }
    }
}

// (the walk to the root halves no path here: a thread writes its own cell only, so what it writes stays)
__global__ void sea_flatten_kernel(int M, int32_t *label)
{
    volatile int32_t *l = label;
    for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < (unsigned)M; c += gridDim.x * blockDim.x) {
        int r = l[c];
        if (r < 0) continue;
        while (l[r] != r) r = l[r];
        l[c] = r;
    }
}

// the area and the lowest surface of each component (two atomics a cell, all on the ocean's root: 6.8 ms at N_c = 1024;
// as here 53 us): a thread keeps the sums of the label it is at, and a warp whose
// lanes are all at one label (the open ocean nearly everywhere) adds its sum once
constexpr int SEA_PER_LANE = 16;
__global__ void sea_stats_kernel(int M, int N, int H, int NE, const double *__restrict__ h, const double *__restrict__ s,
                                 const float *__restrict__ area, const int32_t *__restrict__ label, double *per,
                                 unsigned long long *floorkey)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int w0 = warp; w0 < (M + 32 * SEA_PER_LANE - 1) / (32 * SEA_PER_LANE); w0 += nwarps) {
        int lab = -1;
        double sum = 0.0;
        unsigned long long low = RF_UNREACHED;
        auto flush = [&]() {
            if (lab < 0) return;
            atomicAdd(per + lab, sum);
            atomicMin(floorkey + lab, low);
        };
        for (int t = 0; t < SEA_PER_LANE; t++) {
            const int c = (w0 * SEA_PER_LANE + t) * 32 + lane;
            const int l = c < M ? label[c] : -1;
            if (l < 0) continue;
            if (l != lab) {
                flush();
                lab = l;
                sum = 0.0;
                low = RF_UNREACHED;
            }
            const int row = c / N, j = c - row * N, f = row / N, i = row - f * N, e = (f * NE + i + H) * NE + j + H;
            sum += (double)area[c];
            low = min(low, okey(h[e] + s[e]));
        }
        const int l0 = __reduce_max_sync(full, lab);
        if (__all_sync(full, lab == l0 || lab < 0)) {
            for (int o = 16; o > 0; o >>= 1) {
                sum += __shfl_xor_sync(full, sum, o);
                low = min(low, __shfl_xor_sync(full, low, o));
            }
            lab = l0;
            if (lane == 0) flush();
        } else {
            flush();
        }
    }
}

__global__ void sea_largest_kernel(long long M, const int32_t *__restrict__ label, const double *__restrict__ per,
                                   unsigned long long *maxkey, unsigned long long *largest, int pass)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < M; c += (long long)gridDim.x * blockDim.x) {
        if (label[c] != (int32_t)c) continue;  // one root per component
        const unsigned long long k = okey(per[c]);
        if (pass == 0) atomicMax(maxkey, k);
        else if (k == *maxkey) atomicMin(largest, (unsigned long long)c);  // np.argmax: the first (lowest) component
    }
}

__global__ void sea_base_kernel(long long total, int N, int H, int NE, const int32_t *__restrict__ label, const double *__restrict__ per,
                                const unsigned long long *__restrict__ floorkey, const unsigned long long *__restrict__ largest,
                                double min_area, double *base)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const long long f = e / ((long long)NE * NE), rem = e % ((long long)NE * NE);
        const int ei = (int)(rem / NE), ej = (int)(rem % NE);
        double b = 0.0;
        if (ei >= H && ei < H + N && ej >= H && ej < H + N) {
            const long long c = (f * N + ei - H) * N + ej - H;
            const int l = label[c];
            if (l >= 0 && (unsigned long long)l != *largest && !(per[l] >= min_area)) b = unokey(floorkey[l]);
        }
        base[e] = b;
    }
}

cudaError_t sea_base(const PgeGrid &g, const PgeState &st, const int32_t *owner, const float *area, double min_area, double *base,
                     int32_t *label_out, const Layout &lay, void *ws, long long max_sweeps, long long *sweeps_out, cudaStream_t s)
{
    const int N = g.N, H = g.H, NE = N + 2 * H;
    const long long M = (long long)g.F * N * N;
    int32_t *label = label_out ? label_out : ws_ptr<int32_t>(ws, lay.flags);
    double *per = ws_ptr<double>(ws, lay.cdf);
    unsigned long long *floorkey = reinterpret_cast<unsigned long long *>(per + M);
    unsigned long long *cnt = ws_ptr<unsigned long long>(ws, lay.counters);
    unsigned long long *maxkey = cnt + 10, *largest = cnt + 11;
    const int m = (int)M;  // (check_shape: the cells count in int32)
    sea_init_kernel<<<grid_for(M), 256, 0, s>>>(m, N, H, NE, st.height, st.sediment, label, per, floorkey);
    sea_join_kernel<<<grid_for(M), 256, 0, s>>>(m, N, H, NE, owner, label);
    sea_flatten_kernel<<<grid_for(M), 256, 0, s>>>(m, label);
    if (sweeps_out) *sweeps_out = 1;
    sea_stats_kernel<<<grid_reduce(M / SEA_PER_LANE + 1), 256, 0, s>>>(m, N, H, NE, st.height, st.sediment, area, label, per, floorkey);
    cudaError_t e;
    if ((e = cudaMemsetAsync(maxkey, 0, 8, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(largest, 0xFF, 8, s)) != cudaSuccess) return e;
    sea_largest_kernel<<<grid_for(M), 256, 0, s>>>(M, label, per, maxkey, largest, 0);
    sea_largest_kernel<<<grid_for(M), 256, 0, s>>>(M, label, per, maxkey, largest, 1);
    sea_base_kernel<<<grid_for(lay.ncell), 256, 0, s>>>(lay.ncell, N, H, NE, label, per, floorkey, largest, min_area, base);
    return cudaPeekAtLastError();
}

// ---------------------------------------------------------------------------
// glacial pass (erosion/glacial.py:162-257; the ice line of the evaporation
// field).  Every per-cell rule runs on the whole extended array, neighbours
// wrapping at each face array's edges as numpy's roll does, so the interior
// comes out as the reference's; the sums are float64 atomics.
// ---------------------------------------------------------------------------
namespace {
__device__ __forceinline__ long long glac_nb(long long e, int NE, int k)
{
    const long long f = e / ((long long)NE * NE), rem = e % ((long long)NE * NE);
    int i = (int)(rem / NE) + kRouteD8[k][0], j = (int)(rem % NE) + kRouteD8[k][1];
    i = i < 0 ? i + NE : (i >= NE ? i - NE : i);
    j = j < 0 ? j + NE : (j >= NE ? j - NE : j);
    return (f * NE + i) * NE + j;
}
__device__ __forceinline__ bool glac_interior(long long e, int NE, int H, int N)
{
    const long long rem = e % ((long long)NE * NE);
    const int i = (int)(rem / NE), j = (int)(rem % NE);
    return i >= H && i < H + N && j >= H && j < H + N;
}
struct GlacSums {
    unsigned long long ice_any, ice_interior, margin_any, margin_interior, max_key;
    double carved, wsum, parked;
};
}  // namespace

__global__ void glac_ice_kernel(long long n, int NE, int H, int N, const double *__restrict__ h, const double *__restrict__ s,
                                const float *__restrict__ evap, const uint8_t *__restrict__ mask, const uint8_t *__restrict__ prev,
                                float ice_evap, uint8_t *ice, double *depth, GlacSums *sums)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const bool active = mask ? mask[e] == PGE_MASK_ACTIVE : true;
        const bool cold = evap[e] <= ice_evap;
        bool v = active && cold && (h[e] + s[e] > 0.0);
        if (prev && prev[e] && active && cold) v = true;
        ice[e] = v;
        depth[e] = v ? 1.0 : 0.0;
        if (v) {
            atomicAdd(&sums->ice_any, 1ull);
            if (glac_interior(e, NE, H, N)) atomicAdd(&sums->ice_interior, 1ull);
        }
    }
}

// one ring: a cell stays inside while it and its eight neighbours are
__global__ void glac_ring_kernel(long long n, int NE, const uint8_t *__restrict__ inner, uint8_t *shrunk, double *depth)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        bool v = inner[e];
        for (int k = 0; k < 8 && v; k++) v = inner[glac_nb(e, NE, k)];
        shrunk[e] = v;
        if (v) depth[e] += 1.0;
    }
}

__global__ void glac_dz_kernel(long long n, int NE, int H, int N, const double *__restrict__ h, const double *__restrict__ s,
                               const double *__restrict__ q, const float *__restrict__ hard, const double *__restrict__ base,
                               const uint8_t *__restrict__ ice, const double *__restrict__ depth, int ramp, double rate, double cap,
                               double sat, double dep_floor, double *dz, GlacSums *sums)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        double taper = depth[e];
        if (ramp > 0) {
            taper = taper / (double)(ramp + 1);
            taper = taper < 0.0 ? 0.0 : (taper > 1.0 ? 1.0 : taper);
        }
        const double qq = (q[e] > 0.0 ? q[e] : 0.0) / sat;
        const float hf = __fsub_rn(1.0f, __fmul_rn(0.5f, hard[e]));  // float32, as the reference's array arithmetic
        double d = rate * sqrt(qq) * (double)hf * taper;
        d = d < 0.0 ? 0.0 : (d > cap ? cap : d);
        if (!ice[e]) d = 0.0;
        double room = h[e] + s[e] + dep_floor - base[e];
        if (room < 0.0) room = 0.0;
        if (room < d) d = room;
        dz[e] = d;
        if (d != 0.0 && glac_interior(e, NE, H, N)) {
            atomicAdd(&sums->carved, d);
            atomicMax(&sums->max_key, okey(d));
        }
    }
}

__global__ void glac_carve_kernel(long long n, double *h, const double *__restrict__ dz)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        h[e] -= dz[e];
}

__global__ void glac_margin_kernel(long long n, int NE, int H, int N, const double *__restrict__ h, const double *__restrict__ s,
                                   const double *__restrict__ q, const double *__restrict__ base, const uint8_t *__restrict__ mask,
                                   const uint8_t *__restrict__ ice, double *w, GlacSums *sums)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        bool near = false;
        for (int k = 0; k < 8 && !near; k++) near = ice[glac_nb(e, NE, k)];
        const bool active = mask ? mask[e] == PGE_MASK_ACTIVE : true;
        const bool margin = near && !ice[e] && active && (h[e] + s[e] > base[e]);
        w[e] = margin ? (q[e] > 0.0 ? q[e] : 0.0) + 1e-6 : 0.0;
        if (margin) {
            atomicAdd(&sums->margin_any, 1ull);
            if (glac_interior(e, NE, H, N)) {
                atomicAdd(&sums->margin_interior, 1ull);
                atomicAdd(&sums->wsum, w[e]);
            }
        }
    }
}

__global__ void glac_moraine_kernel(long long n, int NE, int H, int N, const double *__restrict__ w, double wsum, double load, double cap,
                                    double *s, double *pending, GlacSums *sums)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const double add = (w[e] / wsum) * load;
        const double placed = add < cap ? add : cap;
        s[e] += placed;
        pending[e] += add - placed;
        const double parked = add - placed;
        if (parked != 0.0 && glac_interior(e, NE, H, N)) atomicAdd(&sums->parked, parked);
    }
}

int glacial(const PgeGrid &g, PgeState &st, uint8_t *ice_prev, const GlacialArgs &ga, double stats[5], const Layout &lay, void *ws,
            cudaStream_t s)
{
    const int N = g.N, H = g.H, NE = N + 2 * H;
    const long long n = lay.ncell;
    stats[0] = stats[1] = stats[2] = stats[3] = stats[4] = 0.0;
    if (ga.rate <= 0.0) return 0;
    uint8_t *ice = ws_ptr<uint8_t>(ws, lay.flags), *ping = ice + n, *pong = ice + 2 * n;
    double *depth = ws_ptr<double>(ws, lay.thermal), *dz = depth + n, *w = depth + 2 * n;
    GlacSums *sums = reinterpret_cast<GlacSums *>(ws_ptr<unsigned long long>(ws, lay.counters) + 12);
    GlacSums hs;
    cudaError_t e;
    auto read = [&]() -> cudaError_t {
        cudaError_t r = cudaMemcpyAsync(&hs, sums, sizeof(GlacSums), cudaMemcpyDeviceToHost, s);
        return r == cudaSuccess ? cudaStreamSynchronize(s) : r;
    };
    if ((e = cudaMemsetAsync(sums, 0, sizeof(GlacSums), s)) != cudaSuccess) return -(int)e;
    glac_ice_kernel<<<grid_for(n), 256, 0, s>>>(n, NE, H, N, st.height, st.sediment, st.evap, st.mask, ice_prev, ga.ice_evap, ice,
                                                depth, sums);
    if ((e = read()) != cudaSuccess) return -(int)e;
    if (!hs.ice_any) return 0;  // no ice: nothing changes (and the last ice stays as it was)
    if (ice_prev && (e = cudaMemcpyAsync(ice_prev, ice, n, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return -(int)e;
    if (ga.ramp > 0) {
        const uint8_t *inner = ice;
        for (int r = 0; r < ga.ramp; r++) {
            uint8_t *out = (r & 1) ? pong : ping;
            glac_ring_kernel<<<grid_for(n), 256, 0, s>>>(n, NE, inner, out, depth);
            inner = out;
        }
    }
    glac_dz_kernel<<<grid_for(n), 256, 0, s>>>(n, NE, H, N, st.height, st.sediment, st.discharge, st.hardness, st.base, ice, depth,
                                               ga.ramp, ga.rate, ga.cap, ga.sat, ga.dep_floor, dz, sums);
    if ((e = read()) != cudaSuccess) return -(int)e;
    if (!(hs.carved > 0.0)) return 0;  // nothing carved: the reference returns before any change (and empty statistics)
    glac_carve_kernel<<<grid_for(n), 256, 0, s>>>(n, st.height, dz);
    glac_margin_kernel<<<grid_for(n), 256, 0, s>>>(n, NE, H, N, st.height, st.sediment, st.discharge, st.base, st.mask, ice, w, sums);
    if ((e = read()) != cudaSuccess) return -(int)e;
    if (hs.margin_any && ga.moraine_frac > 0.0 && hs.wsum > 0.0) {
        glac_moraine_kernel<<<grid_for(n), 256, 0, s>>>(n, NE, H, N, w, hs.wsum, hs.carved * ga.moraine_frac, ga.iter_deposit,
                                                        st.sediment, st.pending, sums);
        if ((e = read()) != cudaSuccess) return -(int)e;
    }
    stats[0] = (double)hs.ice_interior;
    stats[1] = hs.carved;
    stats[2] = (double)hs.margin_interior;
    {  // the order-preserving key back to its double (host side of unokey)
        const unsigned long long k = hs.max_key;
        const unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
        double v;
        memcpy(&v, &b, sizeof v);
        stats[3] = v;
    }
    stats[4] = hs.parked;
    return 0;
}

cudaError_t window_lakes(const PgeGrid &g, const PgeState &st, double min_depth, uint8_t *flag, int64_t *count, cudaStream_t stream)
{
    const long long NE = g.N + 2LL * g.H, n = (long long)g.F * NE * NE;
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(count);
    if (cnt) {
        const cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), stream);
        if (e != cudaSuccess) return e;
    }
    window_lakes_kernel<<<grid_for(n), 256, 0, stream>>>(n, g.N, g.H, st.height, st.sediment, st.route, st.mask, min_depth, flag, cnt);
    return cudaGetLastError();
}

}  // namespace pge

