// bls_gather.cuh -- the search by prefix gathering (included by bls_engine.cu,
// inside its anonymous namespace).
//
// For time-ordered points the slot of a point is a non-decreasing function of
// its time within one cycle of the period, so the points of cycle k that lie in
// slots 1..j are those before one instant, k*P + j*(bin width).  With V the
// running sum of the points' words (weight and flux) over time, the prefix sum
// the window search needs is
//     C[j] = sum over cycles k of  V(points before boundary (k, j)) - V(points before (k, 0)).
// One boundary costs one table look-up and a 64-bit addition, whatever the number of
// points in a bin; there is no histogram to clear, to add to atomically, to pad or
// to scan.  A curve with N points over a time span T takes N reductions per
// period by scattering and about T / (bin width) look-ups by gathering, so the
// gathering wins wherever bins hold about half a point per cycle or more, and a
// period with more bins than shared memory holds needs no extra passes.
//
// The result is the scattered one, bit for bit: V holds exact integers (sums are
// taken modulo 2^64 and decode exactly), and a boundary whose instant falls within
// one table unit (2^-24 of a cell) of a point is decided by the fold's own
// formula for that point (gather_exact).
//
// Table of a curve (table_kernel): time is cut into cells, at most about one
// point per cell; a cell holds the offset of its point (24 bits of the cell
// width; kOffMulti: several points), V before the cell and the number of points
// before it.  Astropy bins all have the width b = min(duration) / oversample:
// cells are b / S wide (S rows) and cell c is stored at row c % S, column c / S, so
// that the boundaries j, j+1, ... of one cycle -- S cells apart -- are
// consecutive entries of one row and share one offset inside their cells: a
// warp's 32 look-ups are coalesced and need no arithmetic per lane.  Fixed bins
// change their width with the period; their cells are stored in order.
//
// One warp searches one period: it gathers 128 boundaries at a time into a buffer of
// FP32 prefix entries and evaluates the windows that end inside it.  With astropy bins
// the buffer slides, so 384 entries (3 KB) do for a period of any number of bins; fixed
// bins hold the period twice (up to kMaxRing entries).  The warps of a CTA wait for one
// another after each period only to share table lines and instructions
// (gather_periods).  Bound by issue slots and look-up latency.

// 16 warps share table lines and instructions; 8 took 2.15 ms where 16 took 1.95
// (16 one-sector curves), 32 were slower on full batches
constexpr int kGatherBlock = 512;
constexpr int kGatherMinBlocks = 2;
constexpr int kGatherWarps = kGatherBlock / 32;
constexpr int kTableBlock = 512;
constexpr int kMaxRows = 8;                      // rows of an astropy-binned table
constexpr int kOffBits = 24;
constexpr unsigned kOffMask = (1u << kOffBits) - 1u;  // units per cell - 1
constexpr unsigned kOffMulti = 0xffffffffu;      // the cell holds several points
constexpr double kOffUnits = 16777216.0;         // 2^kOffBits
constexpr double kOffHalf = 8388608.0;           // boundaries of cycle 0 lie mid-cell
// Astropy bins: the boundaries of cycle 0 are the same for every period, multiples of the
// bin width from the first point, and all share this offset.  The first point lies on one
// of them, and with an exact cadence every 25th point or so may.  Which side such a point is
// on is decided once, by the fold's formula, when the table is made, and its offset there
// (one or two units off) says so: cycle 0 needs no checks.  With them, 64 curves of 15 000
// points at exactly 2 minutes and 2000 periods took 2.92 ms gathered and 2.77 scattered;
// without them 2.15.
constexpr unsigned kOffMid = 1u << (kOffBits - 1);
constexpr int kRowPad = 128;                     // columns a block of look-ups may pass the last by
constexpr long long kGatherMinPoints = 4096;      // shorter curves search faster than a table is made
constexpr long long kGatherMaxPoints = (1LL << 18) - 1;
constexpr long long kGatherMinPeriods = 32;      // of a curve
// Prices, in the quarters of an SM clock of gather_gain: a table is made by one CTA, 6 ns per
// point, while the rest of the GPU waits for it, and by up to 600 CTAs at a time.
constexpr long long kTableLatency = 12000;       // per point of the longest curve
constexpr long long kTablePrice = kTableLatency / 600;  // per point of every curve
// And what no sum over periods shows, about 40 us: the kernels of the look-up search itself and
// its last, half-empty wave.  (500 drawn batches of 12 000 to 250 000 periods: 133 took the
// tables without it, ten of them longer for it, by up to 160 us; with it, and with the
// shares of gather_gain as they are now, 122 and five, by up to 60.)
constexpr double kGatherPrice = 4.65e7;
constexpr int kPriceClasses = 24;                // curve lengths by quarters of an octave
constexpr int kHeadMax = 17;                     // saved prefix entries 0..oversample (<= 16)

// cells reserved for a curve of n points (0: too short or too long for a table)
__host__ __device__ inline long long gather_cells(long long n) {
    return n < kGatherMinPoints || n > kGatherMaxPoints
               ? 0
               : (2 * n + 1024 + kMaxRows * (kRowPad + 16)) / 8 * 8;
}

// What the curves of one class of lengths (quarters of an octave from kGatherMinPoints)
// would save and cost, summed over the batch by gain_kernel.
struct GatherPrice {
    long long saved[kPriceClasses];   // points scattered, less the look-ups
    long long looks[kPriceClasses];   // the look-ups alone
    long long periods[kPriceClasses];
    long long points[kPriceClasses];
    int longest[kPriceClasses];
};

__host__ __device__ inline int price_class(long long n) {
    int oct = 0;
    while (n >> (oct + 13)) ++oct;  // 4096..8191: 0
    return oct * 4 + (int)(n >> (oct + 10) & 3);
}

// Constants of a curve's windows (and of one fixed-bin period whose trash slot
// holds points): the exact test's totals, and the filter's.
//
// The filter works on FP32 prefix values in "units" (flux: |y| < 2^31 units;
// weight: points, or w below 2^31 units): c the weight prefix and g = c1 c - y, so
// that a window's sigma is g1 - g0 and its weight c1 - c0.  Its error, every
// rounding of the filter and of the exact test included (floor to units,
// conversion, fma, both subtractions), is at most
//     E = e0 + 2^-21 (|g0| + |g1|),
// and for weighted curves a weight difference is off by at most wE.  A window that holds
// a point weighs at least wm: without that bound, every window over an empty stretch of
// phase would pass with a weight of -wE, fill the list and send the period to the
// scatter kernel (48 curves of 15 000 points, 1581 periods of 0.5 to 1.5 spans: 27 % of
// them given back).
struct GatherConsts {
    double wtot, ytot;  // exact totals, scaled like the scan's prefix sums
    float c1, fN;       // as WinConsts
    float f1, e0;       // c1 in units; absolute part of E
    float wE, wN;       // wN: total weight in units, minus 2 wE
    float wm;           // the least weight of a point, rounded down (weighted curves)
};

// A curve's record for the gather kernel.
struct TableStat : CurveStat {
    int g_on;        // the curve has a table
    int g_n;         // points
    int g_bl;        // packed words: bits of the count field (the top bits)
    int g_guard;     // and the left shift of the flux sums below them
    int g_rows;      // table rows: cells per bin width (1 for fixed bins)
    int g_pitch;     // entries per row
    int g_colmax;    // last column a look-up may use
    int lmax;        // longest window in bins (astropy bins)
    double g_scale;  // table units (2^-24 cell) per unit time
    long long n_g;   // periods that are gathered
    GatherConsts gk;
};

struct GatherArgs {
    char* tab;                 // entries (Entry<>), 16 * vs bytes per cell
    unsigned* idx;             // per cell: points before it
    unsigned* bits;            // astropy bins: the offsets near some point, see offset_shift
    const long long* bit_off;  // per curve: first word of `bits`
    const long long* cell_off; // per curve: first cell; cell_off[n_curves] = all
    unsigned long long* counter;  // work counters of the packed and the weighted kernel
    unsigned long long* n_gather;  // periods that are gathered, by kernel
    unsigned long long* n_back;    // of these, given back to the scatter kernel
    int* n_scatter;            // some period is scattered
    GatherPrice* price;
    int warps[2];              // resident warps of the packed and the weighted kernel,
    int one_cta[2];            // and whether they are one CTA per SM
    int vs;                    // 2 when weights are given, else 1
    int ring;                  // prefix entries a warp holds
    int beside;                // plans that run at the same time, this one included
};

// What gathering a period saves, in quarters of an SM clock (about a scattered point of a
// counting curve); -INFINITY where it cannot be gathered.  `look` receives the look-ups'
// share.  Fitted to both kernels' times of 340 batches (15 000 to 150 000 points, periods
// of 0.6 to 150 d, 6 and 8 durations, 0.002 and 0.004 d bins; 592 periods of 32 curves):
//   astropy bins, counting: scattering 0.23 clocks per point and pass, 3.5 per bin (clear,
//     scan, windows) and 2.6 per point of the last bin where max_bins cuts the period (they
//     add to one address); gathering 0.34 per look-up -- whole blocks of 128 per cycle -- and
//     2.2 per bin; within 20 % of the times.  Weighted: 0.37, 3.7, 3.3; 0.71, 1.9 and
//     500 per period.  Of the bins' share, windows of one duration cost gathering
//     0.10 clocks less (0.25 weighted): 64 weighted curves of 20 000 points, 2000 periods of
//     678 bins on average gain 7 % with six durations, nothing with two and 20 % with twenty.
//   fixed bins, whose look-ups take a cache line each: 0.8 to 1.5 per look-up (weighted
//     2 to 3.3).  One look-up for five points (weighted: ten) breaks even: 15 000 points,
//     200 bins and 10 cycles scatter in 5500 clocks and gather in 4400; 150 000 points, 300
//     bins and 40 cycles in 43 000 and 31 000, 119 cycles in 38 500 and 71 400.
//     Neighbouring periods share lines unless the grid is so coarse (`step`) that their
//     boundaries lie far apart: 160 curves of 15 286 points, 333 bins, took 774 us scattered
//     and 939 gathered by 209 periods from 1.5 to 23 d.
//     Where the prefix entries leave an SM one CTA (from 320 bins, `one_cta`), a period
//     costs 5 clocks per bin more (weighted 2.5): 500 bins and one cycle of 15 000 points
//     scatter in 7800 clocks and gather in 8100.
template <int GEOM>
__device__ __forceinline__ double gather_gain(const CurveStat& st, int n, int lmax, double P,
                                              double step, int NB, int os, int cap,
                                              bool one_cta, double& look) {
    // (a period beyond 64 spans would leave the table's number range)
    if (!(P > 0.0) || !(P <= 64.0 * st.dt_absmax)) return -INFINITY;
    const double cycles = floor(st.dt_absmax * (1.0 / P)) + 1.0;
    const bool cnt = st.cnt_win != 0;
    if (GEOM == ATB_GEOM_BINNED) {
        if (NB <= 2 * os) return -INFINITY;  // the padding copy's ranges overlap
        const double bounds = fmin((double)NB + 1.0, P * st.inv_bin_dur + 1.0);
        // a period that does not fit the scatter's shared histogram folds its points
        // once per bin-range pass
        const double passes =
            NB + 2 > cap ? ceil((double)NB / (double)max(cap - 2 - lmax, 64)) : 1.0;
        const double nd = (double)st.n_dur;
        const double cut = fmax(0.0, 1.0 - (double)NB / (P * st.inv_bin_dur));
        look = (cnt ? 1.35 : 2.85) * cycles * 128.0 * ceil(bounds * (1.0 / 128.0));
        return (double)n * ((cnt ? 0.92 : 1.49) * passes + (cnt ? 10.4 : 13.3) * cut) +
               (cnt ? 2.3 + 0.41 * nd : 0.2 + nd) * bounds - look - (cnt ? 0.0 : 2000.0);
    }
    const double apart = step * cycles * 0.5 * (double)n / st.dt_absmax;  // cells
    look = (cnt ? 5.0 : 10.0) * cycles * 128.0 * ceil(((double)NB + 1.0) * (1.0 / 128.0)) *
           (1.0 + 0.6 * fmin(1.0, apart * (1.0 / 96.0)));
    return (double)n - look - (one_cta ? (cnt ? 20.0 : 10.0) * (double)NB : 0.0);
}

// A running sum: packed (counting curves) one word, else weight and flux.
template <bool PK>
struct Sum {
    unsigned long long x;
    __device__ __forceinline__ void add(const Sum& o) { x += o.x; }
    __device__ __forceinline__ void sub(const Sum& o) { x -= o.x; }
};
template <>
struct alignas(16) Sum<false> {
    unsigned long long x, y;
    __device__ __forceinline__ void add(const Sum& o) { x += o.x; y += o.y; }
    __device__ __forceinline__ void sub(const Sum& o) { x -= o.x; y -= o.y; }
};

template <bool PK>
__device__ __forceinline__ Sum<PK> shfl_sum(Sum<PK> v, int l) {
    v.x = __shfl_sync(0xffffffffu, v.x, l);
    if constexpr (!PK) v.y = __shfl_sync(0xffffffffu, v.y, l);
    return v;
}

// A cell: V before it, its point's offset and words.
template <bool PK>
struct alignas(16) Entry {
    unsigned long long x;
    unsigned off;
    int q;
};
template <>
struct alignas(16) Entry<false> {
    unsigned long long x, y;
    unsigned off;
    int qw, qy, pad;
};

// Offsets within one unit of some point's are marked in a curve's bit map of
// 64 to 128 bits per point; an offset's bit is offset >> offset_shift.
__host__ __device__ inline int offset_shift(int bl) { return bl + 6 < kOffBits ? kOffBits - bl - 6 : 0; }
__host__ __device__ inline long long offset_words(int bl) { return 1LL << (kOffBits - offset_shift(bl) - 5); }

template <bool PK>
__device__ __forceinline__ int flux_shift(const TableStat& st) {
    return max(0, st.qbits + st.g_bl - 31);
}

__device__ __forceinline__ unsigned packed_count(unsigned long long x, int bl) {
    return (unsigned)((x + (1ULL << (63 - bl))) >> (64 - bl));
}
// exact flux sum of a packed word
__device__ __forceinline__ long long packed_flux(unsigned long long x, int bl, int guard) {
    return (long long)(x << bl) >> (bl + guard);
}

// totals of the whole curve in table words
template <bool PK>
__device__ __forceinline__ Sum<PK> curve_total(const TableStat& st) {
    Sum<PK> s;
    if constexpr (PK) {
        s.x = ((unsigned long long)st.g_n << (64 - st.g_bl)) +
              ((unsigned long long)st.qy_tot << st.g_guard);
    } else {
        s.x = (unsigned long long)st.qw_tot;
        s.y = (unsigned long long)st.qy_tot;
    }
    return s;
}

template <bool PK>
__device__ __noinline__ void gather_consts(const TableStat& st, const Sum<PK>& tot,
                                           GatherConsts& k) {
    const double sy2 = ldexp(1.0, -st.ey), sw2 = ldexp(1.0, -st.ew);
    const int sh = flux_shift<PK>(st);
    if constexpr (PK) {
        const double fN = (double)packed_count(tot.x, st.g_bl);
        const double fy = ldexp(1.0, st.ey + st.g_guard + st.g_bl - 32);  // scaled -> units
        k.fN = (float)fN;
        k.wtot = fN * ldexp((double)st.qw0, -st.ew);
        k.ytot = (double)packed_flux(tot.x, st.g_bl, st.g_guard) * sy2;
        k.c1 = (float)(k.ytot / fN);
        k.f1 = k.c1 * (float)fy;
        k.wE = 0.0f;
        k.wN = k.fN;
        k.wm = 0.0f;
        k.e0 = 4.0f + 4.76837158203125e-07f * (float)(fabs(k.ytot) * fy);
    } else {
        const double fy = ldexp(1.0, st.ey - sh), fw = ldexp(1.0, st.ew - sh);
        k.fN = 0.0f;
        k.wtot = (double)(long long)tot.x * sw2;
        k.ytot = (double)(long long)tot.y * sy2;
        k.c1 = (float)(k.ytot / k.wtot);
        k.f1 = k.c1 * (float)(fy / fw);
        k.wE = 2.0f + 4.76837158203125e-07f * (float)(k.wtot * fw);
        k.wN = (float)(k.wtot * fw) - 2.0f * k.wE;
        // (1 - 2^-18): the exact test's roundings stay on the safe side
        k.wm = (float)ldexp((double)st.qw_min, -sh) * 0.999996185302734375f;
        k.e0 = 4.0f + 4.76837158203125e-07f * (float)(fabs(k.ytot) * fy);
    }
}

// ----------------------------------------------------------------------------
// table kernel: one CTA per curve, after the stage kernel
// ----------------------------------------------------------------------------

struct TableShared {
    long long red[kTableBlock / 32];
    long long scan[2][kTableBlock / 32];
    int flag;
};

__device__ long long tb_sum(long long v, TableShared& sh) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5] = v;
    __syncthreads();
    long long r = 0;
#pragma unroll
    for (int i = 0; i < kTableBlock / 32; ++i) r += sh.red[i];
    return r;
}

// exclusive block scan of two values; returns the block totals in tx, ty
__device__ void tb_scan2(long long& x, long long& y, long long& tx, long long& ty,
                         TableShared& sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long ix = x, iy = y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long ax = __shfl_up_sync(0xffffffffu, ix, o);
        const long long ay = __shfl_up_sync(0xffffffffu, iy, o);
        if (lane >= o) {
            ix += ax;
            iy += ay;
        }
    }
    __syncthreads();
    if (lane == 31) {
        sh.scan[0][w] = ix;
        sh.scan[1][w] = iy;
    }
    __syncthreads();
    long long ox = 0, oy = 0;
    tx = 0;
    ty = 0;
#pragma unroll
    for (int i = 0; i < kTableBlock / 32; ++i) {
        const long long vx = sh.scan[0][i], vy = sh.scan[1][i];
        if (i < w) {
            ox += vx;
            oy += vy;
        }
        tx += vx;
        ty += vy;
    }
    x = ix - x + ox;
    y = iy - y + oy;
}

// (q_w, q_y) of the point held at staged position q
__device__ __forceinline__ void staged_words(const CurveStat& st, const int* sqw, const int* sqy,
                                             long long q, int& qw, int& qy) {
    const int a = sqw[q], b = sqy[q];
    if (st.packmode == kPackTight) {
        qw = 1;
        qy = b * (1 << st.stage_lob) + (int)((unsigned)a & ((1u << st.stage_lob) - 1u));
    } else {
        qw = a;  // 1 in the count layout
        qy = b;
    }
}

// A point's table words: packed (counting curves) x = count << (64 - bl) plus
// q_y << guard, y unused; else x = q_w, y = q_y.
__device__ __forceinline__ void point_words(const TableStat& st, int qw, int qy, long long& x,
                                            long long& y) {
    if (st.cnt_win) {
        x = (long long)((1ULL << (64 - st.g_bl)) +
                        ((unsigned long long)(long long)qy << st.g_guard));
        y = 0;
    } else {
        x = qw;
        y = qy;
    }
}

__device__ __forceinline__ unsigned long long cell_units(double d, double scale) {
    return (unsigned long long)(long long)__double2ll_rd(d * scale) + (unsigned long long)kOffHalf;
}

// Which curves can have a table, which of their periods it would take and what that
// saves: before any table is made, so that a batch it does not pay for loses no more
// than this pass over the grids.  One CTA per curve, after the stage kernel.
template <int GEOM>
__global__ void __launch_bounds__(kTableBlock) gain_kernel(const SearchArgs a, const GatherArgs ga,
                                                           TableStat* stats) {
    __shared__ TableShared sh;
    chain_next();
    chain_start();
    const int c = blockIdx.x, tid = threadIdx.x;
    const long long n = a.pt_off[c + 1] - a.pt_off[c];
    const long long cells = ga.cell_off[c + 1] - ga.cell_off[c];
    const long long np = a.per_cnt[c];
    TableStat sg;
    static_cast<CurveStat&>(sg) = a.stats[c];
    const double T = sg.dt_absmax;
    int lmax = 0;
    if (GEOM == ATB_GEOM_BINNED)
        for (int k = 0; k < sg.n_dur; ++k) lmax = max(lmax, a.dbins[c * kMaxDur + k]);
    // packed words: a flux field that holds twice the absolute total, shifted up to
    // fill it (the filter converts its top 32 bits)
    sg.g_guard = min(24, 61 - bitlen64(n) - bitlen64(2 * sg.qy_abs));
    // Split weights need two words per cell.  A flat curve's windows are all equal: its
    // periods' lists overflow, one and all, and each would be searched twice (64 flat
    // curves of 15 000 points: 12.1 ms, 8.9 scattered).
    bool on = cells > 0 && !sg.flat && T > 0.0 && T < 1.0e300 &&
              (sg.cnt_win ? sg.g_guard >= 0 : ga.vs == 2);
    if (GEOM == ATB_GEOM_BINNED)
        on = on && sg.thr_unit && sg.bin_dur > 0.0 && sg.inv_bin_dur < 1.0e300 &&
             a.oversample < kHeadMax && lmax <= ga.ring - 192 &&
             // (a period's look-ups are at least T / b, and bin-range passes rarely double
             // the scattering)
             T * sg.inv_bin_dur <= 1.55 * (double)n;
    else
        on = on && 2 * a.n_bins_fixed + 1 <= ga.ring;
    unsigned char* scatter = a.scatter + a.flag_off[c];
    long long n_g = 0, saved = 0, looks = 0;
    if (on) {
        const bool one_cta = ga.one_cta[sg.cnt_win ? 0 : 1] != 0;
#pragma unroll 4
        for (long long i = tid; i < np; i += kTableBlock) {
            const double P = a.periods[a.per_beg[c] + i];
            const int NB = GEOM == ATB_GEOM_BINNED
                               ? binned_nbins(P, sg.inv_bin_dur, a.oversample, a.max_bins)
                               : a.n_bins_fixed;
            double look = 0.0;
            const double gain = gather_gain<GEOM>(
                sg, (int)n, lmax, P, fabs(a.periods[a.per_beg[c] + (i + 1 < np ? i + 1 : i - 1)] - P),
                NB, a.oversample, a.cap, one_cta, look);
            // astropy bins: every period that can be, or none -- the look-ups per point
            // hardly depend on the period, and a curve split over both kernels took
            // longer than in either; fixed bins: the periods that gain
            const bool g = gain > (GEOM == ATB_GEOM_BINNED ? -INFINITY : 0.0);
            scatter[i] = g ? 0 : 1;
            n_g += g ? 1 : 0;
            if (g) {
                saved += (long long)fmin(gain, 1.0e9);
                looks += (long long)fmin(look, 1.0e9);
            }
        }
        n_g = tb_sum(n_g, sh);
        saved = tb_sum(saved, sh);
        looks = tb_sum(looks, sh);
        on = n_g > 0 && saved >= kTablePrice * n;
    }
    if (!on) {
        __syncthreads();
        for (long long i = tid; i < np; i += kTableBlock) scatter[i] = 1;
    }
    if (tid == 0) {
        sg.g_on = on ? 1 : 0;
        sg.g_n = (int)min(n, (long long)INT_MAX);
        sg.lmax = lmax;
        sg.n_g = n_g;
        sg.g_rows = sg.g_pitch = sg.g_colmax = sg.g_bl = 0;
        sg.g_scale = 0.0;
        stats[c] = sg;
        if (on) {
            const int k = price_class(n);
            atomicAdd((unsigned long long*)ga.price->saved + k, (unsigned long long)saved);
            atomicAdd((unsigned long long*)ga.price->looks + k, (unsigned long long)looks);
            atomicAdd((unsigned long long*)ga.price->periods + k, (unsigned long long)n_g);
            atomicAdd((unsigned long long*)ga.price->points + k, (unsigned long long)n);
            atomicMax(ga.price->longest + k, (int)n);
        }
        if (!on || n_g < np) atomicOr(ga.n_scatter, 1);
    }
}

// The last class of lengths that gets tables (-1: none): with it, what they save less
// what they cost is largest.  Too few periods leave warps of the gather kernel idle and
// their look-ups take as much longer.  Of what only leaves the GPU idle, `beside` plans that
// run at the same time each bear a share (24 curves of 34 536 points, 6000 periods, as a
// session of four: 4.55 ms scattered, 3.36 by tables).
__device__ __forceinline__ int priced_class(const GatherPrice& p, int warps, int beside) {
    long long saved = 0, looks = 0, periods = 0, points = 0;
    double best = 0.0;
    int last = -1;
    for (int k = 0; k < kPriceClasses; ++k) {
        if (p.periods[k] == 0) continue;
        saved += p.saved[k];
        looks += p.looks[k];
        periods += p.periods[k];
        points += p.points[k];
        const double idle = fmax(0.0, (double)(warps / beside) / (double)periods - 1.0);
        const double net = (double)saved - (double)looks * idle -
                           fmax((double)(kTableLatency / beside) * (double)p.longest[k],
                                (double)kTablePrice * (double)points) -
                           kGatherPrice / (double)beside;
        if (net >= best) {
            best = net;
            last = k;
        }
    }
    return last;
}

// The tables of the curves that pay (CTAs of others end at once).
template <int GEOM>
__global__ void __launch_bounds__(kTableBlock) table_kernel(const SearchArgs a, const GatherArgs ga,
                                                            TableStat* stats) {
    __shared__ TableShared sh;
    chain_start();
    const int c = blockIdx.x, tid = threadIdx.x;
    if (!stats[c].g_on) return;
    TableStat sg = stats[c];
    const CurveStat& st = sg;
    const long long n = a.pt_off[c + 1] - a.pt_off[c];
    const long long so = a.stage_off[c];
    const long long cells = ga.cell_off[c + 1] - ga.cell_off[c];
    const long long np = a.per_cnt[c];
    const long long n_full = st.ilv ? (n + kR - 1) / kR * kR / kChunk * kChunk : 0;
    const double* sdt = a.sdt + so;
    const double T = st.dt_absmax;
    if (tid == 0) sh.flag = price_class(n) <=
                           priced_class(*ga.price, ga.warps[st.cnt_win ? 0 : 1], ga.beside);
    __syncthreads();
    bool on = sh.flag != 0;
    const long long most_shared = GEOM == ATB_GEOM_BINNED ? 0 : n / 512;
    double scale = 0.0;  // units per time
    int rows = 1;
    if (on) {
        // spacings below each candidate cell width (astropy bins: b/1 .. b/8; fixed:
        // T/n * 2^(-m/4)); the widest with at most n/1024 of them is taken
        double w[kMaxRows];
#pragma unroll
        for (int m = 0; m < kMaxRows; ++m)
            w[m] = 0.9999 * (GEOM == ATB_GEOM_BINNED ? st.bin_dur / (double)(m + 1)
                                                     : T / (double)n * exp2(-0.25 * (m + 1)));
        int cnt[kMaxRows] = {0, 0, 0, 0, 0, 0, 0, 0};
        int unsorted = 0;
        for (long long i = tid; i + 1 < n; i += kTableBlock) {
            const double dd = sdt[staged_pos(i + 1, n_full)] - sdt[staged_pos(i, n_full)];
            unsorted |= !(dd >= 0.0);
#pragma unroll
            for (int m = 0; m < kMaxRows; ++m) cnt[m] += dd < w[m] ? 1 : 0;
        }
        on = !__syncthreads_or(unsorted);
        int pick = -1;
        long long close = 0;  // spacings below the chosen width
#pragma unroll
        for (int m = kMaxRows - 1; m >= 0; --m) {
            const long long k = tb_sum(cnt[m], sh);
            if (k <= n / 1024) {
                pick = m;
                close = k;
            }
        }
        on = on && pick >= 0;
        if (on) {
            if (GEOM == ATB_GEOM_BINNED) {
                rows = pick + 1;
                scale = kOffUnits * (double)rows * st.inv_bin_dur;
            } else {
                scale = kOffUnits * (double)n / T * exp2(0.25 * (pick + 1));
            }
            on = T * scale / kOffUnits + (double)(rows * (kRowPad + 16)) < (double)cells;
        }
        // Points that share a cell are decided exactly.  With fixed bins a look-up sees
        // that; with astropy bins every cycle would have to be looked up with every check,
        // since its boundaries are (64 curves of 15 000 points, one time repeated: 10.5 ms
        // against 6.0 without it and 7.5 scattered), so such a curve is scattered.
        if (on && close > 0) {
            long long shared = 0;
            for (long long i = tid; i + 1 < n; i += kTableBlock)
                shared += cell_units(sdt[staged_pos(i, n_full)], scale) >> kOffBits ==
                                  cell_units(sdt[staged_pos(i + 1, n_full)], scale) >> kOffBits
                              ? 1 : 0;
            on = tb_sum(shared, sh) <= most_shared;
        }
    }
    if (on) {
        const int bl = bitlen64(n);
        // the padding copy can repeat every point once: counts below 2^(bl + 1), flux
        // sums within twice the absolute total
        sg.g_bl = bl + 1;
        const long long c_last = (long long)(cell_units(sdt[staged_pos(n - 1, n_full)], scale) >> kOffBits);
        const int ncol = (int)(c_last / rows) + 3;
        const int pitch = (ncol + (GEOM == ATB_GEOM_BINNED ? kRowPad : 0) + 7) / 8 * 8;
        sg.g_rows = rows;
        sg.g_pitch = pitch;
        sg.g_colmax = ncol - 2;
        sg.g_scale = scale;
        unsigned* idx = ga.idx + ga.cell_off[c];
        Entry<true>* e1 = reinterpret_cast<Entry<true>*>(ga.tab + ga.cell_off[c] * (16 * ga.vs));
        Entry<false>* e2 = reinterpret_cast<Entry<false>*>(e1);
        unsigned* bits = GEOM == ATB_GEOM_BINNED ? ga.bits + ga.bit_off[c] : nullptr;
        const int bsh = offset_shift(bl);
        const bool pk = st.cnt_win != 0;
        if (GEOM == ATB_GEOM_BINNED) {
            for (long long k = tid; k < offset_words(bl); k += kTableBlock) bits[k] = 0u;
            __syncthreads();
        }
        const int lane = tid & 31;
        long long bx = 0, by = 0, multi = 0;
        auto put = [&](long long cell, unsigned o, long long x, long long y, long long i, int qw,
                       int qy) {
            const int p = (int)(cell % rows) * pitch + (int)(cell / rows);
            idx[p] = (unsigned)i;
            if (pk)
                e1[p] = Entry<true>{(unsigned long long)x, o, qy};
            else
                e2[p] = Entry<false>{(unsigned long long)x, (unsigned long long)y, o, qw, qy, 0};
        };
        // point i writes the cells after point i-1's up to its own
        for (long long i0 = 0; i0 < n; i0 += kTableBlock) {
            const long long i = i0 + tid;
            long long x = 0, y = 0;
            int qw = 0, qy = 0;
            unsigned long long u = 0;
            long long prev = -1, next = -1;
            if (i < n) {
                const long long q = staged_pos(i, n_full);
                staged_words(st, a.sqw + so, a.sqy + so, q, qw, qy);
                point_words(sg, qw, qy, x, y);
                u = cell_units(sdt[q], scale);
                if (i > 0) prev = (long long)(cell_units(sdt[staged_pos(i - 1, n_full)], scale) >> kOffBits);
                if (i + 1 < n)
                    next = (long long)(cell_units(sdt[staged_pos(i + 1, n_full)], scale) >> kOffBits);
            }
            long long tx, ty;
            tb_scan2(x, y, tx, ty, sh);
            x += bx;
            y += by;
            bx += tx;
            by += ty;
            const long long cell = (long long)(u >> kOffBits);
            long long beg = prev + 1, end = i < n ? cell : -1;  // empty cells [beg, end)
            if (i < n) {
                unsigned o = (unsigned)(u & kOffMask);
                if (GEOM == ATB_GEOM_BINNED && o - kOffMid + 1u <= 2u && cell % rows == 0) {
                    // on boundary (0, cell / rows): see kOffMid
                    const int slot = max(trunc1_magic(sdt[staged_pos(i, n_full)] * st.inv_bin_dur), 1);
                    o = slot <= (int)(cell / rows) ? min(o, kOffMid - 1u) : max(o, kOffMid);
                }
                if (cell == prev) ++multi;
                else put(cell, next == cell ? kOffMulti : o, x, y, i, qw, qy);
                if (GEOM == ATB_GEOM_BINNED)
                    for (int d = -1; d <= 1; ++d) {  // neighbours wrap into the next cell
                        const unsigned b = (((unsigned)u + (unsigned)d) & kOffMask) >> bsh;
                        atomicOr(bits + (b >> 5), 1u << (b & 31u));
                    }
            }
            if (beg < end && end - beg <= 16) {
                for (long long k = beg; k < end; ++k) put(k, kOffMask, x, y, i, 0, 0);
                end = beg;
            }
            unsigned wide = __ballot_sync(0xffffffffu, beg < end);
            while (wide) {  // long gaps: the whole warp writes
                const int l = __ffs(wide) - 1;
                wide &= wide - 1;
                const long long kb = __shfl_sync(0xffffffffu, beg, l);
                const long long ke = __shfl_sync(0xffffffffu, end, l);
                const long long gx = __shfl_sync(0xffffffffu, x, l);
                const long long gy = __shfl_sync(0xffffffffu, y, l);
                const long long gi = __shfl_sync(0xffffffffu, i, l);
                for (long long k = kb + lane; k < ke; k += 32) put(k, kOffMask, gx, gy, gi, 0, 0);
            }
        }
        for (long long k = c_last + 1 + tid; k < (long long)ncol * rows; k += kTableBlock)
            put(k, kOffMask, bx, by, n, 0, 0);
        multi = tb_sum(multi, sh);
        // fixed bins: a point at the first or last unit of its cell may decide a
        // boundary of the neighbouring cell, which is marked to be decided exactly
        // (astropy bins: the boundary's offset is common to a cycle and checked there)
        if (GEOM == ATB_GEOM_FIXED) {
            __syncthreads();
            for (long long i = tid; i < n; i += kTableBlock) {
                const unsigned long long u = cell_units(sdt[staged_pos(i, n_full)], scale);
                const unsigned o = (unsigned)(u & kOffMask);
                const long long cell = (long long)(u >> kOffBits);
                for (int d = -1; d <= 1; d += 2) {
                    if (o != (d < 0 ? 0u : kOffMask) || cell + d < 0) continue;
                    if (pk) e1[cell + d].off = kOffMulti;
                    else e2[cell + d].off = kOffMulti;
                }
            }
        }
        if (multi > most_shared) on = false;  // (spacings just below the cell's width)
        if (tid == 0) {
            if (pk) gather_consts<true>(sg, curve_total<true>(sg), sg.gk);
            else gather_consts<false>(sg, curve_total<false>(sg), sg.gk);
        }
    }
    __syncthreads();  // (every thread has read stats[c])
    if (!on)
        for (long long i = tid; i < np; i += kTableBlock) a.scatter[a.flag_off[c] + i] = 1;
    if (tid == 0) {
        sg.g_on = on ? 1 : 0;
        stats[c] = sg;
        if (on) atomicAdd(ga.n_gather + (st.cnt_win ? 0 : 1), (unsigned long long)sg.n_g);
        else atomicOr(ga.n_scatter, 1);
    }
}

// ----------------------------------------------------------------------------
// gather search
// ----------------------------------------------------------------------------

// A finished period: its winning window and exact sums; written out by
// gather_flush, one lane per period.
template <bool PK>
struct GatherResult {
    Sum<PK> d, tot;
    int key;
};

// A period to search (set up one lane each).
struct GatherPeriod {
    double P, IP, Ps;  // Ps: table units per period
    int NB, jlook, K;  // bins; last boundary looked up; cycles
    int period;        // index in the curve's grid
    int sure0;         // astropy bins: cycle 0 needs no checks
};

constexpr int kMaxRing = 1024;  // longest buffer of prefix entries (fixed bins)
constexpr int kMaxPop = 4;    // periods of a tile a warp sets up together
constexpr int kMaxCyc = 64;   // cycles whose table positions a warp holds
constexpr int kMaxList = 64;  // windows within reach of the best, before the exact test

// What the filter of one period knows.  `lim` is a lower bound, in filter units,
// of a ratio some window of the period reaches: a window whose upper bound is
// below it cannot win.
struct FilterState {
    float lim;
    float eA;      // astropy bins: e0; fixed bins: the whole error bound E of the period
    float wE, wN;  // GatherConsts
};

// Shared memory of one warp besides its prefix entries.
template <bool PK>
struct WarpState {
    Sum<PK> head[kHeadMax + 1];  // first prefix sums, the source of the V42 padding
    GatherResult<PK> res[kMaxPop];
    GatherPeriod per[kMaxPop];
    GatherConsts k;              // of a fixed-bin period with points in the trash slot
    int2 cyc[kMaxCyc + 1];       // astropy bins: table position of boundary (k, 0), see fill_cycles
    float2 list[kMaxList];       // (upper bound, key bits) of windows that may win
    int n_list;                  // -1: more than the list holds
    int len[kMaxDur];            // window lengths
    // the period being searched (in shared memory: the look-up loop needs the registers)
    Sum<PK> A0, tot;             // sum before boundary 0; totals
    Sum<PK> cm1, hnb;            // astropy bins: C[M-1] and C[NB] - C[NB-1] of the padding copy
    FilterState f;
    float wm;                    // GatherConsts; weighted curves only
    float guess;                 // see gather_period
    const TableStat* st;
    const Entry<PK>* tab;
    const unsigned* idx;
    const double* sdt;
    const int* sqw;
    const int* sqy;
    const unsigned* bits;
    long long n_full;
    int rows, pitch, colmax, bsh, gmul;
    unsigned cinc;
};

// a warp's prefix entries, with room for the NaN entry after a full buffer
__host__ __device__ inline unsigned gather_ring_bytes(int ring) { return 8u * (ring + 2); }

__host__ __device__ inline int gather_state_bytes(int vs) {
    return (int)(vs == 1 ? sizeof(WarpState<true>) : sizeof(WarpState<false>)) / 16 * 16 + 16;
}

// dynamic shared memory of a CTA of the gather kernel
inline int gather_smem_bytes(int ring, int vs) {
    return kGatherWarps * ((int)gather_ring_bytes(ring) + gather_state_bytes(vs));
}

// Look-up of the boundary at offset f of an entry's cell: V before the cell,
// plus the cell's point when it lies before the boundary.
__device__ __forceinline__ void add_entry(Sum<true>& s, const uint4& w, unsigned f, int gmul,
                                          unsigned cinc) {
    const bool b = w.z < f;
    s.x += ((unsigned long long)w.y << 32 | w.x) + ((unsigned long long)(b ? cinc : 0u) << 32);
    s.x += (unsigned long long)((long long)(int)w.w * (b ? gmul : 0));
}
__device__ __forceinline__ void add_entry(Sum<false>& s, const uint4& w, const uint4& u,
                                          unsigned f) {
    const int b = u.x < f ? 1 : 0;
    s.x += ((unsigned long long)w.y << 32 | w.x) + (unsigned long long)((long long)(int)u.y * b);
    s.y += ((unsigned long long)w.w << 32 | w.z) + (unsigned long long)((long long)(int)u.z * b);
}

// The points before boundary (k, j) decided by the fold's own formula: starting
// from the table's cell, walk to the first point whose (cycle, slot) is beyond
// (k, j), correcting the running sum.
template <int GEOM, bool PK>
__device__ __noinline__ Sum<PK> gather_exact(const WarpState<PK>* ws, int i_per, int k, int j,
                                             int cell) {
    const TableStat& st = *ws->st;
    const double P = ws->per[i_per].P, IP = ws->per[i_per].IP;
    const int NB = ws->per[i_per].NB;
    const double kd = (double)k;
    auto before = [&](double d) {
        const double m = d * IP;
        const double kk = floor(m);
        if (kk != kd) return kk < kd;
        if (GEOM == ATB_GEOM_BINNED)
            return min(max(trunc1_magic(fma(-P, kk, d) * st.inv_bin_dur), 1), NB) <= j;
        return (int)min((unsigned)trunc1_magic((m - kk) * (double)NB), (unsigned)NB + 1u) <= j;
    };
    auto words = [&](int i) {
        int qw, qy;
        long long x, y;
        staged_words(st, ws->sqw, ws->sqy, staged_pos(i, ws->n_full), qw, qy);
        point_words(st, qw, qy, x, y);
        Sum<PK> s;
        s.x = (unsigned long long)x;
        if constexpr (!PK) s.y = (unsigned long long)y;
        return s;
    };
    Sum<PK> s;
    s.x = ws->tab[cell].x;
    if constexpr (!PK) s.y = ws->tab[cell].y;
    int i = (int)ws->idx[cell];
    const int n = st.g_n;
    while (i > 0 && !before(ws->sdt[staged_pos(i - 1, ws->n_full)])) s.sub(words(--i));
    while (i < n && before(ws->sdt[staged_pos(i, ws->n_full)])) s.add(words(i++));
    return s;
}

// The look-up with every check: offsets within one unit of the boundary's (three: an
// entry's offset may have been moved by two, see kOffMid),
// cells with several points, and -- astropy bins -- boundaries at the ends of
// their cells, whose point may lie in the neighbouring one, are decided exactly.
template <int GEOM, bool PK>
__device__ __noinline__ Sum<PK> gather_checked(const WarpState<PK>* ws, int ip, int k, int j,
                                                  int cell, unsigned f) {
    const Entry<PK> e = ws->tab[cell];
    if (e.off - f + 3u <= 6u || e.off > kOffMask ||
        (GEOM == ATB_GEOM_BINNED && (f == 0 || f == kOffMask)))
        return gather_exact<GEOM, PK>(ws, ip, k, j, cell);
    Sum<PK> s;
    s.x = e.x;
    if constexpr (PK) {
        if (e.off < f) {
            long long x, y;
            point_words(*ws->st, 1, e.q, x, y);
            s.x += (unsigned long long)x;
        }
    } else {
        s.y = e.y;
        if (e.off < f) {
            s.x += (unsigned long long)(long long)e.qw;
            s.y += (unsigned long long)(long long)e.qy;
        }
    }
    return s;
}

// Table position of boundary (k, 0) in an astropy-binned table: column, row, offset.
__device__ __forceinline__ void cycle_cell(int k, double Ps, unsigned rows, int& col, int& row,
                                           unsigned& f) {
    const unsigned long long u =
        (unsigned long long)__double2ll_rd(fma((double)k, Ps, kOffHalf));
    const unsigned cell = (unsigned)(u >> kOffBits);
    const unsigned q = cell / rows;
    col = (int)q;
    row = (int)(cell - q * rows);
    f = (unsigned)u & kOffMask;
}

// Table position of boundary (k, j) with fixed bins.
__device__ __forceinline__ void fixed_cell(double kd, double Ps, double xj, int colmax, int& cell,
                                           unsigned& f) {
    // 2^52 + floor(x): the integer is in the low 52 bits
    const double u = __dadd_rd(fma(kd, Ps, xj), 4503599627370496.0);
    const unsigned lo = (unsigned)__double2loint(u), hi = (unsigned)__double2hiint(u) & 0xfffffu;
    cell = (int)min(__funnelshift_r(lo, hi, kOffBits), (unsigned)colmax);
    f = lo & kOffMask;
}

constexpr int kCareful = 1 << 30;  // of cyc[].y

// whether some point's offset may lie within one unit of f
template <bool PK>
__device__ __forceinline__ bool near_point(const WarpState<PK>& ws, unsigned f, int bsh) {
    const unsigned b = f >> bsh;
    return (ws.bits[b >> 5] >> (b & 31u)) & 1u;
}

// cyc[q] = (entry index, offset | kCareful) of cycles k0 + q < k1, whose look-ups
// all lie inside the table.  A cycle whose offset may lie within one unit of
// some point's (`bits`: a bit per 2^bsh offsets) is looked up with every check.
template <bool PK>
__device__ __noinline__ void fill_cycles(WarpState<PK>& ws, int k0, int k1, double Ps, int sure0) {
    const int lane = threadIdx.x & 31;
    const int rows = ws.rows, pitch = ws.pitch, bsh = ws.bsh;
    for (int k = k0 + lane; k < k1; k += 32) {
        int col, row;
        unsigned f;
        cycle_cell(k, Ps, (unsigned)rows, col, row, f);
        const bool care = !(sure0 && k == 0) && near_point<PK>(ws, f, bsh);
        ws.cyc[k - k0] = make_int2(row * pitch + col, (int)f | (care ? kCareful : 0));
    }
}

// Sums over all K cycles of V before the boundaries jb + 32 m + lane (m < J);
// boundaries beyond jlook give values nobody uses.
template <int GEOM, bool PK, int J>
__device__ __forceinline__ void gather_block(WarpState<PK>& ws, int ip, int jb,
                                             Sum<PK> (&acc)[J]) {
    const int jl = jb + (int)(threadIdx.x & 31);
    const uint4* tab = reinterpret_cast<const uint4*>(ws.tab);
    const int K = ws.per[ip].K, colmax = ws.colmax, gmul = ws.gmul;
    const unsigned cinc = ws.cinc;
#pragma unroll
    for (int m = 0; m < J; ++m) {
        acc[m].x = 0;
        if constexpr (!PK) acc[m].y = 0;
    }
    if constexpr (GEOM == ATB_GEOM_BINNED) {
        for (int kb = 0; kb < K - 1; kb += kMaxCyc) {
            const int ke = min(kMaxCyc, K - 1 - kb);
            if (K - 1 > kMaxCyc) {  // refilled for every block
                __syncwarp();
                fill_cycles<PK>(ws, kb, kb + ke, ws.per[ip].Ps, ws.per[ip].sure0);
                __syncwarp();
            }
#pragma unroll 1
            for (int q = 0; q < ke; ++q) {
                const int2 e = ws.cyc[q];
                const unsigned f = (unsigned)e.y & kOffMask;
                if (!(e.y & kCareful)) {
                    const uint4* p = tab + (PK ? 1 : 2) * (e.x + jl);
                    if constexpr (PK) {
                        uint4 w[J];
#pragma unroll
                        for (int m = 0; m < J; ++m) w[m] = __ldg(p + 32 * m);
#pragma unroll
                        for (int m = 0; m < J; ++m) add_entry(acc[m], w[m], f, gmul, cinc);
                    } else {
                        uint4 w[J], u[J];
#pragma unroll
                        for (int m = 0; m < J; ++m) {
                            w[m] = __ldg(p + 64 * m);
                            u[m] = __ldg(p + 64 * m + 1);
                        }
#pragma unroll
                        for (int m = 0; m < J; ++m) add_entry(acc[m], w[m], u[m], f);
                    }
                } else {
                    const int jlook = ws.per[ip].jlook;
#pragma unroll
                    for (int m = 0; m < J; ++m)
                        if (jl + 32 * m <= jlook)
                            acc[m].add(gather_checked<GEOM, PK>(&ws, ip, kb + q, jl + 32 * m,
                                                                e.x + jl + 32 * m, f));
                }
            }
        }
        // the last cycle: boundaries beyond the table see every point
        const int2 e = ws.cyc[kMaxCyc];
        const unsigned f = (unsigned)e.y & kOffMask;
        const int base = ((e.y & ~kCareful) >> kOffBits) * ws.pitch, jlook = ws.per[ip].jlook;
#pragma unroll
        for (int m = 0; m < J; ++m) {
            const int j = min(jl + 32 * m, jlook);
            const int ix = base + min(e.x + j, colmax);
            if (e.y & kCareful) {
                acc[m].add(gather_checked<GEOM, PK>(&ws, ip, K - 1, j, ix, f));
            } else if constexpr (PK) {
                add_entry(acc[m], __ldg(tab + ix), f, gmul, cinc);
            } else {
                add_entry(acc[m], __ldg(tab + 2 * ix), __ldg(tab + 2 * ix + 1), f);
            }
        }
    } else {
        const double Ps = ws.per[ip].Ps;
        const int NB = ws.per[ip].NB;
        double xj[J];
#pragma unroll
        for (int m = 0; m < J; ++m)
            xj[m] = (double)min(jl + 32 * m, NB) / (double)NB * Ps + kOffHalf;
        double kd = 0.0;
#pragma unroll 1
        for (int k = 0; k < K; ++k, kd += 1.0) {
            int ix[J];
            unsigned f[J], close = 0xffffffffu, top = 0u;
            uint4 w[J], u[J];
#pragma unroll
            for (int m = 0; m < J; ++m) {
                fixed_cell(kd, Ps, xj[m], colmax, ix[m], f[m]);
                w[m] = __ldg(tab + (PK ? 1 : 2) * ix[m]);
                if constexpr (!PK) u[m] = __ldg(tab + 2 * ix[m] + 1);
            }
#pragma unroll
            for (int m = 0; m < J; ++m) {
                if constexpr (PK) add_entry(acc[m], w[m], f[m], gmul, cinc);
                else add_entry(acc[m], w[m], u[m], f[m]);
                const unsigned o = PK ? w[m].z : u[m].x;
                close = min(close, o - f[m] + 1u);
                top |= o;
            }
            if (close <= 2u || top > kOffMask) {
#pragma unroll
                for (int m = 0; m < J; ++m) {
                    const unsigned o = PK ? w[m].z : u[m].x;
                    if (o - f[m] + 1u <= 2u || o > kOffMask) {
                        Sum<PK> s;
                        s.x = 0;
                        if constexpr (PK) {
                            add_entry(s, w[m], f[m], gmul, cinc);
                        } else {
                            s.y = 0;
                            add_entry(s, w[m], u[m], f[m]);
                        }
                        acc[m].sub(s);
                        acc[m].add(gather_exact<GEOM, PK>(&ws, ip, k, min(jl + 32 * m, NB), ix[m]));
                    }
                }
            }
        }
    }
}

// Prefix sum C[j] of the finished period, gathered again by the whole warp (lanes
// over cycles): A(j) - A(0), or the total beyond the last boundary.
template <int GEOM, bool PK>
__device__ __noinline__ Sum<PK> prefix_at(const WarpState<PK>* ws, int ip, int j, Sum<PK> A0) {
    const TableStat& st = *ws->st;
    const GatherPeriod& g = ws->per[ip];
    if (j > g.jlook) return curve_total<PK>(st);
    Sum<PK> s;
    s.x = 0;
    if constexpr (!PK) s.y = 0;
    for (int k = threadIdx.x & 31; k < g.K; k += 32) {
        int cell;
        unsigned f;
        if (GEOM == ATB_GEOM_BINNED) {
            int col, row;
            cycle_cell(k, g.Ps, (unsigned)st.g_rows, col, row, f);
            cell = row * st.g_pitch + min(col + j, st.g_colmax);
        } else {
            fixed_cell((double)k, g.Ps, (double)j / (double)g.NB * g.Ps + kOffHalf, st.g_colmax,
                       cell, f);
        }
        s.add(gather_checked<GEOM, PK>(ws, ip, k, j, cell, f));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Sum<PK> t;
        t.x = __shfl_xor_sync(0xffffffffu, s.x, o);
        if constexpr (!PK) t.y = __shfl_xor_sync(0xffffffffu, s.y, o);
        s.add(t);
    }
    s.sub(A0);
    return s;
}

// Exact sums of window `key` (warp-wide).  Astropy bins: entries M = NB - os and
// beyond hold the padding copy (vbls_v42_parity.cu:78-80), on prefix sums
//   C'[M+m] = C[M-1] + C[1+m],  C'[NB] = C'[NB-1] + (C[NB] - C[NB-1]).
template <int GEOM, bool PK>
__device__ __noinline__ Sum<PK> window_sums(const WarpState<PK>* ws, int ip, int key, int nd,
                                            int os, Sum<PK> A0, Sum<PK> tot) {
    const int s = key / nd, NB = ws->per[ip].NB, M = NB - os;
    int e = s + ws->len[key % nd];
    auto prefix = [&](int j) {
        if (GEOM == ATB_GEOM_FIXED || j < M) return prefix_at<GEOM, PK>(ws, ip, j, A0);
        Sum<PK> v = prefix_at<GEOM, PK>(ws, ip, M - 1, A0);
        v.add(ws->head[j < NB ? j - M + 1 : os]);
        if (j == NB) {
            v.add(tot);
            v.sub(prefix_at<GEOM, PK>(ws, ip, NB - 1, A0));
        }
        return v;
    };
    Sum<PK> d;
    if (GEOM == ATB_GEOM_FIXED && e > NB) {
        d = prefix(e - NB);
        d.add(tot);
    } else {
        d = prefix(e);
    }
    d.sub(prefix(s));
    return d;
}

// A prefix entry of the filter: astropy bins (g + 2^-21 |g|, c), fixed bins (g, c).
template <int GEOM, bool PK>
__device__ __forceinline__ float2 filter_entry(const Sum<PK>& s, float f1, int bl, int sh) {
    float c, y;
    if constexpr (PK) {
        const unsigned lo = (unsigned)s.x, hi = (unsigned)(s.x >> 32);
        y = (float)(int)__funnelshift_l(lo, hi, bl);
        c = (float)((hi + (1u << (31 - bl))) >> (32 - bl));
    } else {
        y = (float)(int)((long long)s.y >> sh);
        c = (float)(unsigned)(s.x >> sh);
    }
    const float g = __fmaf_rn(f1, c, -y);
    return make_float2(GEOM == ATB_GEOM_BINNED ? __fmaf_rn(4.76837158203125e-07f, fabsf(g), g) : g,
                       c);
}

// prefix entries by their 32-bit shared address
__device__ __forceinline__ float2 ent_load(unsigned addr) {
    float2 r;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(addr));
    return r;
}
__device__ __forceinline__ void ent_store(unsigned addr, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
// entry + n in one packed addition; n packed by ent_pack
__device__ __forceinline__ unsigned long long ent_pack(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 ent_add(unsigned addr, unsigned long long n) {
    unsigned long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(v), "l"(n));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// The exact test of the scan path: (num, den), or num = -1 when the window is skipped.
template <int GEOM, bool PK>
__device__ __noinline__ float2 exact_window(const TableStat* st, const GatherConsts* k, Sum<PK> d) {
    WinConsts kc;
    kc.wtot = k->wtot;
    kc.ytot = k->ytot;
    kc.c1 = k->c1;
    kc.fN = k->fN;
    kc.thr = 0.0;  // below one unit (checked when the table was made)
    kc.qw0s = 0.0;
    const double sy2 = ldexp(1.0, -st->ey);
    float num, den;
    bool ok;
    if constexpr (PK)
        ok = window_eval_cnt<GEOM, true>((float)packed_count(d.x, st->g_bl),
                                         (double)packed_flux(d.x, st->g_bl, st->g_guard) * sy2, kc,
                                         num, den);
    else
        ok = window_eval<GEOM, true>((double)(long long)d.x * ldexp(1.0, -st->ew),
                                     (double)(long long)d.y * sy2, kc, num, den);
    return ok && num >= 0.0f ? make_float2(num, den) : make_float2(-1.0f, 1.0f);
}

// The rare step after some lane's windows at start s (lengths k0, k0 + 1) passed
// the filter: raise the bound and list the windows that may still win.  base, last:
// addresses of the buffer's entry of bin 0 and of the entry after the last.
template <int GEOM, bool PK>
__device__ __noinline__ float gather_pass(WarpState<PK>* ws, unsigned base, unsigned last, int s,
                                          bool ok, int k0, int k1) {
    const int lane = threadIdx.x & 31;
    FilterState f = ws->f;
    float wm = 0.0f;
    if constexpr (!PK) wm = ws->wm;
    const int nd = ws->st->n_dur;
    const float up = 1.0f + 3.814697265625e-06f, dn = 1.0f - 3.814697265625e-06f;  // 2^-18
    const unsigned as = base + 8u * (unsigned)s;
    const float2 e0 = ent_load(min(as, last));
    for (int q = k0; q < k1; ++q) {
        const float2 e1 = ent_load(min(as + 8u * (unsigned)min(ws->len[q], 1 << 24), last));
        const float dw = e1.y - (e0.y + f.wE);
        float t, lo;  // bounds of sigma (fixed bins: of |sigma|)
        if (GEOM == ATB_GEOM_BINNED) {
            t = (e1.x - e0.x) + fmaf(1.0e-6f, fabsf(e0.x), f.eA);
            lo = t - 2.0f * fmaf(1.0e-6f, fabsf(e0.x) + fabsf(e1.x), f.eA);
        } else {
            const float dg = fabsf(e1.x - e0.x);
            t = dg + f.eA;
            lo = dg - f.eA;
        }
        const float den0 = dw * (f.wN - dw);
        // weighted: a window holds a point, or is none; with fixed bins, whose windows
        // count no point twice, so does the rest of the curve
        float den = den0;
        if constexpr (!PK) {
            const float di = fmaxf(dw, wm);
            den = di * (GEOM == ATB_GEOM_BINNED ? f.wN - di : fmaxf(f.wN - di, wm));
        }
        const float num = GEOM == ATB_GEOM_BINNED ? t * fabsf(t) : t * t;
        // An entry beyond the last is NaN: no window.  No weight inside or outside is
        // none either (the padding copy can put more than the total inside).
        const bool in = ok && (PK ? den > 0.0f : f.wN - dw > -4.0f * f.wE) &&
                        num >= f.lim * dn * den;
        if (!__any_sync(0xffffffffu, in)) continue;
        float l = 0.0f, hi = INFINITY;
        if (den > 0.0f) {
            hi = __fdividef(num, den) * up;
            // den0 of weighted curves is low by at most 2 wE (wN + 4 wE)
            const float den_hi = PK ? den : fmaf(2.0f * f.wE, f.wN + 4.0f * f.wE, den0) * up;
            if (in && lo > 0.0f && den0 > 0.0f) l = __fdividef(lo * lo, den_hi) * dn;
        }
        // non-negative floats order like their bit patterns
        f.lim = fmaxf(f.lim, __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(l))));
        const unsigned who = __ballot_sync(0xffffffffu, in && hi >= f.lim);
        const int n = ws->n_list;
        if (n < 0) return f.lim;
        int at = n;
        if (n + __popc(who) > kMaxList) {  // drop what can no longer win
            at = 0;
            for (int i = 0; i < n; i += 32) {
                const float2 v = i + lane < n ? ws->list[i + lane] : make_float2(-1.0f, 0.0f);
                const unsigned keep = __ballot_sync(0xffffffffu, v.x >= f.lim);
                if (v.x >= f.lim) ws->list[at + __popc(keep & ((1u << lane) - 1u))] = v;
                at += __popc(keep);
                __syncwarp();
            }
        }
        const bool full = at + __popc(who) > kMaxList;
        if (!full && (who >> lane & 1u))
            ws->list[at + __popc(who & ((1u << lane) - 1u))] =
                make_float2(hi, __int_as_float(s * nd + q));
        __syncwarp();
        if (lane == 0) {
            ws->n_list = full ? -1 : at + __popc(who);
            ws->f.lim = f.lim;
        }
        __syncwarp();
        if (full) return f.lim;
    }
    return f.lim;
}

// Windows of the starts [s_beg, s_end), whose prefix entries are in the buffer; two
// starts per lane and two lengths at a time.  A window's score is
// sigma^2 / (dw (wN - dw)); it can only beat `lim` when
//   r = t |t| - lim dw (wN - dw) >= 0
// with t an upper bound of sigma, evaluated as two fused multiply-adds (weighted:
// dw no less than wm, see GatherConsts).  The entry
// at `last`, where longer windows end, is NaN, and r is too.
// (Out of line, KC = 3 for every call: copies of this loop specialised by caller,
// number of lengths and range made the kernel miss the instruction cache.)
template <int GEOM, bool PK, int KC>
__device__ __noinline__ void gather_windows(WarpState<PK>* ws, unsigned base, unsigned last,
                                            int nd, int k0, int s_beg, int s_end) {
    const int lane = threadIdx.x & 31;
    FilterState f = ws->f;
    float wm = 0.0f;
    if constexpr (!PK) wm = ws->wm;
    unsigned l8[KC];
#pragma unroll
    for (int q = 0; q < KC; ++q) l8[q] = 8u * (unsigned)min(ws->len[min(k0 + q, nd - 1)], 1 << 24);
    for (int s0 = s_beg; s0 < s_end; s0 += 64) {
        // (1 - 2^-20): the rounding of lim * wN - lim * dw stays on the safe side
        const float lN = -f.lim * f.wN * 0.99999904632568359375f;
        float lm = 0.0f;
        if constexpr (!PK) lm = -f.lim * wm * 0.99999904632568359375f;
        float top[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const unsigned as = base + 8u * (unsigned)(s0 + 32 * i + lane);
            const float2 e0 = ent_load(min(as, last));
            const unsigned long long n =
                ent_pack(GEOM == ATB_GEOM_BINNED ? fmaf(1.0e-6f, fabsf(e0.x), f.eA) - e0.x : -e0.x,
                         -(e0.y + f.wE));
            top[i] = -1.0f;
#pragma unroll
            for (int q = 0; q < KC; ++q) {
                const float2 v = ent_add(min(as + l8[q], last), n);
                const float t = GEOM == ATB_GEOM_BINNED ? v.x : fabsf(v.x) + f.eA;
                float dw = v.y;
                if constexpr (!PK) dw = fmaxf(dw, wm);
                float a = fmaf(f.lim, dw, lN);
                if (!PK && GEOM == ATB_GEOM_FIXED) a = fminf(a, lm);
                const float r = fmaf(a, dw, GEOM == ATB_GEOM_BINNED ? t * fabsf(t) : t * t);
                top[i] = fmaxf(top[i], r);
            }
        }
        const bool p0 = top[0] >= 0.0f && s0 + lane < s_end;
        const bool p1 = top[1] >= 0.0f && s0 + 32 + lane < s_end;
        if (__any_sync(0xffffffffu, p0 || p1)) {
#pragma unroll 1
            for (int i = 0; i < 2; ++i) {
                const bool ok = i ? p1 : p0;
                if (__any_sync(0xffffffffu, ok))
                    f.lim = gather_pass<GEOM, PK>(ws, base, last, s0 + 32 * i + lane, ok, k0,
                                                  min(k0 + KC, nd));
            }
        }
    }
}

template <int GEOM, bool PK>
__device__ __forceinline__ void gather_starts(WarpState<PK>* ws, unsigned base, unsigned last,
                                              int nd, int s_beg, int s_end) {
    int k0 = 0;
    for (; k0 < nd; k0 += 3)
        gather_windows<GEOM, PK, 3>(ws, base, last, nd, k0, s_beg, s_end);
}

// The windows of fixed bins, once every prefix entry is in the buffer.
template <int GEOM, bool PK>
__device__ __noinline__ void fixed_windows(WarpState<PK>* ws, unsigned fb, int NB) {
    const TableStat* st = ws->st;
    const int lane = threadIdx.x & 31, nd = st->n_dur;
    const Sum<PK> all = curve_total<PK>(*st), tot = ws->tot;
    const GatherConsts* gk = &st->gk;
    bool some, same = tot.x == all.x;
    if constexpr (PK) {
        some = packed_count(tot.x, st->g_bl) != 0;
    } else {
        some = tot.x != 0;
        same = same && tot.y == all.y;
    }
    if (!some) return;
    float df = 0.0f, eA = gk->e0;
    if (!same) {  // points in the trash slot: the period's own totals
        if (lane == 0) {
            gather_consts<PK>(*st, tot, ws->k);
            ws->f.wN = ws->k.wN;
            ws->f.wE = fmaxf(gk->wE, ws->k.wE);
        }
        __syncwarp();
        df = ws->k.f1 - gk->f1;  // entries g = f1 c - y with the other f1
        eA = 2.0f * fmaxf(eA, ws->k.e0);
    } else if (lane == 0) {
        ws->k = *gk;
    }
    // windows that wrap end at entries NB + 1 .. NB + lm: the first ones plus
    // the totals; then the NaN entry, where windows as long as the period end
    int lm = 0;
    for (int k = 0; k < nd; ++k) lm = max(lm, ws->len[k] < NB ? ws->len[k] : 0);
    const float2 vT = ent_load(fb + 8u * (unsigned)NB);
    __syncwarp();
    float gmax = fabsf(vT.x);
    for (int j = lane; j <= NB; j += 32) {
        float2 v = ent_load(fb + 8u * (unsigned)j);
        gmax = fmaxf(gmax, fabsf(v.x));
        v.x = fmaf(df, v.y, v.x);
        gmax = fmaxf(gmax, fabsf(v.x));
        if (df != 0.0f) ent_store(fb + 8u * (unsigned)j, v);
        if (j >= 1 && j <= lm)
            ent_store(fb + 8u * (unsigned)(NB + j),
                      make_float2(v.x + fmaf(df, vT.y, vT.x), v.y + vT.y));
    }
    const unsigned last = fb + 8u * (unsigned)(NB + lm + 1);
    gmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(gmax)));
    if (lane == 0) {
        ent_store(last, make_float2(NAN, 0.0f));
        ws->f.eA = fmaf(3.814697265625e-06f, gmax, eA);  // 2^-18 gmax: up to four roundings
    }
    if (lane < nd && ws->len[lane] >= NB) ws->len[lane] = kLenCap;
    __syncwarp();
    gather_starts<GEOM, PK>(ws, fb, last, nd, 0, NB);
}

// The winner among the listed windows: alone within reach of `lim` it wins
// without the exact test (the window that gave `lim` is in the list).
template <int GEOM, bool PK>
__device__ __noinline__ void gather_winner(WarpState<PK>* ws, int ip, int os) {
    const int lane = threadIdx.x & 31, n = ws->n_list, nd = ws->st->n_dur;
    const float lim = ws->f.lim;
    const GatherConsts* gk = GEOM == ATB_GEOM_FIXED ? &ws->k : &ws->st->gk;
    unsigned live[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
        live[i] = __ballot_sync(0xffffffffu, 32 * i + lane < n && ws->list[32 * i + lane].x >= lim);
    const bool alone = __popc(live[0]) + __popc(live[1]) == 1 && lim > 0.0f;
    Cand win{-1.0f, 1.0f, 0x7fffffff};
    Sum<PK> wd = ws->tot;
#pragma unroll 1
    while (live[0] | live[1]) {
        const int b = live[0] ? __ffs(live[0]) - 1 : 32 + __ffs(live[1]) - 1;
        if (live[0]) live[0] &= live[0] - 1;
        else live[1] &= live[1] - 1;
        const int key = __float_as_int(ws->list[b].y);
        const Sum<PK> d = window_sums<GEOM, PK>(ws, ip, key, nd, os, ws->A0, ws->tot);
        if (alone) {
            win.key = key;
            wd = d;
        } else {
            const float2 w = exact_window<GEOM, PK>(ws->st, gk, d);
            if (w.x >= 0.0f && cand_better(w.x, w.y, key, win.num, win.den, win.key)) {
                win = Cand{w.x, w.y, key};
                wd = d;
            }
        }
    }
    if (lane == 0) {
        GatherResult<PK>& r = ws->res[ip];
        r.d = wd;
        r.tot = ws->tot;
        r.key = win.key;
    }
    __syncwarp();
}

// Prefix sums C[jb ..] of one block into the filter's buffer at bin s_done + ...
template <int GEOM, bool PK, int J>
__device__ __forceinline__ void gather_step(WarpState<PK>& ws, unsigned fb, int ip, int jb,
                                            int s_done, int os) {
    const int lane = threadIdx.x & 31;
    Sum<PK> acc[J];
    gather_block<GEOM, PK, J>(ws, ip, jb, acc);
    const TableStat* st = ws.st;
    const int NB = ws.per[ip].NB, bl = st->g_bl, sh = flux_shift<PK>(*st);
    const float f1 = st->gk.f1;
    if (jb == 0) {
        if (lane == 0) ws.A0 = acc[0];
        __syncwarp();
    }
    const Sum<PK> A0 = ws.A0;
#pragma unroll
    for (int m = 0; m < J; ++m) acc[m].sub(A0);
    if constexpr (GEOM == ATB_GEOM_FIXED) {
        // the last boundary gives the period's totals (points of the trash slot excluded)
#pragma unroll
        for (int m = 0; m < J; ++m) {
            const int j = jb + 32 * m + lane;
            if (j == NB) ws.tot = acc[m];
            if (j <= NB) ent_store(fb + 8u * (unsigned)j, filter_entry<GEOM, PK>(acc[m], f1, bl, sh));
        }
    } else {
        const int M = NB - os;  // the padding copy starts here, see window_sums
        if (jb == 0) {
            if (lane <= os) ws.head[lane] = acc[0];
            __syncwarp();
        }
        if (jb + 32 * J >= M) {
            const int jlook = ws.per[ip].jlook;
#pragma unroll
            for (int m = 0; m < J; ++m) {
                const int j = jb + 32 * m + lane;
                if (j > jlook) acc[m] = ws.tot;
                if (j == M - 1) ws.cm1 = acc[m];
                if (j == NB - 1) {
                    ws.hnb = ws.tot;
                    ws.hnb.sub(acc[m]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < J; ++m) {
                const int j = jb + 32 * m + lane;
                if (j >= M && j <= NB) {
                    acc[m] = ws.cm1;
                    acc[m].add(ws.head[j < NB ? j - M + 1 : os]);
                    if (j == NB) acc[m].add(ws.hnb);
                }
            }
        }
        const unsigned ab = fb + 8u * (unsigned)(jb + lane - s_done);
#pragma unroll
        for (int m = 0; m < J; ++m)
            ent_store(ab + 256u * m, filter_entry<GEOM, PK>(acc[m], f1, bl, sh));
    }
    __syncwarp();
}

// Searches period `ip` of the warp's set; its result goes to ws.res[ip].  False
// when more windows are within the filter's error of the best than the list
// holds (a flat light curve, say): the period is left to the scatter kernel.
// The bound starts at half the last period's: neighbouring periods reach similar
// ratios, so few windows pass on the way up.  When no window reaches that
// guess, the period is searched again from zero; the result never depends on it.
template <int GEOM, bool PK>
__device__ __forceinline__ bool gather_period(const SearchArgs& a, WarpState<PK>& ws, unsigned fb,
                                              int ring, int c, int ip) {
    const int lane = threadIdx.x & 31;
    const int nd = ws.st->n_dur, NB = ws.per[ip].NB, os = a.oversample;
    if (GEOM == ATB_GEOM_BINNED) {
        const double Ps = ws.per[ip].Ps;
        const int K = ws.per[ip].K;
        if (K - 1 <= kMaxCyc) fill_cycles<PK>(ws, 0, K - 1, Ps, ws.per[ip].sure0);
        if (lane == 31) {
            int col, row;
            unsigned f;
            cycle_cell(K - 1, Ps, (unsigned)ws.rows, col, row, f);
            const bool care = !(ws.per[ip].sure0 && K == 1) && near_point<PK>(ws, f, ws.bsh);
            ws.cyc[kMaxCyc] =
                make_int2(col, (int)(f | ((unsigned)row << kOffBits)) | (care ? kCareful : 0));
        }
    } else if (lane < nd) {
        const double Lf = fma(a.durations[a.dur_beg[c] + lane] * ws.per[ip].IP, (double)NB, 0.5);
        ws.len[lane] = Lf >= (double)kLenCap ? kLenCap : (Lf >= 1.0 ? (int)Lf : 1);
    }
    float guess = ws.guess;
    for (;;) {
        __syncwarp();
        if (lane == 0) {
            const GatherConsts& gk = ws.st->gk;
            ws.n_list = 0;
            ws.f = FilterState{guess, gk.e0, gk.wE, gk.wN};
            if constexpr (!PK) ws.wm = gk.wm;
            ws.tot = curve_total<PK>(*ws.st);
        }
        __syncwarp();
        const int lmax = min(ws.st->lmax, NB);
        int s_done = 0;  // starts searched; the buffer's first entry (astropy bins)
        for (int jb = 0; jb <= NB;) {
            // (one instance of the step: shorter ones for the last rows would not fit
            // the instruction cache)
            const int next = jb + 128;
            gather_step<GEOM, PK, 4>(ws, fb, ip, jb, s_done, os);
            if (GEOM == ATB_GEOM_BINNED) {
                const int s_end = next - lmax;  // window ends up to next - 1
                // as late as the buffer allows: long loops over the starts
                if (next > NB || next + 128 - s_done > ring) {
                    const unsigned base = fb - 8u * (unsigned)s_done;
                    const unsigned last = next > NB ? base + 8u * (unsigned)(NB + 1) : 0xffffffffu;
                    if (next > NB && lane == 0) ent_store(last, make_float2(NAN, 0.0f));
                    __syncwarp();
                    gather_starts<GEOM, PK>(&ws, base, last, nd, s_done, next > NB ? NB : s_end);
                    if (ws.n_list < 0) break;
                    __syncwarp();
                    if (next <= NB) {  // the pending starts' entries move to the front
                        const unsigned sh8 = 8u * (unsigned)(s_end - s_done);
                        for (int i = lane; i < ((lmax + 31) & ~31); i += 32) {
                            const float2 v = ent_load(fb + sh8 + 8u * (unsigned)i);
                            __syncwarp();
                            ent_store(fb + 8u * (unsigned)i, v);
                            __syncwarp();
                        }
                        s_done = s_end;
                    }
                }
            }
            jb = next;
        }
        if (GEOM == ATB_GEOM_FIXED) fixed_windows<GEOM, PK>(&ws, fb, NB);
        __syncwarp();
        if (ws.f.lim > guess || guess == 0.0f) break;
        guess = 0.0f;  // nothing reached the guess
    }
    const int n = ws.n_list;
    if (lane == 0) ws.guess = 0.5f * ws.f.lim;
    if (n >= 0) gather_winner<GEOM, PK>(&ws, ip, os);
    __syncwarp();
    return n >= 0;
}

// Writes the outputs of the `n` finished periods of curve c (those in `done`),
// one lane each.
template <int GEOM, bool PK>
__device__ __noinline__ void gather_flush(const SearchArgs* ap, const WarpState<PK>* ws, int c,
                                          int n, unsigned done) {
    const SearchArgs& a = *ap;
    const int lane = threadIdx.x & 31;
    if (lane < n && (done >> lane & 1u)) {
        const TableStat& st = *ws->st;
        const GatherResult<PK>& r = ws->res[lane];
        const int nd = st.n_dur, period = ws->per[lane].period;
        const double P = ws->per[lane].P;
        const long long slot = a.out_beg[c] + period;
        const double sy2 = ldexp(1.0, -st.ey), sw2 = ldexp(1.0, -st.ew);
        float o_pw = 0.0f, o_dep = 0.0f, o_de = 0.0f, o_dur = 0.0f;
        double o_t0 = 0.0;
        const bool none = r.key == 0x7fffffff;
        if (!none) {
            const int s = r.key / nd, k = r.key % nd;
            double dw, dy, wtot, ytot;
            if constexpr (PK) {
                const double qw0s = ldexp((double)st.qw0, -st.ew);
                dw = (double)packed_count(r.d.x, st.g_bl) * qw0s;
                dy = (double)packed_flux(r.d.x, st.g_bl, st.g_guard) * sy2;
                wtot = (double)packed_count(r.tot.x, st.g_bl) * qw0s;
                ytot = (double)packed_flux(r.tot.x, st.g_bl, st.g_guard) * sy2;
            } else {
                dw = (double)(long long)r.d.x * sw2;
                dy = (double)(long long)r.d.y * sy2;
                wtot = (double)(long long)r.tot.x * sw2;
                ytot = (double)(long long)r.tot.y * sy2;
            }
            if (GEOM == ATB_GEOM_BINNED) {
                const double durv = (double)ws->len[k] * st.bin_dur;
                o_dur = (float)durv;
                o_t0 = fmod((double)s * st.bin_dur + 0.5 * durv + st.t_start, P);
            } else {
                o_dur = (float)a.durations[a.dur_beg[c] + k];
                o_t0 = fma((double)s / (double)a.n_bins_fixed, 1.0 / ws->per[lane].IP, st.t_start);
            }
            double pw, dep, de;
            window_stats(dw, dy, wtot, ytot, st.s_w - st.ew, st.s_y - st.ey, a.objective, &pw,
                         &dep, &de);
            o_pw = (float)pw;
            o_dep = (float)dep;
            o_de = (float)de;
            if (a.best_key)
                atomicMax(a.best_key + c,
                          ((unsigned long long)__float_as_uint(o_pw) << 32) |
                              (unsigned long long)(0xffffffffu - (unsigned)period));
        }
        if (a.power) a.power[slot] = o_pw;
        if (a.depth) a.depth[slot] = o_dep;
        if (a.depth_err) a.depth_err[slot] = o_de;
        if (a.t0) a.t0[slot] = o_t0;
        if (a.duration) a.duration[slot] = o_dur;
        if (a.window) a.window[slot] = none ? -1 : r.key;
    }
    __syncwarp();
}

// The periods t0 + warp, t0 + warp + kGatherWarps, ... below p1 of curve c, those of them
// that are gathered.
// The CTA's warps search neighbouring periods in step (a barrier after each), so
// that they read the same table entries from L1 and the same instructions.
template <int GEOM, bool PK>
__device__ __forceinline__ void gather_periods(const SearchArgs& a, const GatherArgs& ga,
                                               WarpState<PK>& ws, unsigned fb, int c, long long t0,
                                               long long p1) {
    const int lane = threadIdx.x & 31;
    const TableStat* st = a.tstats + c;
    double P = 0.0;
    int NB = 0;
    bool on = false;
    const long long p = t0 + (threadIdx.x >> 5) + (long long)lane * kGatherWarps;
    if (lane < kMaxPop && p < p1) {
        P = a.periods[a.per_beg[c] + p];
        NB = GEOM == ATB_GEOM_BINNED ? binned_nbins(P, st->inv_bin_dur, a.oversample, a.max_bins)
                                     : a.n_bins_fixed;
        on = a.scatter[a.flag_off[c] + p] == 0;
    }
    const unsigned who = __ballot_sync(0xffffffffu, on);
    const int n = __popc(who);
    if (on) {
        GatherPeriod g;
        g.P = P;
        g.IP = 1.0 / P;
        g.Ps = P * st->g_scale;
        g.NB = NB;
        g.K = (int)floor(st->dt_absmax * g.IP) + 1;
        g.jlook = NB;
        // astropy bins: the boundaries inside the cycle, j * b <= P within a quarter unit
        if (GEOM == ATB_GEOM_BINNED)
            g.jlook = min((int)floor(P * st->inv_bin_dur + 0.25 / (kOffUnits * st->g_rows)), NB - 1);
        g.period = (int)p;
        // unless a boundary lies at the very end of the cycle, where the point on it
        // may fall into the next one
        const double x = P * st->inv_bin_dur;
        g.sure0 = GEOM == ATB_GEOM_BINNED && fabs(x - rint(x)) * kOffUnits * st->g_rows > 8.0;
        ws.per[__popc(who & ((1u << lane) - 1u))] = g;
    }
    if (GEOM == ATB_GEOM_BINNED && lane < st->n_dur) ws.len[lane] = a.dbins[c * kMaxDur + lane];
    if (lane == 0) {
        const long long co = ga.cell_off[c], so = a.stage_off[c];
        ws.st = st;
        ws.idx = ga.idx + co;
        ws.tab = reinterpret_cast<const Entry<PK>*>(ga.tab + co * (16 * ga.vs));
        ws.bits = ga.bits + ga.bit_off[c];
        ws.sdt = a.sdt + so;
        ws.sqw = a.sqw + so;
        ws.sqy = a.sqy + so;
        ws.rows = st->g_rows;
        ws.pitch = st->g_pitch;
        ws.colmax = st->g_colmax;
        ws.bsh = offset_shift(st->g_bl - 1);
        ws.gmul = 1 << st->g_guard;
        ws.cinc = 1u << (32 - st->g_bl);
        ws.guess = 0.0f;
        ws.n_full = st->ilv ? ((long long)st->g_n + kR - 1) / kR * kR / kChunk * kChunk : 0;
    }
    __syncwarp();
    unsigned done = 0;
    for (int i = 0; __syncthreads_or(i < n); ++i)
        if (i < n && gather_period<GEOM, PK>(a, ws, fb, ga.ring, c, i)) done |= 1u << i;
    gather_flush<GEOM, PK>(&a, &ws, c, n, done);
    if (lane < n) {
        if (!(done >> lane & 1u)) {  // left to the scatter kernel
            a.scatter[a.flag_off[c] + ws.per[lane].period] = 1;
            atomicOr(ga.n_scatter, 1);
            atomicAdd(ga.n_back, 1ULL);
        }
    }
    __syncwarp();
}

// Persistent CTAs; each takes up to kMaxPop periods per warp of a work-queue tile at
// a time -- fewer when there are not about 16 turns for every CTA, since a long
// period alone keeps a warp busy for a millisecond.
template <int GEOM, bool PK>
__global__ void __launch_bounds__(kGatherBlock, kGatherMinBlocks)
    gather_kernel(const __grid_constant__ SearchArgs a, const __grid_constant__ GatherArgs ga) {
    extern __shared__ __align__(16) char g_smem[];
    __shared__ long long s_beg, s_end;  // the part's periods (s_beg < 0: no more parts)
    __shared__ int s_curve;
    chain_start();
    if (ga.n_gather[PK ? 0 : 1] == 0) return;
    const int warp = threadIdx.x >> 5;
    const unsigned fsz = gather_ring_bytes(ga.ring);
    const unsigned fb = (unsigned)__cvta_generic_to_shared(g_smem) + warp * fsz;
    WarpState<PK>& ws = *reinterpret_cast<WarpState<PK>*>(
        g_smem + kGatherWarps * fsz + warp * gather_state_bytes(PK ? 1 : 2));
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            int chunk = kGatherWarps * kMaxPop;
            while (chunk > kGatherWarps && ga.n_gather[PK ? 0 : 1] / chunk < 16 * gridDim.x)
                chunk /= 2;
            const unsigned subs = (unsigned)((a.tile_p + chunk - 1) / chunk);
            const unsigned long long units = (unsigned long long)a.n_tiles * subs;
            s_beg = -1;
            for (;;) {  // the next part of a tile of a curve of this kernel
                const unsigned long long u = atomicAdd(ga.counter + (PK ? 0 : 1), 1ULL);
                if (u >= units) break;
                const long long tile = (long long)(u / subs);
                int lo = 0, hi = a.n_curves;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (a.tile_off[mid] <= tile) lo = mid; else hi = mid;
                }
                const int c = a.order[lo];
                const TableStat* st = a.tstats + c;
                if (!st->g_on || (st->cnt_win != 0) != PK) continue;
                const long long t0 = tile_start(a, tile, lo, c);
                const long long beg = t0 + (long long)(u % subs) * chunk;
                const long long end = min(min(t0 + a.tile_p, beg + chunk), a.per_cnt[c]);
                if (beg >= end) continue;
                s_beg = beg;
                s_end = end;
                s_curve = c;
                break;
            }
        }
        __syncthreads();
        if (s_beg < 0) break;
        gather_periods<GEOM, PK>(a, ga, ws, fb, s_curve, s_beg, s_end);
    }
}
