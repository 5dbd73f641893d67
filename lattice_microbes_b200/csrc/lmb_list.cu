// lmb_list.cu -- one launch per MPD timestep, worked by particle: the x, y
// and z sweeps and the reaction of a tile of full x-rows, with the tile's
// particles in a shared-memory list.
//
// A block owns Ty x Tz full rows and loads them with one halo row on each
// side in y and z (periodic), as the dense fused kernel (lmb_fused.cu) does,
// but it keeps no copy of the sites: every particle becomes one list entry
// (species, region site, slot), and a site exists only as the slot masks of
// its stayers, minus movers and plus movers in the sweep at hand.  A
// particle's place after a sweep follows from those masks alone (a stayer
// comes after its site's stayers of lower slots; an arrival from the minus
// side after every stayer and that neighbour's plus movers of lower slots;
// one from the plus side after those, the minus neighbour's plus movers and
// its own site's minus movers of lower slots: the order
// byte_diffusion_1d_dev.cu:199-269 builds site by site), so the thread that
// places a particle in one sweep draws its choice for the next one in the
// same pass:
//
//   load     the rows' particles into the list
//   pass 0   draw x
//   pass 1   place x, draw y
//   pass 2   place y (particles that leave the owned y rows are dropped), draw z
//   pass 3   place z (only what lands on owned sites), write
//   react    the few sites whose draw allows a reaction
//
// The work of a pass is the number of particles, spread evenly over the
// block, whatever the number of sites and however the particles cluster; the
// dense kernel's list passes over the occupancy bits, its three draws per
// particle and sweep (own, minus and plus side) and its site-by-site sweeps,
// whose warps wait for their fullest site, are gone.
//
// Halo rows are recomputed by several blocks; every decision is a pure
// function of (seed, step, site, slot, site types), so the copies agree, and
// only the owner of a site queues its overflows.  The last block of a launch
// to finish resolves the overflow queue (lmb_overflow.cuh).
//
// A tile whose particles do not fit the list is worked as smaller sub-tiles
// one after another (down to one row, whose region always fits), before
// anything is written or queued, so any density gives the same result.
//
// Measured per timestep, autotuned, against the per-phase or dense fused
// kernels the autotuner took before: crowded cell (128 x 128 x 256,
// IntLattice of 16 slots, 1M particles) 250 -> 112 us, 96^3 with 1.25
// particles per site 100 -> 54 us, IntLattice of 8 slots with obstacles
// 124 -> 30 us (default plan), rod cell 16.7 -> 10.3 us, 32^3 with 2,000
// particles 11.6 -> 6.3 us.  It is bound by instructions issued (hashes and
// placement per particle, list building per site of the region) on the large
// lattices and by the chain of passes, load and completion count on the small.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "lmb.h"
#include "lmb_device.cuh"
#include "lmb_fused.h"
#include "lmb_internal.h"
#include "lmb_overflow.cuh"
#include "lmb_site.cuh"
#include "lmb_stage.cuh"

namespace lmb {

constexpr uint32_t LIST_HIST = LIST_MAX_COUNTED;  // species-count histogram entries
constexpr uint32_t LIST_MAX_REGION = 1u << 14;    // region sites a list entry can name
constexpr uint32_t LIST_RLIM = 32;                // site types whose reaction bound a tile keeps
constexpr uint32_t LIST_CAND = 512;               // reaction candidates of a sub-tile; more: every site is looked at

// Row flags above a row's number among the owned rows: the halo rows of the
// region's y and z ends.
constexpr uint32_t ROW_YL = 1u << 12, ROW_YH = 1u << 13, ROW_ZL = 1u << 14, ROW_ZH = 1u << 15;
constexpr uint32_t ROW_HALO = ROW_YL | ROW_YH | ROW_ZL | ROW_ZH, ROW_INDEX = ROW_YL - 1u;

// n / d by the multiplier list_magic(d) gives (exact for n < 2^16).
__device__ __forceinline__ uint32_t fast_div(uint32_t n, uint32_t magic) { return magic ? __umulhi(n, magic) : n; }

// A list entry: species, the choice drawn for the sweep at hand (0 stay,
// 1 minus, 2 plus), region site and slot.  0 is a dropped particle.
constexpr uint32_t LIST_P = 20, LIST_C = 18, LIST_L = 4;
__device__ __forceinline__ uint32_t entry_site(uint32_t e) { return (e >> LIST_L) & 0x3FFFu; }

// A sweep's choices of the region's sites: the slots of a site that stay,
// move to the minus and to the plus neighbour.  Up to 8 slots: one word per
// site (8 bits each).  16 slots: a word of minus | plus << 16 per site, then
// the stayers, two sites to a word.
template <int S>
struct Choices {
    static constexpr uint32_t STAY = 0xFFu, MINUS = S <= 8 ? 0xFF00u : 0xFFFFu, PLUS = S <= 8 ? 0xFF0000u : 0xFFFF0000u;
    uint32_t *m;
    uint32_t R;
    static __host__ __device__ uint32_t words(uint32_t R)
    {
        const uint32_t w = S <= 8 ? R : R + (R + 1u) / 2u;
        return (w + 3u) & ~3u;
    }
    __device__ __forceinline__ const uint16_t *stays() const { return reinterpret_cast<const uint16_t *>(m + R); }
    __device__ __forceinline__ uint32_t stay(uint32_t l) const { return S <= 8 ? m[l] & STAY : (uint32_t)stays()[l]; }
    __device__ __forceinline__ uint32_t plus(uint32_t l) const { return m[l] & PLUS; }
    __device__ __forceinline__ void put(uint32_t l, uint32_t k, uint32_t c) const
    {
        if (S <= 8) {
            atomicOr(&m[l], 1u << (8u * c + k));
        } else {
            uint32_t *at = c == 0 ? m + R + (l >> 1) : m + l;
            const uint32_t sh = c == 0 ? 16u * (l & 1u) : 16u * (c - 1u);
            atomicOr(at, 1u << (sh + k));
        }
    }
    // Place of the particle in slot k of site l with choice c, whose new site
    // is d: after d's stayers when it moves, after the plus movers of d's
    // minus neighbour dm when it comes from the plus side, and after the
    // lower slots of its own site with the same choice.
    __device__ __forceinline__ uint32_t place(uint32_t l, uint32_t k, uint32_t c, uint32_t d, uint32_t dm) const
    {
        uint32_t own;
        if (S <= 8) own = (m[l] >> (8u * c)) & ((1u << k) - 1u);
        else own = (c == 0 ? (uint32_t)stays()[l] : m[l] >> (16u * (c - 1u))) & ((1u << k) - 1u);
        uint32_t pos = __popc(own);
        if (c != 0) pos += __popc(stay(d));
        if (c == 1) pos += __popc(plus(dm));
        return pos;
    }
    // Particles of site d after the sweep: its stayers and the arrivals from
    // its neighbours dm and dp (bit fields that do not overlap).
    __device__ __forceinline__ uint32_t count(uint32_t d, uint32_t dm, uint32_t dp) const
    {
        return clamp(m[d], S <= 8 ? 0u : (uint32_t)stays()[d], m[dm], m[dp]);
    }
    static __device__ __forceinline__ uint32_t clamp(uint32_t own, uint32_t stay, uint32_t below, uint32_t above)
    {
        uint32_t n = __popc((below & PLUS) | (above & MINUS) | (S <= 8 ? own & STAY : 0u));
        if (S > 8) n += __popc(stay);
        return n < (uint32_t)S ? n : (uint32_t)S;
    }
};

// Zeroes n words (a multiple of 4) at 16-byte aligned p, by the whole block.
template <int NT>
__device__ __forceinline__ void clear_words(uint32_t *p, uint32_t n)
{
    uint4 *q = reinterpret_cast<uint4 *>(p);
    for (uint32_t i = threadIdx.x; i < n / 4u; i += NT) q[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Particles in a word: its nonzero bytes (ByteLattices), or the word itself.
template <int BPS>
__device__ __forceinline__ uint32_t particles_in(uint32_t w)
{
    if (BPS != 1) return w != 0u ? 1u : 0u;
    return __popc((w | ((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu)) & 0x80808080u);
}

// Room in the list for n entries of each lane, by a whole warp: one shared
// atomic.  Null for a warp whose particles pass C (they are only counted).
__device__ __forceinline__ uint32_t *list_reserve(uint32_t n, uint32_t *list, uint32_t C, uint32_t *count)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(count, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    return base + total > C ? nullptr : list + base + incl - n;  // the same for the warp
}

// Writes the entries of word plane `plane` of V consecutive sites (words v,
// first region site l0) at q, which moves on; the whole warp takes part.
template <int BPS, int V>
__device__ __forceinline__ void list_emit(const uint32_t (&v)[V], uint32_t l0, uint32_t plane, uint32_t *&q)
{
    const uint32_t at = l0 << LIST_L;
#pragma unroll
    for (int j = 0; j < V; j++) {
        if (BPS == 1 && !__any_sync(0xffffffffu, v[j] != 0u)) continue;
#pragma unroll
        for (int b = 0; b < (BPS == 1 ? 4 : 1); b++) {
            const uint32_t p = BPS == 1 ? (v[j] >> (8 * b)) & 0xFFu : v[j];
            if (p) *q++ = (p << LIST_P) + at + (BPS == 1 ? 4u * plane + b : plane) + (j << LIST_L);
        }
    }
}

// Appends the particles of one word plane of V sites per lane to the list.
template <int BPS, int V>
__device__ __forceinline__ void list_plane(const uint32_t (&v)[V], uint32_t l0, uint32_t plane, uint32_t *list,
                                           uint32_t C, uint32_t *count)
{
    uint32_t any = 0, n = 0;
#pragma unroll
    for (int j = 0; j < V; j++) {
        any |= v[j];
        n += particles_in<BPS>(v[j]);
    }
    if (!__any_sync(0xffffffffu, any != 0u)) return;
    uint32_t *q = list_reserve(n, list, C, count);
    if (q) list_emit<BPS, V>(v, l0, plane, q);
}

template <int V>
__device__ __forceinline__ void load_sites(const uint32_t *p, uint32_t (&v)[V])
{
    if constexpr (V == 4) {
        const uint4 t = *reinterpret_cast<const uint4 *>(p);
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    } else {
        v[0] = *p;
    }
}

// Lists every particle of the region's rows.  An item is V consecutive sites
// of a row (`q` items per row, mq its multiplier), one per thread and
// iteration; planes 0 and 1 are read with the plane bound rather than after
// it (planes at or above a bound hold zeros) and share one prefix sum, the
// planes above are read only below the bound.  Planes and sites no lane of the
// warp holds anything in are skipped by votes: at a few particles per hundred
// sites that is most of them.
template <int BPS, int S, int V, int NT>
__device__ __forceinline__ void list_rows(const uint32_t *__restrict__ src, const uint32_t *__restrict__ pb,
                                          uint32_t N, uint32_t X, uint32_t rows, uint32_t q, uint32_t mq,
                                          const uint32_t *rowbase, uint32_t *list, uint32_t C, uint32_t *count)
{
    constexpr uint32_t W = SiteWords<BPS, S>::W;
    constexpr uint32_t EARLY = W < 2 ? W : 2;
    const uint32_t nit = rows * q;
    // The next item's loads are in flight while this one is listed: a region
    // is several iterations long, each a round trip to L2 otherwise.
    uint32_t v[EARLY][V], w[EARLY][V], l0 = 0, g0 = 0, npl = 0, l1 = 0, g1 = 0, npl1 = 0;
    auto fetch = [&](uint32_t i) {
        l1 = g1 = npl1 = 0;
#pragma unroll
        for (uint32_t k = 0; k < EARLY; k++)
#pragma unroll
            for (int j = 0; j < V; j++) w[k][j] = 0u;
        if (i < nit) {
            const uint32_t r = fast_div(i, mq), c = i - r * q;
            l1 = r * X + c * V;
            g1 = rowbase[r] + c * V;
#pragma unroll
            for (uint32_t k = 0; k < EARLY; k++) load_sites<V>(src + (size_t)k * N + g1, w[k]);
            if (W > EARLY) npl1 = pb ? min(pb[g1 >> PB_SHIFT], W) : W;
        }
    };
    fetch(threadIdx.x);
    for (uint32_t i0 = 0; i0 < nit; i0 += NT) {
#pragma unroll
        for (uint32_t k = 0; k < EARLY; k++)
#pragma unroll
            for (int j = 0; j < V; j++) v[k][j] = w[k][j];
        l0 = l1;
        g0 = g1;
        npl = npl1;
        if (i0 + NT < nit) fetch(i0 + NT + threadIdx.x);
        uint32_t n = 0;
        bool held[EARLY];
#pragma unroll
        for (uint32_t k = 0; k < EARLY; k++) {
            uint32_t any = 0;
#pragma unroll
            for (int j = 0; j < V; j++) any |= v[k][j];
            held[k] = __any_sync(0xffffffffu, any != 0u);
            if (held[k]) {
#pragma unroll
                for (int j = 0; j < V; j++) n += particles_in<BPS>(v[k][j]);
            }
        }
        if (held[0] || held[EARLY - 1]) {
            uint32_t *at = list_reserve(n, list, C, count);
            if (at) {
#pragma unroll
                for (uint32_t k = 0; k < EARLY; k++)
                    if (held[k]) list_emit<BPS, V>(v[k], l0, k, at);
            }
        }
        if constexpr (W > EARLY) {
            const uint32_t most = __reduce_max_sync(0xffffffffu, npl);
            for (uint32_t k = EARLY; k < most; k++) {
                uint32_t u[V];
#pragma unroll
                for (int j = 0; j < V; j++) u[j] = 0u;
                if (k < npl) load_sites<V>(src + (size_t)k * N + g0, u);
                list_plane<BPS, V>(u, l0, k, list, C, count);
            }
        }
    }
}

// Reaction of one site, kept out of line: a few sites per tile reach it.
template <int BPS, int S>
__device__ __noinline__ bool list_react(SiteWords<BPS, S> &s, uint32_t t, uint32_t gi, unsigned long long th,
                                        const DevTables &m, RunState *rs, OverflowEntry *list, uint32_t cap)
{
    if (m.nr <= 32u) return react_site<BPS, S, -1>(s, t, gi, th, m, rs, list, cap);
    return react_site<BPS, S, 0>(s, t, gi, th, m, rs, list, cap);
}

// Static shared memory of a tile.
struct ListShared {
    uint32_t last, count, ncand;
    uint32_t rowbase[FUSED_MAX_ROWS];
    uint16_t rowinfo[FUSED_MAX_ROWS], ownrow[FUSED_MAX_ROWS];
    uint16_t cand[LIST_CAND];
    float rlim[LIST_RLIM];  // per site type: no site reacts on a draw above it, however full
    DevTables mt;           // the model tables, staged or not
};

// A tile's timestep.
template <int BPS, int S, int NT>
struct ListTile {
    static constexpr uint32_t W = SiteWords<BPS, S>::W;
    static constexpr int CB = CountBits<S>::value;
    // Up to 8 slots keep two mask buffers, so that a pass can place by one
    // sweep's choices and draw the next one's.  16 slots keep one, cleared
    // between sweeps, and set the choices drawn in a pass of their own: at 6
    // bytes a site the smaller region's halo costs more than the pass.
    static constexpr bool TWO = S <= 8;
    using Ch = Choices<S>;

    const Geometry &g;
    const DevTables &m;
    RunState *rs;
    OverflowEntry *queue;
    const uint32_t cap;
    const TileShape &ts;
    const int with_reaction;
    ListShared &sh;
    const DevTables &mt;
    const float *Ttab;
    const uint32_t X, mX, tid, ns, nst;
    const bool scan_all;       // zeroth-order reactions: every site may react
    uint32_t ty0, tz0;         // the tile
    uint32_t cty, ctz, y0, z0; // the sub-tile at hand
    uint32_t Ry, rows, R, RO, C, dz;
    uint32_t *hist, *work, work_words;
    Ch P, Q;
    uint32_t *out, *list;
    uint8_t *T;
    unsigned long long th[4];  // the timestep's sub-step hashes
    bool counting;             // species counts are taken after this timestep

    // Dynamic shared memory: the staged tables, then per sub-tile the choice
    // masks, a ByteLattice's new words (in the second mask buffer where
    // that is free again), the site types and the list in what is left (its
    // end the species histogram in the timesteps that count).
    __device__ __forceinline__ ListTile(uint32_t *smem, uint32_t smem_bytes, const Geometry &g_, const DevTables &m_,
                                        RunState *rs_, OverflowEntry *queue_, uint32_t cap_, const TileShape &ts_,
                                        int with_reaction_, ListShared &sh_, uint32_t tile)
        : g(g_), m(m_), rs(rs_), queue(queue_), cap(cap_), ts(ts_), with_reaction(with_reaction_), sh(sh_), mt(sh_.mt),
          Ttab(m_.stage_bytes ? reinterpret_cast<const float *>(smem) : m_.T), X(g_.X), mX(ts_.magic_x),
          tid(threadIdx.x), ns(m_.ns), nst(m_.nst), scan_all(with_reaction_ && m_.zeroth)
    {
        uint8_t *tables = reinterpret_cast<uint8_t *>(smem);
        work = reinterpret_cast<uint32_t *>(tables + m.stage_bytes);
        work_words = (smem_bytes - m.stage_bytes) / 4u;
        ty0 = (tile % ts.tiles_y) * ts.Ty;
        tz0 = (tile / ts.tiles_y) * ts.Tz;
        cty = ts.Ty;
        ctz = ts.Tz;
        y0 = z0 = 0;
        counting = false;
        const DevTables staged = m.stage_bytes ? stage_tables(m, tables, tid, NT) : m;
        if (tid == 0) sh.mt = staged;
        if (with_reaction && tid < LIST_RLIM && tid < nst) sh.rlim[tid] = reaction_bound((uint32_t)S, react_bound(tid, m));
    }

    // Row tables, mask clearing and site types of the sub-tile: nothing here
    // depends on the previous timestep.
    __device__ __forceinline__ void begin()
    {
        Ry = cty + 2u;
        rows = Ry * (ctz + 2u);
        R = rows * X;
        RO = cty * ctz * X;
        dz = Ry * X;
        const uint32_t mw = Ch::words(R), ow = BPS == 1 ? (W * RO + 3u) & ~3u : 0u;
        P.m = work;
        P.R = Q.R = R;
        Q.m = TWO ? work + mw : work;
        out = work + mw;
        T = reinterpret_cast<uint8_t *>(out + (TWO ? max(mw, ow) : ow));
        list = reinterpret_cast<uint32_t *>(T + ((R + 15u) & ~15u));
        C = work_words - (uint32_t)(list - work);
        for (uint32_t r = tid; r < rows; r += NT) {
            const uint32_t lz = r / Ry, ly = r - lz * Ry;
            // Row ly - 1 of the sub-tile, one period at most outside.
            uint32_t y = ty0 + y0 + ly, z = tz0 + z0 + lz;
            y = y == 0 ? g.Y - 1u : (y > g.Y ? 0u : y - 1u);
            z = z == 0 ? g.Z - 1u : (z > g.Z ? 0u : z - 1u);
            sh.rowbase[r] = y * X + z * g.XY;
            uint32_t f = (ly == 0 ? ROW_YL : 0u) | (ly == Ry - 1u ? ROW_YH : 0u) | (lz == 0 ? ROW_ZL : 0u) |
                         (lz == ctz + 1u ? ROW_ZH : 0u);
            if (f == 0) {
                f = (lz - 1u) * cty + ly - 1u;
                sh.ownrow[f] = (uint16_t)r;
            }
            sh.rowinfo[r] = (uint16_t)f;
        }
        if (tid == 0) sh.count = sh.ncand = 0;
        clear_words<NT>(P.m, mw);
        if (TWO) clear_words<NT>(Q.m, mw);
        __syncthreads();
    }

    __device__ __forceinline__ void load_types(const uint8_t *__restrict__ sites)
    {
        if (X % 16u == 0) {
            for (uint32_t i = tid; i < R / 16u; i += NT) {
                const uint32_t r = fast_div(4u * i, ts.magic_q);
                reinterpret_cast<uint4 *>(T)[i] =
                    __ldg(reinterpret_cast<const uint4 *>(sites + sh.rowbase[r] + (16u * i - r * X)));
            }
        } else {
            for (uint32_t l = tid; l < R; l += NT) {
                const uint32_t r = fast_div(l, mX);
                T[l] = __ldg(sites + sh.rowbase[r] + (l - r * X));
            }
        }
    }

    // In a timestep that counts species the list's end is the histogram.
    __device__ __forceinline__ void take_histogram()
    {
        if (counting) {
            C -= LIST_HIST;
            hist = list + C;
        }
    }

    // The choice of particle p in slot k of lattice site gi: its region site
    // lt with neighbours lm and lp.  Every transition probability is at most
    // 0.5, so a draw of 0.5 or more can only move plus and a lower one only
    // minus.
    __device__ __forceinline__ uint32_t hop(uint32_t p, uint32_t gi, uint32_t k, unsigned long long h, uint32_t lt,
                                            uint32_t lm, uint32_t lp) const
    {
        const float rv = hash_float(((unsigned long long)gi << CB) | k, h);
        const bool hi = rv >= 0.5f;
        const uint32_t t = nst > 1u ? T[lt] : 0u, tn = nst > 1u ? T[hi ? lp : lm] : 0u;
        float q = 0.0f;
        if (p - 1u < ns && t < nst && tn < nst) q = Ttab[(t * nst + tn) * ns + (p - 1u)];
        if (hi) return rv < __fadd_rn(q, 0.5f) ? 2u : 0u;
        return rv < q ? 1u : 0u;
    }

    // Sets the masks from the choices the entries hold (one mask buffer).
    __device__ __forceinline__ void put_choices(uint32_t n) const
    {
        for (uint32_t j = tid; j < n; j += NT) {
            const uint32_t e = list[j];
            if (e) P.put(entry_site(e), e & 15u, (e >> LIST_C) & 3u);
        }
    }

    __device__ __forceinline__ void overflow(uint32_t phase, uint32_t gi, uint32_t seq, uint32_t p) const
    {
        push_overflow(rs, queue, cap, phase, gi, seq, p);
    }

    // Lists the particles of the region's rows.
    __device__ __forceinline__ void load(const uint32_t *__restrict__ src, const uint32_t *__restrict__ pb)
    {
        if (X % 4u == 0)
            list_rows<BPS, S, 4, NT>(src, pb, g.N, X, rows, X / 4u, ts.magic_q, sh.rowbase, list, C, &sh.count);
        else
            list_rows<BPS, S, 1, NT>(src, pb, g.N, X, rows, X, mX, sh.rowbase, list, C, &sh.count);
    }

    // The three sweeps of the n listed particles.  On return a ByteLattice's
    // owned rows are in `out`, an IntLattice's particles in dst; P holds the
    // z sweep's choices and sh.cand the sites that may react.
    __device__ __forceinline__ void sweeps(uint32_t n, uint32_t *__restrict__ dst)
    {
        // Pass 0: draw x.
        for (uint32_t j = tid; j < n; j += NT) {
            const uint32_t e = list[j], l = entry_site(e), k = e & 15u;
            const uint32_t r = fast_div(l, mX), x = l - r * X;
            const uint32_t c = hop(e >> LIST_P, sh.rowbase[r] + x, k, th[0], l, x ? l - 1u : l + X - 1u,
                                   x + 1u < X ? l + 1u : l + 1u - X);
            P.put(l, k, c);
            list[j] = e | (c << LIST_C);
        }
        __syncthreads();

        // Pass 1: place x, draw y.
        for (uint32_t j = tid; j < n; j += NT) {
            const uint32_t e = list[j], k = e & 15u, c = (e >> LIST_C) & 3u, p = e >> LIST_P, l = entry_site(e);
            const uint32_t r = fast_div(l, mX), row = r * X, x = l - row;
            const uint32_t xm = x ? x - 1u : X - 1u, xp = x + 1u < X ? x + 1u : 0u;
            const uint32_t xd = c == 0 ? x : (c == 1 ? xm : xp), d = row + xd;
            const uint32_t pos = P.place(l, k, c, d, row + (xm ? xm - 1u : X - 1u));
            const uint32_t info = sh.rowinfo[r], gi = sh.rowbase[r] + xd;
            uint32_t ne = 0;
            if (pos >= (uint32_t)S) {
                if (!(info & ROW_HALO)) overflow(1u, gi, pos - (uint32_t)S, p);
            } else {
                // A halo row matters for what it sends into the owned rows.
                const bool lo = info & ROW_YL, up = info & ROW_YH;
                const uint32_t cy = hop(p, gi, pos, th[1], d, lo ? d : d - X, up ? d : d + X);
                if (!((lo && cy != 2u) || (up && cy != 1u))) {
                    if (TWO) Q.put(d, pos, cy);
                    ne = (p << LIST_P) | (cy << LIST_C) | (d << LIST_L) | pos;
                }
            }
            list[j] = ne;
        }
        __syncthreads();
        clear_words<NT>(P.m, Ch::words(R));
        __syncthreads();
        if (!TWO) {
            put_choices(n);
            __syncthreads();
        }

        // Pass 2: place y, draw z.
        for (uint32_t j = tid; j < n; j += NT) {
            const uint32_t e = list[j], k = e & 15u, c = (e >> LIST_C) & 3u, p = e >> LIST_P, l = entry_site(e);
            if (e == 0) continue;
            const uint32_t r0 = fast_div(l, mX), x = l - r0 * X;
            const uint32_t r = r0 + (c == 2u ? 1u : 0u) - (c == 1u ? 1u : 0u);
            const uint32_t d = l + (c == 2u ? X : 0u) - (c == 1u ? X : 0u);
            const uint32_t info = sh.rowinfo[r];
            uint32_t ne = 0;
            if (!(info & (ROW_YL | ROW_YH))) {
                const uint32_t pos = Q.place(l, k, c, d, d - X), gi = sh.rowbase[r] + x;
                if (pos >= (uint32_t)S) {
                    if (!(info & ROW_HALO)) overflow(2u, gi, pos - (uint32_t)S, p);
                } else {
                    const bool lo = info & ROW_ZL, up = info & ROW_ZH;
                    const uint32_t cz = hop(p, gi, pos, th[2], d, lo ? d : d - dz, up ? d : d + dz);
                    if (!((lo && cz != 2u) || (up && cz != 1u))) {
                        if (TWO) P.put(d, pos, cz);
                        ne = (p << LIST_P) | (cz << LIST_C) | (d << LIST_L) | pos;
                    }
                }
            }
            list[j] = ne;
        }
        __syncthreads();
        if (!TWO) {
            clear_words<NT>(P.m, Ch::words(R));
            __syncthreads();
            put_choices(n);
        }
        if (BPS == 1) clear_words<NT>(out, (W * RO + 3u) & ~3u);
        if (!TWO || BPS == 1) __syncthreads();

        // Pass 3: place z and write: an IntLattice particle into its word of
        // the lattice, a ByteLattice particle into its byte of the words
        // assembled in shared memory.  The first particle of a site takes the
        // exits of react_site that need no table sums.
        for (uint32_t j = tid; j < n; j += NT) {
            const uint32_t e = list[j], k = e & 15u, c = (e >> LIST_C) & 3u, p = e >> LIST_P, l = entry_site(e);
            if (e == 0) continue;
            const uint32_t r0 = fast_div(l, mX), x = l - r0 * X;
            const uint32_t r = r0 + (c == 2u ? Ry : 0u) - (c == 1u ? Ry : 0u);
            const uint32_t d = l + (c == 2u ? dz : 0u) - (c == 1u ? dz : 0u);
            const uint32_t info = sh.rowinfo[r];
            uint32_t ne = 0;
            if (!(info & ROW_HALO)) {
                const uint32_t pos = P.place(l, k, c, d, d - dz), gi = sh.rowbase[r] + x;
                if (pos >= (uint32_t)S) {
                    overflow(3u, gi, pos - (uint32_t)S, p);
                } else {
                    ne = e;
                    if (BPS == 1)
                        reinterpret_cast<uint8_t *>(&out[(pos >> 2) * RO + info * X + x])[pos & 3u] = (uint8_t)p;
                    else
                        dst[(size_t)pos * g.N + gi] = p;
                    if (pos == 0 && with_reaction && !scan_all) {
                        // The bound grows with the count: most draws lie
                        // above that of a full site.
                        const float rv = hash_float((unsigned long long)gi << 1, th[3]);
                        const uint32_t t = T[d];
                        if (!(t < LIST_RLIM && rv > sh.rlim[t]) &&
                            reaction_may_fire(P.count(d, d - dz, d + dz), react_bound(t, mt), rv)) {
                            const uint32_t at = atomicAdd(&sh.ncand, 1u);
                            if (at < LIST_CAND) sh.cand[at] = (uint16_t)d;
                        }
                    }
                }
            }
            if (counting) list[j] = ne;
        }
        __syncthreads();
    }

    // Dense write of the owned rows (empty sites as zeros), up to the larger
    // of the segment's new plane bound and the destination's old one; the new
    // bound is stored.
    __device__ __forceinline__ void write_rows(uint32_t *__restrict__ dst, uint32_t *__restrict__ pb_dst) const
    {
        if constexpr (BPS == 1) {
            if (X % 4u == 0) {
                const uint32_t q = X / 4u, nit = cty * ctz * q;
                for (uint32_t i0 = 0; i0 < nit; i0 += NT) {
                    const uint32_t i = i0 + tid;
                    const bool in = i < nit;
                    uint4 v[W];
                    uint32_t gi = 0, nw = 0;
                    if (in) {
                        const uint32_t oq = fast_div(i, ts.magic_q);
                        gi = sh.rowbase[sh.ownrow[oq]] + 4u * (i - oq * q);
#pragma unroll
                        for (uint32_t k = 0; k < W; k++) {
                            v[k] = reinterpret_cast<const uint4 *>(out + k * RO)[i];
                            if (v[k].x | v[k].y | v[k].z | v[k].w) nw = k + 1u;
                        }
                    }
                    uint32_t lim = W;
                    if (W > 2 && pb_dst) {
                        // Eight lanes hold a segment of 32 sites; all have
                        // read the old bound when the shuffles are done.
                        const uint32_t old = in ? min(pb_dst[gi >> PB_SHIFT], W) : 0u;
#pragma unroll
                        for (int o = 1; o < 8; o <<= 1) nw = max(nw, __shfl_xor_sync(0xffffffffu, nw, o));
                        lim = max(nw, old);
                        if (in && (tid & 7u) == 0) pb_dst[gi >> PB_SHIFT] = nw;
                    }
                    if (in) {
#pragma unroll
                        for (uint32_t k = 0; k < W; k++)
                            if (k < lim) *reinterpret_cast<uint4 *>(dst + (size_t)k * g.N + gi) = v[k];
                    }
                }
            } else {
                for (uint32_t o = tid; o < RO; o += NT) {
                    const uint32_t oq = fast_div(o, mX), gi = sh.rowbase[sh.ownrow[oq]] + (o - oq * X);
#pragma unroll
                    for (uint32_t k = 0; k < W; k++) dst[(size_t)k * g.N + gi] = out[k * RO + o];
                }
            }
        } else {
            // IntLattices: the particles are written, zeros above them follow.
            if (X % 4u == 0) {
                const uint32_t q = X / 4u, nit = cty * ctz * q;
                for (uint32_t i0 = 0; i0 < nit; i0 += NT) {
                    const uint32_t i = i0 + tid;
                    const bool in = i < nit;
                    uint32_t gi = 0, held[4] = {0, 0, 0, 0}, top = 0;
                    if (in) {
                        const uint32_t oq = fast_div(i, ts.magic_q), r = sh.ownrow[oq], x = 4u * (i - oq * q);
                        const uint32_t l = r * X + x;
                        gi = sh.rowbase[r] + x;
                        uint32_t below[4], above[4], own[4] = {0, 0, 0, 0}, st[4] = {0, 0, 0, 0};
                        load_sites<4>(P.m + l - dz, below);
                        load_sites<4>(P.m + l + dz, above);
                        if constexpr (S <= 8) {
                            load_sites<4>(P.m + l, own);
                        } else {
                            const uint2 h = *reinterpret_cast<const uint2 *>(P.stays() + l);
                            st[0] = h.x & 0xFFFFu;
                            st[1] = h.x >> 16;
                            st[2] = h.y & 0xFFFFu;
                            st[3] = h.y >> 16;
                        }
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            held[j] = Ch::clamp(own[j], st[j], below[j], above[j]);
                            top = max(top, held[j]);
                        }
                    }
                    uint32_t lim = W;
                    const uint32_t most = top;
                    if (pb_dst) {
                        // Eight lanes hold a segment of 32 sites.
                        const uint32_t old = in ? min(pb_dst[gi >> PB_SHIFT], W) : 0u;
#pragma unroll
                        for (int o = 1; o < 8; o <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
                        lim = max(top, old);
                        if (in && (tid & 7u) == 0) pb_dst[gi >> PB_SHIFT] = top;
                    }
                    if (in) {
                        for (uint32_t k = 0; k < lim; k++) {
                            uint32_t *at = dst + (size_t)k * g.N + gi;
                            if (k >= most) {
                                *reinterpret_cast<uint4 *>(at) = make_uint4(0u, 0u, 0u, 0u);
                            } else {
#pragma unroll
                                for (int j = 0; j < 4; j++)
                                    if (k >= held[j]) at[j] = 0u;
                            }
                        }
                    }
                }
            } else {
                for (uint32_t o = tid; o < RO; o += NT) {
                    const uint32_t oq = fast_div(o, mX), r = sh.ownrow[oq], x = o - oq * X, l = r * X + x;
                    for (uint32_t k = P.count(l, l - dz, l + dz); k < W; k++)
                        dst[(size_t)k * g.N + sh.rowbase[r] + x] = 0u;
                }
            }
        }
    }

    // The reactions of the listed sites, or of every site that may react when
    // the model has zeroth-order reactions or the list was too short, and the
    // species counts of the tile when they are taken.
    __device__ __forceinline__ void react(uint32_t n, uint32_t *__restrict__ dst, uint32_t *__restrict__ pb_dst)
    {
        const uint32_t ncand = sh.ncand;
        const bool scan = scan_all || ncand > LIST_CAND;
        if (counting)
            for (uint32_t b = tid; b < LIST_HIST; b += NT) hist[b] = 0;
        if (counting || scan || ncand) __syncthreads();
        const uint32_t count_ns = counting ? rs->count_ns : 0u;
        if (counting) {
            for (uint32_t j = tid; j < n; j += NT) {
                const uint32_t p = list[j] >> LIST_P;
                if (p) atomicAdd(&hist[p <= count_ns ? p : 0u], 1u);
            }
        }
        if (scan || ncand) {
            const uint32_t total = scan ? RO : ncand;
            // Candidates go round the warps, so that the few of a tile do not
            // share one.
            constexpr uint32_t NW = NT / 32;
            for (uint32_t c0 = 0; c0 < total; c0 += NT) {
                const uint32_t c = c0 + (scan ? tid : (tid & 31u) * NW + (tid >> 5));
                if (c >= total) continue;
                uint32_t l, r;
                if (scan) {
                    const uint32_t oq = fast_div(c, mX);
                    r = sh.ownrow[oq];
                    l = r * X + (c - oq * X);
                } else {
                    l = sh.cand[c];
                    r = fast_div(l, mX);
                }
                const uint32_t x = l - r * X, gi = sh.rowbase[r] + x, t = T[l];
                const uint32_t np = P.count(l, l - dz, l + dz);
                if (scan) {
                    const ReactBound b = react_bound(t, mt);
                    if (np == 0 && b.a0 == 0.0f) continue;
                    if (!reaction_may_fire(np, b, hash_float((unsigned long long)gi << 1, th[3]))) continue;
                }
                SiteWords<BPS, S> s;
                if constexpr (BPS == 1) {
                    const uint32_t o = (sh.rowinfo[r] & ROW_INDEX) * X + x;
#pragma unroll
                    for (uint32_t k = 0; k < W; k++) s.w[k] = out[k * RO + o];
                } else {
                    s.load_first(dst, g.N, gi, np);
                }
                if (counting) {
#pragma unroll
                    for (int k = 0; k < S; k++) {
                        const uint32_t p = s.slot(k);
                        if (p) atomicSub(&hist[p <= count_ns ? p : 0u], 1u);
                    }
                }
                if (list_react<BPS, S>(s, t, gi, th[3], mt, rs, queue, cap)) {
                    s.store(dst, g.N, gi);
                    if (pb_dst) {
                        const uint32_t held = (uint32_t)__popc(occupied_slots<BPS, S>(s));
                        if (held) cover_slot<BPS>(pb_dst, gi, held - 1u);
                    }
                }
                if (counting) {
#pragma unroll
                    for (int k = 0; k < S; k++) {
                        const uint32_t p = s.slot(k);
                        if (p) atomicAdd(&hist[p <= count_ns ? p : 0u], 1u);
                    }
                }
            }
        }
        if (counting) {
            __syncthreads();
            for (uint32_t b = tid; b < LIST_HIST && b <= count_ns; b += NT)
                if (hist[b]) atomicAdd(rs->counts + b, (unsigned long long)hist[b]);
        }
    }
};

template <int BPS, int S, int NT>
__device__ __forceinline__ void list_tile(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst,
                                          const uint8_t *__restrict__ sites, const Geometry &g, const DevTables &m,
                                          RunState *__restrict__ rs, OverflowEntry *__restrict__ queue, uint32_t cap,
                                          const TileShape &ts, int with_reaction, const uint32_t *__restrict__ pb_src,
                                          uint32_t *__restrict__ pb_dst, uint32_t smem_bytes, uint32_t tile,
                                          uint32_t ntiles)
{
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ ListShared sh;
    ListTile<BPS, S, NT> t(smem, smem_bytes, g, m, rs, queue, cap, ts, with_reaction, sh, tile);
    const uint32_t tid = threadIdx.x;
    t.begin();
    t.load_types(sites);
    chain_enter();  // everything below may depend on the timestep before
    const int32_t status = rs->status;
    const uint32_t seed = rs->seed, step = rs->step, end_step = rs->end_step;
    t.counting = step == rs->count_step;
#pragma unroll
    for (int k = 0; k < 4; k++) t.th[k] = rs->th[k];

    bool first = true;
    for (;;) {
        if (!first) {
            t.begin();
            t.load_types(sites);
        }
        t.take_histogram();
        t.load(src, pb_src);
        if (status != LMB_OK || step >= end_step) return;  // the same for the whole block
        __syncthreads();
        const uint32_t n = sh.count;
        first = false;
        if (n > t.C) {
            // Too many particles for the list (the host sizes the next run's
            // list for more): a smaller sub-tile from the same corner.  z
            // first, then y (with one z plane, so that y pieces only ever
            // split a single plane of rows).
            if (tid == 0 && t.R == ts.R) {
                atomicAdd(&rs->list_split, 1u);
                atomicAdd(&rs->list_over, (unsigned long long)n);
                atomicMax(&rs->list_most, n);
            }
            if (t.y0 == 0 && t.ctz > 1u) {
                t.ctz = (t.ctz + 1u) / 2u;
            } else if (t.cty > 1u) {
                t.cty = (t.cty + 1u) / 2u;
            } else {  // not reached: the plan leaves room for a full region of one row
                if (tid == 0) rs->status = LMB_E_UNSUPPORTED;
                return;
            }
            __syncthreads();
            continue;
        }
        t.sweeps(n, dst);
        t.write_rows(dst, pb_dst);
        t.react(n, dst, pb_dst);

        // The next sub-tile, if the tile was split.
        t.y0 += t.cty;
        if (t.y0 >= ts.Ty) {
            t.y0 = 0;
            t.z0 += t.ctz;
            if (t.z0 >= ts.Tz) break;
            t.cty = ts.Ty;
            if (t.z0 + t.ctz > ts.Tz) t.ctz = ts.Tz - t.z0;
        } else if (t.y0 + t.cty > ts.Ty) {
            t.cty = ts.Ty - t.y0;
        }
        __syncthreads();
    }

    // The last block to finish resolves the overflow queue and advances the
    // step counter.  The count of finished blocks comes with the queue's
    // length (pushes and counts are atomics on one word), so an empty queue
    // costs no further round trip.
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const unsigned long long prev = atomicAdd(run_word(rs), 1ull);
        sh.last = (uint32_t)prev == ntiles - 1u;
        sh.count = (uint32_t)(prev >> 32);
    }
    __syncthreads();
    if (!sh.last) return;
    if (sh.count == 0) {
        if (tid < 4u) rs->th[tid] = timestep_hash(seed, step + 1u, tid);
        if (tid == 0) {
            rs->step = step + 1u;
            rs->tiles_done = 0;
        }
        return;
    }
    __threadfence();
    if (tid == 0) rs->tiles_done = 0;
    resolve_block_flat<BPS, S>(dst, sites, g, rs, queue, cap, reinterpret_cast<OverflowEntry *>(smem), tid, NT, pb_dst,
                               t.counting ? rs->counts : nullptr);
}

template <int BPS, int S, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) list_step_kernel(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst,
                                                            const uint8_t *__restrict__ sites, Geometry g,
                                                            const __grid_constant__ DevTables m,
                                                            RunState *__restrict__ rs,
                                                            OverflowEntry *__restrict__ queue, uint32_t cap,
                                                            const __grid_constant__ TileShape ts, int with_reaction,
                                                            const uint32_t *pb_src, uint32_t *pb_dst,
                                                            uint32_t smem_bytes)
{
    list_tile<BPS, S, NT>(src, dst, sites, g, m, rs, queue, cap, ts, with_reaction, pb_src, pb_dst, smem_bytes,
                          blockIdx.x, gridDim.x);
}

// A batch of lattices advanced together, as fused_batch_kernel does it.  The
// threads look for the block's job side by side (a binary search is a chain of
// round trips), and the job is worked from a copy in shared memory.
template <int BPS, int S, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) list_batch_kernel(const FusedJob *__restrict__ jobs, uint32_t njobs,
                                                             uint32_t parity, uint32_t smem_bytes)
{
    __shared__ uint32_t s_job;
    __shared__ __align__(16) uint32_t s_copy[(sizeof(FusedJob) + 3) / 4];
    for (uint32_t j = threadIdx.x; j < njobs; j += NT)
        if (jobs[j].tile_begin <= blockIdx.x && (j + 1u == njobs || jobs[j + 1u].tile_begin > blockIdx.x)) s_job = j;
    __syncthreads();
    const uint32_t *from = reinterpret_cast<const uint32_t *>(jobs + s_job);
    for (uint32_t w = threadIdx.x; w < sizeof(FusedJob) / 4u; w += NT) s_copy[w] = from[w];
    __syncthreads();
    const FusedJob &j = *reinterpret_cast<const FusedJob *>(s_copy);
    const uint32_t c = j.cur0 ^ parity;
    list_tile<BPS, S, NT>(j.buf[c], j.buf[c ^ 1], j.sites, j.g, j.m, j.rs, j.list, j.cap, j.ts, j.with_reaction,
                          nullptr, nullptr, smem_bytes, blockIdx.x - j.tile_begin, j.ts.tiles_y * j.ts.tiles_z);
}

// ---------------------------------------------------------------------------
// Planning and launch
// ---------------------------------------------------------------------------

// Static shared memory of the kernels, and the alignment it costs.
constexpr size_t LIST_STATIC_SMEM = sizeof(ListShared) + 64;

static uint32_t list_magic(uint32_t d) { return d <= 1 ? 0u : (uint32_t)((0x100000000ull + d - 1) / d); }

// Bytes of a Ty x Tz region besides the list (the tables excluded).
static size_t list_fixed_bytes(uint32_t X, int bps, int slots, uint32_t Ty, uint32_t Tz)
{
    const uint32_t W = bps == 1 ? slots / 4 : slots;
    const uint32_t R = X * (Ty + 2) * (Tz + 2), RO = X * Ty * Tz;
    const uint32_t mw = slots <= 8 ? Choices<8>::words(R) : Choices<16>::words(R);
    const uint32_t ow = bps == 1 ? (W * RO + 3u) & ~3u : 0u, second = std::max(slots <= 8 ? mw : 0u, ow);
    return 4 * (size_t)(mw + second) + ((R + 15u) & ~15u);
}

size_t list_smem_bytes(const Geometry &g, int bps, int slots, uint32_t Ty, uint32_t Tz, float density, bool &fits)
{
    fits = false;
    if (slots > 16 || g.X > 1024) return 0;
    const size_t R = (size_t)g.X * (Ty + 2) * (Tz + 2);
    if (R > LIST_MAX_REGION) return 0;
    // Always room for a full region of one row, the smallest sub-tile, and
    // the histogram.
    const size_t fixed = list_fixed_bytes(g.X, bps, slots, Ty, Tz);
    const size_t least = std::max(list_fixed_bytes(g.X, bps, slots, 1, 1) + 4 * ((size_t)9 * g.X * slots + LIST_HIST),
                                  fixed + 4 * (size_t)(LIST_HIST + 256));
    if (least > LIST_MAX_SMEM) return 0;
    // The list: the region's expected particles, an eighth and five standard
    // deviations of an even spread more; never more than its slots.  A list
    // cut short by the limit, or by particles that crowd, costs splits, not
    // results.
    const double mean = (double)density * (double)R;
    const double want = std::min(1.125 * mean + 5.0 * std::sqrt(mean) + 64.0, (double)R * slots);
    const size_t bytes = (std::max(fixed + 4 * (size_t)want, least) + 1023) & ~(size_t)1023;
    fits = bytes <= LIST_MAX_SMEM;
    return std::min(bytes, LIST_MAX_SMEM);
}

// Blocks with `smem` bytes of dynamic shared memory that an SM's 228 KB hold
// (the static part and 1 KB reserved per block included).
static uint32_t list_blocks_fit(size_t smem) { return (uint32_t)((228u * 1024u) / (smem + LIST_STATIC_SMEM + 1024u)); }

// Threads of a block: 256 for small regions, whose few particles finish their
// passes sooner with fewer warps at each barrier; 512, two blocks to an SM;
// 1024 where the region leaves room for one block only.
static uint32_t list_threads(uint32_t R, size_t smem)
{
    if (R <= LIST_SMALL_REGION) return 256u;
    return list_blocks_fit(smem) >= 2u ? 512u : 1024u;
}

// Estimated SM cycles of a timestep with tiles of this shape, for choosing
// among shapes.  Fitted to the shapes measured on the crowded cell (0.24
// particles per site), 96^3 at 1.25, the rod cell (0.01) and two ragged
// lattices: about 5 instructions per region site and 15 per region particle,
// an SM's rate growing with its resident warps towards 3 per cycle, a floor of
// 6000 cycles for a block's chain of passes; waves of 148 SMs.
// Where particles crowd, the launch lasts at least as long as its fullest
// tile, whose SM's other tiles are soon done.
double list_cost(uint32_t tiles, uint32_t R, size_t smem, float density, float crowd)
{
    const uint32_t warps = list_threads(R, smem) / 32u, fit = list_blocks_fit(smem);
    const uint32_t per_sm = std::max(1u, std::min(fit, 32u / warps));  // blocks an SM holds
    auto wave = [&](uint32_t blocks, float d) {
        const double instr = 3000.0 + (5.1 + 15.1 * (double)d) * (double)R;
        const double w = (double)(warps * blocks), rate = 3.0 * w / (w + 14.0);
        return std::max(6000.0, blocks * instr / rate);
    };
    const uint32_t slots = 148u * per_sm, full = tiles / slots, rest = tiles - full * slots;
    const double even = full * wave(per_sm, density) + (rest ? wave((rest + 147u) / 148u, density) : 0.0);
    return crowd > density ? std::max(even, wave(1u, crowd)) : even;
}

void list_fill_shape(const Geometry &g, TileShape &ts)
{
    ts.magic_x = list_magic(g.X);
    ts.magic_q = list_magic(g.X / 4);
}

#define LIST_VARIANTS(X_)                                        \
    X_(1, 4) X_(1, 8) X_(1, 16) X_(4, 4) X_(4, 8) X_(4, 16)

cudaError_t launch_list(int bps, int slots, const uint32_t *src, uint32_t *dst, const uint8_t *sites,
                        const Geometry &g, const DevTables &m, RunState *rs, OverflowEntry *queue, uint32_t cap,
                        const TileShape &ts, int with_reaction, const uint32_t *pb_src, uint32_t *pb_dst,
                        cudaStream_t stream)
{
    const size_t sort = (size_t)pow2_at_least(cap) * sizeof(OverflowEntry);
    const dim3 grid(ts.tiles_y * ts.tiles_z);
    size_t smem = std::max((size_t)ts.list_smem + m.stage_bytes, sort);
    // More tiles than fit at once: the list takes what the blocks of an SM
    // leave (a tile where particles crowd is split less often).  With fewer,
    // the room lets the next timestep's blocks in early.
    const uint32_t fit = std::min(list_blocks_fit(smem), 1024u / list_threads(ts.R, smem));
    if (fit >= 1u && grid.x > 148u * fit)
        smem = std::max(smem, std::min((228u * 1024u / fit - LIST_STATIC_SMEM - 1024u) & ~(size_t)1023, LIST_MAX_SMEM));
    const bool small = list_threads(ts.R, smem) == 256u;
    cudaError_t e = cudaErrorInvalidValue;
    count_launch();
#define LIST_LAUNCH(BPS_, S_)                                                                                     \
    if (bps == BPS_ && slots == S_) {                                                                             \
        if (small) {                                                                                              \
            if ((e = raise_smem_limit<list_step_kernel<BPS_, S_, 256, 4>>(smem)) != cudaSuccess) return e;          \
            return launch_chain(list_step_kernel<BPS_, S_, 256, 4>, grid, dim3(256), smem, stream, src, dst, sites, \
                                g, m, rs, queue, cap, ts, with_reaction, pb_src, pb_dst, (uint32_t)smem);          \
        }                                                                                                         \
        if (list_threads(ts.R, smem) == 1024u) {                                                                  \
            if ((e = raise_smem_limit<list_step_kernel<BPS_, S_, 1024, 1>>(smem)) != cudaSuccess) return e;         \
            return launch_chain(list_step_kernel<BPS_, S_, 1024, 1>, grid, dim3(1024), smem, stream, src, dst, sites, \
                                g, m, rs, queue, cap, ts, with_reaction, pb_src, pb_dst, (uint32_t)smem);          \
        }                                                                                                         \
        if ((e = raise_smem_limit<list_step_kernel<BPS_, S_, 512, 2>>(smem)) != cudaSuccess) return e;              \
        return launch_chain(list_step_kernel<BPS_, S_, 512, 2>, grid, dim3(512), smem, stream, src, dst, sites, g, m, \
                            rs, queue, cap, ts, with_reaction, pb_src, pb_dst, (uint32_t)smem);                    \
    }
    LIST_VARIANTS(LIST_LAUNCH)
#undef LIST_LAUNCH
    return e;
}

cudaError_t launch_list_batch(int bps, int slots, const FusedJob *jobs, uint32_t njobs, uint32_t total_tiles,
                              size_t smem, uint32_t parity, cudaStream_t stream)
{
    cudaError_t e = cudaErrorInvalidValue;
    count_launch();
#define LIST_LAUNCH(BPS_, S_)                                                                                  \
    if (bps == BPS_ && slots == S_) {                                                                          \
        if ((e = raise_smem_limit<list_batch_kernel<BPS_, S_, 512, 2>>(smem)) != cudaSuccess) return e;          \
        return launch_chain(list_batch_kernel<BPS_, S_, 512, 2>, dim3(total_tiles), dim3(512), smem, stream, jobs, \
                            njobs, parity, (uint32_t)smem);                                                    \
    }
    LIST_VARIANTS(LIST_LAUNCH)
#undef LIST_LAUNCH
    return e;
}

}  // namespace lmb
