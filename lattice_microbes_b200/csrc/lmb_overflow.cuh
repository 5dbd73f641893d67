// lmb_overflow.cuh -- on-device overflow resolution, shared by the per-phase
// resolve kernel and the last block of the fused timestep kernel.
//
// The reference copies the whole lattice to the host when any particle
// overflowed and reinserts there (MpdRdmeSolver.cu:1103-1189).  Here one
// block sorts the step's queue by (phase, site, seq) -- one of the orders the
// reference's atomicAdd list can take -- and reinserts in that order with the
// same search, on the device.  Lattice words are read through L2 (ld.cg):
// other blocks of the same launch may have just written them.
#pragma once

#include "lmb.h"
#include "lmb_device.cuh"
#include "lmb_internal.h"
#include "lmb_site.cuh"

namespace lmb {

template <int BPS, int S>
__device__ __forceinline__ void load_site_cg(const uint32_t *lat, uint32_t N, uint32_t i, SiteWords<BPS, S> &s)
{
#pragma unroll
    for (int k = 0; k < SiteWords<BPS, S>::W; k++) s.w[k] = __ldcg(lat + (size_t)k * N + i);
}

// Raises the plane bound of site i's segment to cover slot k (pb may be
// null: the lattice keeps no plane bounds).
template <int BPS>
__device__ __forceinline__ void cover_slot(uint32_t *pb, uint32_t i, uint32_t k)
{
    if (pb) {
        const uint32_t planes = (BPS == 1 ? k >> 2 : k) + 1u;
        if (__ldcg(pb + (i >> PB_SHIFT)) < planes) atomicMax(pb + (i >> PB_SHIFT), planes);
    }
}

// First empty slot of site i gets p (ByteLattice.cpp:265-289); false if full.
template <int BPS, int S>
__device__ bool add_particle(uint32_t *lat, uint32_t N, uint32_t i, uint32_t p, uint32_t *pb)
{
    SiteWords<BPS, S> s;
    load_site_cg<BPS, S>(lat, N, i, s);
#pragma unroll
    for (int j = 0; j < S; j++) {
        if (s.slot(j) == 0) {
            s.put(j, p);
            s.store(lat, N, i);
            cover_slot<BPS>(pb, i, (uint32_t)j);
            return true;
        }
    }
    return false;
}

// A site has room exactly when its last slot is empty: resolution follows
// the sweeps, which leave every site packed (occupied slots first), and so do
// the reaction step and the insertions made here.
template <int BPS, int S>
__device__ __forceinline__ bool has_room(const uint32_t *lat, uint32_t N, uint32_t i)
{
    const uint32_t last = __ldcg(lat + (size_t)(SiteWords<BPS, S>::W - 1) * N + i);
    return BPS == 1 ? (last >> 24) == 0u : last == 0u;
}

constexpr uint32_t NO_SITE = ~0u;

// Target of a classic reinsertion (MpdRdmeSolver.cu:1113-1156): shells of
// radius 0..4 from Lattice::getNearbySites (Lattice.cpp:106-128: clamped to
// the lattice, x outer, y, z inner), first site of the same type with a free
// slot; NO_SITE when there is none.  The site itself and its six neighbours
// (radius 0 and 1) are looked at together, their loads in flight at once:
// nearly every search ends there.
template <int BPS, int S>
__device__ uint32_t classic_target(const uint32_t *lat, const uint8_t *sites, const Geometry &g, uint32_t idx)
{
    const uint32_t zc = idx / g.XY, rem = idx - zc * g.XY, yc = rem / g.X, xc = rem - yc * g.X;
    const uint32_t at[7] = {idx,
                            xc > 0 ? idx - 1u : NO_SITE,
                            yc > 0 ? idx - g.X : NO_SITE,
                            zc > 0 ? idx - g.XY : NO_SITE,
                            zc + 1u < g.Z ? idx + g.XY : NO_SITE,
                            yc + 1u < g.Y ? idx + g.X : NO_SITE,
                            xc + 1u < g.X ? idx + 1u : NO_SITE};
    uint8_t type[7];
    bool room[7];
#pragma unroll
    for (int j = 0; j < 7; j++) {
        const uint32_t i = at[j] != NO_SITE ? at[j] : idx;
        type[j] = sites[i];
        room[j] = has_room<BPS, S>(lat, g.N, i);
    }
    const uint8_t tc = type[0];
    uint32_t ok = 0;
#pragma unroll
    for (int j = 0; j < 7; j++) ok |= (at[j] != NO_SITE && type[j] == tc && room[j] ? 1u : 0u) << j;
#pragma unroll
    for (int j = 0; j < 7; j++)
        if ((ok >> j) & 1u) return at[j];
    for (uint32_t radius = 2; radius <= 4; radius++) {
        const uint32_t mind = radius - 1u, maxd = radius;
        const uint32_t min2 = mind * mind, max2 = maxd * maxd;
        const uint32_t x0 = xc >= maxd ? xc - maxd : 0, x1 = (xc + maxd < g.X) ? xc + maxd : g.X - 1;
        const uint32_t y0 = yc >= maxd ? yc - maxd : 0, y1 = (yc + maxd < g.Y) ? yc + maxd : g.Y - 1;
        const uint32_t z0 = zc >= maxd ? zc - maxd : 0, z1 = (zc + maxd < g.Z) ? zc + maxd : g.Z - 1;
        for (uint32_t x = x0; x <= x1; x++)
            for (uint32_t y = y0; y <= y1; y++)
                for (uint32_t z = z0; z <= z1; z++) {
                    const int32_t dx = (int32_t)(x - xc), dy = (int32_t)(y - yc), dz = (int32_t)(z - zc);
                    const uint32_t r2 = (uint32_t)(dx * dx + dy * dy + dz * dz);
                    if (r2 > max2 || r2 <= min2) continue;
                    const uint32_t j = x + y * g.X + z * g.XY;
                    if (sites[j] == tc && has_room<BPS, S>(lat, g.N, j)) return j;
                }
    }
    return NO_SITE;
}

// Smallest power of two >= n (n >= 1).
__host__ __device__ __forceinline__ uint32_t pow2_at_least(uint32_t n)
{
    uint32_t p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Resolves the step's overflow queue with the whole block (thread `tid` of
// `nthreads`); `sh` holds pow2_at_least(cap) entries.  On success the step
// counter advances.  pb: the lattice's plane bounds, raised for every slot
// filled here (null when it keeps none).  counts (when not null): species
// counts 0 .. rs->count_ns of the lattice being taken, to which every particle
// of those species put back is added.
template <int BPS, int S>
__device__ __noinline__ void resolve_block_flat(uint32_t *lat, const uint8_t *sites, const Geometry &g, RunState *rs,
                                   OverflowEntry *list, uint32_t cap, OverflowEntry *sh, uint32_t tid,
                                   uint32_t nthreads, uint32_t *pb, unsigned long long *counts = nullptr)
{
    const uint32_t n = *(volatile uint32_t *)&rs->ovf_count;
    const uint32_t carried = rs->carried;
    if (n == 0) {
        if (tid == 0) set_step(rs, rs->seed, rs->step + 1);
        return;
    }
    if (n > cap) {
        if (tid == 0) {
            rs->overflows += (unsigned long long)(n - carried);
            rs->status = LMB_E_OVERFLOW_EXHAUSTED;
            rs->failed_step = rs->step;
        }
        return;
    }
    const uint32_t p2 = pow2_at_least(n);
    for (uint32_t e = tid; e < p2; e += nthreads) {
        if (e < n) {
            OverflowEntry v;
            v.key = __ldcg(&list[e].key);
            v.site = __ldcg(&list[e].site);
            v.particle = __ldcg(&list[e].particle);
            sh[e] = v;
        } else {
            sh[e].key = ~0ull;
            sh[e].site = 0;
            sh[e].particle = 0;
        }
    }
    __syncthreads();
    if (n <= nthreads) {
        // Few entries: each thread counts the keys below its entry's (keys
        // are distinct) and moves it there.
        OverflowEntry v = {0ull, 0u, 0u};
        uint32_t rank = 0;
        if (tid < n) {
            v = sh[tid];
            for (uint32_t e = 0; e < n; e++) rank += sh[e].key < v.key ? 1u : 0u;
        }
        __syncthreads();
        if (tid < n) sh[rank] = v;
        __syncthreads();
    } else {
        // Bitonic sort by key.
        for (uint32_t k = 2; k <= p2; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t e = tid; e < p2; e += nthreads) {
                    const uint32_t o = e ^ j;
                    if (o > e) {
                        const bool up = (e & k) == 0;
                        const OverflowEntry a = sh[e], b = sh[o];
                        if ((a.key > b.key) == up) {
                            sh[e] = b;
                            sh[o] = a;
                        }
                    }
                }
                __syncthreads();
            }
        }
    }
    if (tid == 0) rs->overflows += (unsigned long long)(n - carried);
    if (rs->mode == LMB_OVERFLOW_CLASSIC) {
        // One entry per thread, in queue order.  Every thread finds its
        // entry's target from the lattice as it stands.  An insertion only
        // ever takes room away, from its own target, so an entry's target is
        // the one a search entry by entry finds as long as the target still
        // has room after the entries before it with the same one; they fill
        // its slots in order.  Up to the first entry for which it has none
        // left (or which has no target at all) everything is inserted at
        // once, and the rest search again.  (Entry by entry, each search and
        // insertion a chain of L2 round trips with the whole device waiting,
        // 107 entries of a 64^3 lattice took over 30 us of a timestep.)
        __shared__ uint32_t s_first;
        for (uint32_t base = 0; base < n;) {
            const uint32_t cnt = n - base < nthreads ? n - base : nthreads;
            const bool mine = tid < cnt;
            OverflowEntry v = {0ull, 0u, 0u};
            uint32_t target = NO_SITE, held = 0;
            if (tid == 0) s_first = cnt;
            if (mine) {
                v = sh[base + tid];
                target = classic_target<BPS, S>(lat, sites, g, v.site);
                if (target != NO_SITE) {
                    SiteWords<BPS, S> w;
                    load_site_cg<BPS, S>(lat, g.N, target, w);
                    held = (uint32_t)__popc(occupied_slots<BPS, S>(w));
                }
                sh[base + tid].key = target;  // the keys have served
            }
            __syncthreads();
            uint32_t slot = held;
            if (mine) {
                for (uint32_t e = 0; e < tid; e++) slot += (uint32_t)sh[base + e].key == target ? 1u : 0u;
                if (target == NO_SITE || slot >= (uint32_t)S) atomicMin(&s_first, tid);
            }
            __syncthreads();
            const uint32_t take = s_first;
            if (tid < take) {
                if (BPS == 1)
                    reinterpret_cast<uint8_t *>(lat + (size_t)(slot >> 2) * g.N + target)[slot & 3u] = (uint8_t)v.particle;
                else
                    lat[(size_t)slot * g.N + target] = v.particle;
                cover_slot<BPS>(pb, target, slot);
                if (counts && v.particle <= rs->count_ns) atomicAdd(counts + v.particle, 1ull);
            }
            const bool failed = take < cnt && (uint32_t)sh[base + take].key == NO_SITE;
            __syncthreads();
            if (failed) {  // the entries before it are in place
                if (tid == 0) {
                    rs->status = LMB_E_OVERFLOW_UNRESOLVED;
                    rs->failed_step = rs->step;
                }
                return;
            }
            base += take;
        }
        if (tid == 0) {
            rs->ovf_count = 0;
            rs->carried = 0;
        }
    } else if (tid == 0) {
        // Relaxed (MpdRdmeSolver.cu:1677-1761): own site only; the rest stay
        // queued, in order, for the next timestep.
        uint32_t kept = 0;
        for (uint32_t e = 0; e < n; e++) {
            if (!add_particle<BPS, S>(lat, g.N, sh[e].site, sh[e].particle, pb)) {
                OverflowEntry o = sh[e];
                o.key = (unsigned long long)kept;  // phase 0, list order
                list[kept++] = o;
            } else if (counts && sh[e].particle <= rs->count_ns) {
                atomicAdd(counts + sh[e].particle, 1ull);
            }
        }
        rs->ovf_count = kept;
        rs->carried = kept;
    }
    __threadfence();
    if (tid == 0) set_step(rs, rs->seed, rs->step + 1);
}

template <int BPS, int S>
__device__ void resolve_block(uint32_t *lat, const uint8_t *sites, const Geometry &g, RunState *rs,
                              OverflowEntry *list, uint32_t cap, OverflowEntry *sh, uint32_t *pb)
{
    resolve_block_flat<BPS, S>(lat, sites, g, rs, list, cap, sh, threadIdx.x, blockDim.x, pb);
}

}  // namespace lmb
