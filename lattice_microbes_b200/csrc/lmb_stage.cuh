// lmb_stage.cuh -- a block's copy of the model tables in shared memory.
#pragma once

#include "lmb_internal.h"

namespace lmb {

// Copies the model tables into shared memory at `dst` (16-byte aligned;
// stage_bytes long, each table at a 16-byte boundary) and returns a table set
// pointing there.  The device tables sit at 256-byte boundaries of one block
// (zero padded), so the copy moves whole 16-byte granules, every thread's
// loads independent of each other.
constexpr int NTABLES = 15;
__device__ __forceinline__ DevTables stage_tables(const DevTables &m, uint8_t *dst, uint32_t tid, uint32_t nthr)
{
    DevTables s = m;
    const void *srcs[NTABLES] = {m.T, m.qp0, m.qp1, m.qp2, m.order, m.D1, m.D2, m.rate, m.RL, m.stoich_off,
                                 m.stoich_sp, m.stoich_d, m.qpmax, m.rx_off, m.rx_list};
    const uint32_t sizes[NTABLES] = {m.nst * m.nst * m.ns * 4, m.nst * 4, m.nst * m.ns * 4,
                                     m.nst * m.ns * m.ns * 4, m.nr * 4, m.nr * 4, m.nr * 4, m.nr * 4,
                                     m.nr * m.nst, (m.nr + 1) * 4, m.nnz * 4, m.nnz * 4, 2 * m.nst * 4,
                                     (m.ns + 2) * 4, m.nr * 4};
    uint32_t first[NTABLES + 1];
    first[0] = 0;
#pragma unroll
    for (int k = 0; k < NTABLES; k++) first[k + 1] = first[k] + (sizes[k] + 15u) / 16u;
    uint4 *out = (uint4 *)dst;
    for (uint32_t gr = tid; gr < first[NTABLES]; gr += nthr) {
        const uint4 *src = (const uint4 *)srcs[0];
        uint32_t f = 0;
#pragma unroll
        for (int j = 1; j < NTABLES; j++)
            if (gr >= first[j]) {
                src = (const uint4 *)srcs[j];
                f = first[j];
            }
        out[gr] = __ldg(src + (gr - f));
    }
    const void *outs[NTABLES];
#pragma unroll
    for (int k = 0; k < NTABLES; k++) outs[k] = dst + 16u * first[k];
    s.T = (const float *)outs[0];
    s.qp0 = (const float *)outs[1];
    s.qp1 = (const float *)outs[2];
    s.qp2 = (const float *)outs[3];
    s.order = (const uint32_t *)outs[4];
    s.D1 = (const uint32_t *)outs[5];
    s.D2 = (const uint32_t *)outs[6];
    s.rate = (const float *)outs[7];
    s.RL = (const uint8_t *)outs[8];
    s.stoich_off = (const uint32_t *)outs[9];
    s.stoich_sp = (const uint32_t *)outs[10];
    s.stoich_d = (const int32_t *)outs[11];
    s.qpmax = (const float *)outs[12];
    s.rx_off = (const uint32_t *)outs[13];
    s.rx_list = (const uint32_t *)outs[14];
    return s;
}

}  // namespace lmb
