// fk_groups.h -- how the stages of a unit are split into accumulator groups and
// chunks (fk_tc_contract.cuh: the MMA issuer and the epilogue walk the same groups).
// No CUDA types: a CPU test walks it.
#pragma once

#ifdef __CUDACC__
#define FK_HD __host__ __device__ __forceinline__
#else
#define FK_HD inline
#endif

namespace fk {

// The stage behind the group that starts at stage sg0 of nst: at most `width` stages, and not
// across a multiple of `bound` stages (0: no bound).
FK_HD int group_end(int sg0, int nst, int width, int bound) {
    int e = sg0 + width < nst ? sg0 + width : nst;
    if (bound) {
        const int m = (sg0 / bound + 1) * bound;
        e = m < e ? m : e;
    }
    return e;
}
// The stage behind the chunk of at most ch stages that starts at st0 of a group that ends at sg1.
FK_HD int chunk_end(int st0, int ch, int sg1) { return st0 + ch < sg1 ? st0 + ch : sg1; }
// Chunks of the group [sg0, sg1).
FK_HD int group_chunks(int sg0, int sg1, int ch) { return (sg1 - sg0 + ch - 1) / ch; }

}  // namespace fk
