// Order of a block's staged candidates by receptor type.
#pragma once

namespace agb {

// The place of this thread's candidate when the block's candidates are ordered
// by type (0-31), thread order within a type: a stable counting sort.  Each
// warp ranks its own candidates (its row of `cnt`: the count of each type),
// then one warp turns the counts into the first place of each (warp, type).
// cnt: WARPS rows of 32 ints in shared memory.  All threads call it, those
// without a candidate (in = false) with type 32; their result means nothing.
// It ends without a barrier: a thread may not write to memory that `cnt`
// shares before one.
template <int WARPS, class Counts>
__device__ __forceinline__ int type_sorted_place(Counts &cnt, int type, bool in)
{
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    cnt[w][lane] = 0;
    const unsigned same = __match_any_sync(0xffffffffu, type);
    const int rank = __popc(same & ((1u << lane) - 1u));
    // a type's count may be stored by another lane than its zero, and the
    // vote orders no memory
    __syncwarp();
    if (in && rank == 0) cnt[w][type] = __popc(same);
    __syncthreads();
    if (w == 0) {  // lane: a type's places, warps in order, after every lower type
        int n[WARPS], run = 0;
#pragma unroll
        for (int k = 0; k < WARPS; k++) {
            n[k] = cnt[k][lane];
            run += n[k];
        }
        int first = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, first, o);
            if (lane >= o) first += u;
        }
        first -= run;
#pragma unroll
        for (int k = 0; k < WARPS; k++) {
            cnt[k][lane] = first;
            first += n[k];
        }
    }
    __syncthreads();
    return in ? cnt[w][type] + rank : 0;
}

}  // namespace agb
