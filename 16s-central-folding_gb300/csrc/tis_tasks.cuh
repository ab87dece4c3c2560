// Neighbour-list entries of a block's particles dealt out as equal tasks.
//
// The lists are short and uneven (2.9 SR entries on average, 0 to 40), so a thread per
// particle runs a warp as long as its longest list.  Here the entries are cut into tasks
// of one list chunk (nb_idx: four entries, 16 bytes) for one thread, full chunks first,
// then those with 3, 2 and 1 entries, so that the threads of a warp do equal work and a
// task's partners can be loaded together.
#pragma once
#include "tis_device.cuh"

namespace tis {

constexpr int kPairTasks = 512;  // tasks held in shared memory at a time

template <int PB>
struct TaskSmem {
    int4 at[PB];        // places of a particle's tasks: first full chunk, remainders (SR | LR << 16); its SR and LR entries
    int4 cnt[PB / 32];  // per 32 particles: tasks of a full chunk, of 3, 2, 1 entries
    int task[kPairTasks];
};

// a task: particle, list and entries of the chunk
__device__ __forceinline__ int task_particle(int t) { return t & 127; }
__device__ __forceinline__ bool task_lr(int t) { return (t >> 7) & 1; }
__device__ __forceinline__ int task_entries(int t) { return ((t >> 8) & 3) + 1; }
__device__ __forceinline__ int task_chunk(int t) { return t >> 10; }

// by threads tid = 0 .. PB - 1 (whole warps), each with its particle's list lengths; then a barrier.
// U: entries per task, 4 or 1
template <int PB, int U>
__device__ __forceinline__ void tasks_count(TaskSmem<PB> &sm, int tid, int ns, int nl)
{
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int UL = U == 4 ? 2 : 0;
    const int lane = tid & 31;
    const int full = (ns >> UL) + (nl >> UL);
    int incl = full;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += t;
    }
    const unsigned lt = (1u << lane) - 1u;
    int c[3] = {0, 0, 0}, as = 0, al = 0;
    if (U > 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned ms = __ballot_sync(kAll, (ns & 3) == 3 - k), ml = __ballot_sync(kAll, (nl & 3) == 3 - k);
            c[k] = __popc(ms) + __popc(ml);
            if ((ns & 3) == 3 - k) as = __popc(ms & lt);
            if ((nl & 3) == 3 - k) al = __popc(ms) + __popc(ml & lt);
        }
    sm.at[tid] = make_int4(incl - full, as | (al << 16), ns, nl);
    if (lane == 31) sm.cnt[tid >> 5] = make_int4(incl, c[0], c[1], c[2]);
}

template <int PB>
__device__ __forceinline__ int tasks_total(const TaskSmem<PB> &sm)
{
    int total = 0;
#pragma unroll
    for (int v = 0; v < PB / 32; ++v) total += sm.cnt[v].x + sm.cnt[v].y + sm.cnt[v].z + sm.cnt[v].w;
    return total;
}

// tasks win .. win + kPairTasks - 1 into sm.task, by threads tid = 0 .. PB - 1; then a barrier
template <int PB, int U>
__device__ __forceinline__ void tasks_window(TaskSmem<PB> &sm, int tid, int win)
{
    constexpr int UL = U == 4 ? 2 : 0;
    int4 first = make_int4(-win, -win, -win, -win);  // first task of each class of this particle's 32
#pragma unroll
    for (int v = 0; v < PB / 32; ++v) {
        const int4 n = sm.cnt[v];
        const bool lower = v < (tid >> 5);
        first.x += lower ? n.x : 0;
        first.y += n.x + (lower ? n.y : 0);
        first.z += n.x + n.y + (lower ? n.z : 0);
        first.w += n.x + n.y + n.z + (lower ? n.w : 0);
    }
    const int4 at = sm.at[tid];
    const int ns = at.z, nl = at.w;
    int to = first.x + at.x;
    for (int k = 0; k < (ns >> UL); ++k, ++to)
        if ((unsigned)to < (unsigned)kPairTasks) sm.task[to] = tid | ((U - 1) << 8) | (k << 10);
    for (int k = 0; k < (nl >> UL); ++k, ++to)
        if ((unsigned)to < (unsigned)kPairTasks) sm.task[to] = tid | (1 << 7) | ((U - 1) << 8) | (k << 10);
    if (U > 1) {
        const int rs = ns & 3, rl = nl & 3;
        to = (rs == 3 ? first.y : rs == 2 ? first.z : first.w) + (at.y & 0xffff);
        if (rs && (unsigned)to < (unsigned)kPairTasks) sm.task[to] = tid | ((rs - 1) << 8) | ((ns >> 2) << 10);
        to = (rl == 3 ? first.y : rl == 2 ? first.z : first.w) + (at.y >> 16);
        if (rl && (unsigned)to < (unsigned)kPairTasks) sm.task[to] = tid | (1 << 7) | ((rl - 1) << 8) | ((nl >> 2) << 10);
    }
}

}  // namespace tis
