// Scene-major sweep on a thread-block cluster with the scene in distributed shared memory.
//
// For scenes small enough to live on-chip (the CPU-runnable 10^3 drop: 1000 vertices,
// 14.6k incidences), a cluster of C blocks (C <= 16, one per SM) takes one scene at a
// time from a work counter and runs all its iterations without touching global memory
// for positions or records:
//   * every block holds a copy of all the scene's states and rest positions (active and
//     fixed vertices) in its shared memory, and the neighbour and incidence records of the
//     vertices it owns: of each color, the block of rank r owns a chunk of whole slices of
//     kSlice vertices, whose records are one contiguous range of each record array;
//   * per color, each block solves its chunk (L lanes per vertex, neighbour states and
//     records from its own shared memory) and writes every new state into all C copies:
//     its own, and the other blocks' through distributed shared memory;
//   * a cluster barrier (release / acquire at cluster scope) separates colors, so the
//     next color reads the updated states from the local copy;
//   * after the last iteration each block writes its owned vertices back to global memory.
// Per color the critical path is shared-memory loads, the element arithmetic, the lane
// reduction, the 3x3 solve, C remote stores and one cluster barrier: no launch and no
// L2 round trip between colors. The per-vertex arithmetic is the solve kernels' (same
// incidence function, lane reduction and tail), so the results equal the merged and the
// single-block scene sweeps' for the same lanes per vertex.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vbd_kernels.cuh"

namespace gaia {
namespace dev {

namespace cg = cooperative_groups;

constexpr int kClusterMaxColors = 64;  // colors per scene that the per-block color table holds

// Neighbour states and rest positions from the block's shared copies; the staged neighbour
// records hold positions in those copies instead of slots.
template <typename ST>
struct FetchCluster {
    const typename ST::U* u;
    const float4* rest;
    __device__ __forceinline__ void operator()(int i, typename ST::U& q, float4& X) const {
        q = ST::nb(u[i]);
        X = rest[i];
    }
};

// Vertices of a color of n that one of C blocks owns: whole slices.
__host__ __device__ __forceinline__ int cluster_chunk(int n, int C) {
    const int per = (n + C - 1) / C;
    return (per + kSlice - 1) / kSlice * kSlice;
}

// The same where only the states fit in shared memory: records and rest positions are read
// through the caches, and the records' slots are looked up in the copy.
template <typename ST>
struct FetchClusterLean {
    const typename ST::U* u;
    const float4* rest;
    int4 sl;
    __device__ __forceinline__ void operator()(int s, typename ST::U& q, float4& X) const {
        q = ST::nb(u[s < sl.y ? s - sl.x : (sl.y - sl.x) + (s - sl.z)]);
        X = __ldg(rest + s);
    }
};

struct ClusterScenes {
    const int4* colors;        // slot ranges of the scenes' colors (scene-major slot layout): first,
                               // first of the vertices with long lists, end
    const int32_t* scene_ofs;  // colors of scene m: colors[scene_ofs[m] .. scene_ofs[m + 1])
    const int32_t* scene_order;
    const int4* scene_slots;   // per scene: active slots [x, y), fixed slots [z, w)
    int32_t nscenes, iterations, friction_start;
    int32_t pos_cap;           // states each block's shared copy holds
    int32_t nbr_cap, inc_cap;  // neighbour and incidence records each block holds
    SweepStage stage;
    const int4* ranges;        // per color, rank and kind of list (short, long): its record rows in the global
                               // arrays (colors of all scenes, 2 C per color): first and last + 1 of NbrRec
                               // and IncRec
};

// A compile-time number as an argument.
template <int N>
struct IntC {
    static constexpr int value = N;
};

// A state broadcast from lane src of the warp (every field of the trait's state type).
template <typename ST>
__device__ __forceinline__ typename ST::U shfl_state(typename ST::U u, int src) {
    constexpr int kWords = int(sizeof(typename ST::U) / 4);
    static_assert(sizeof(typename ST::U) % 4 == 0, "state of whole 32-bit words");
    uint32_t w[kWords];
    memcpy(w, &u, sizeof(u));
#pragma unroll
    for (int k = 0; k < kWords; ++k) w[k] = __shfl_sync(0xffffffffu, w[k], src);
    memcpy(&u, w, sizeof(u));
    return u;
}

// One block's chunk [beg, end) of a color's short or long lists: solved, and every new state
// written into all copies. nbr, inc: the records that vrec's rows count from.
template <int L, bool MULTI, bool LEAN, typename ST, typename R, typename Fetch>
__device__ __forceinline__ void cluster_range(const Ptrs<ST, R>& P, const Consts<R>& c, cg::cluster_group& cluster, int C,
                                              int beg, int end, const int4& sl, typename ST::U* spos, const float4* srest,
                                              const NbrRec<R>* nbr, const IncRec<R>* inc, unsigned char* stage, int cap,
                                              int warp_bytes, const Fetch& fetch, int friction) {
    using U = typename ST::U;
    constexpr int NB = L >= 16 ? 1 : 2;
    constexpr int RR = LEAN ? kRecKept : kRecShared;
    const int groups = int(blockDim.x) / L;
    const int g = int(threadIdx.x >> 5) * Lanes<L>::kW + Lanes<L>::vertex();
    const int sub = Lanes<L>::sub();
    for (int base = beg; base < end; base += groups) {
        const int v = base + g;
        const bool valid = v < end;
        Acc<R> acc = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        U uo{};
        MeshMat<R> mat{};
        float4 Xo = make_float4(0.f, 0.f, 0.f, 0.f);
        int4 seg = make_int4(0, 0, 0, 0);
        if (valid) {
            if (sub == 0) prefetch_tail<L>(P, v);
            seg = P.vrec[v];
            mat = P.mats[P.slot_mesh[v]];
            uo = spos[v - sl.x];
            Xo = LEAN ? __ldg(P.rest + v) : srest[v - sl.x];
        }
        const U uon = ST::nb(uo);
        SegRecs<R, NB> rec;
        const Stage<32 / L, ST, R> st = warp_stage<L, ST, R>(stage, cap, size_t(warp_bytes));
        preload<L, RR>(rec, nbr, inc, seg, sub);
        accumulate_segment<L, RR, false, ST>(rec, sub, st, fetch, uon, Xo, mat.mu, mat.lmbd, acc);
        if constexpr (MULTI)
            if (valid)
                accumulate_more<L, RR, false, ST>(rec, P, nbr, inc, P.vmore[v], sub, st, fetch, uon, Xo, mat.mu, mat.lmbd,
                                                  acc);
        __syncwarp();
        reduce_group<L, R>(acc);
        // lane 0 solves; the group's lanes then write the new state into the C
        // copies, one remote store each, instead of lane 0 writing all of them
        U un{};
        int moved = 0;
        if (valid && sub == 0) {
            finish_acc(acc, mat.mu, mat.lmbd);
            moved = vertex_tail<ST, R, false>(P, c, v, uo, Xo, frame_offset(P, v), mat, acc, friction, nullptr, nullptr, &un) ? 1 : 0;
        }
        const int src = Lanes<L>::vertex();
        moved = __shfl_sync(0xffffffffu, moved, src);
        un = shfl_state<ST>(un, src);
        if (valid && moved) {
            const int lv = v - sl.x;
            for (int r = sub; r < C; r += L) *cluster.map_shared_rank(&spos[lv], r) = un;
        }
    }
}

// LEAN: only the states in shared memory (nbr_cap and inc_cap 0), for a scene whose records
// and rest positions do not fit beside them. LONG: there are vertices with long lists.
template <int L, bool LONG, bool LEAN, typename ST, typename R>
__global__ void __launch_bounds__(256) k_sweep_cluster(Ptrs<ST, R> P, Consts<R> c, ClusterScenes S, int32_t* work) {
    using U = typename ST::U;
    constexpr int kKinds = LONG ? 2 : 1;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int C = int(cluster.num_blocks());
    extern __shared__ __align__(16) unsigned char smem[];
    U* spos = reinterpret_cast<U*>(smem);
    float4* srest = reinterpret_cast<float4*>(smem + sizeof(U) * size_t(S.pos_cap));
    NbrRec<R>* snbr = reinterpret_cast<NbrRec<R>*>(srest + (LEAN ? 0 : S.pos_cap));
    IncRec<R>* sinc = reinterpret_cast<IncRec<R>*>(snbr + S.nbr_cap);
    unsigned char* stage = reinterpret_cast<unsigned char*>(sinc + S.inc_cap);
    __shared__ int s_scene;
    __shared__ int2 s_rec_base[2 * kClusterMaxColors];
    for (;;) {
        // rank 0 takes the next scene and hands it to every block of the cluster
        if (rank == 0 && threadIdx.x == 0) {
            const int k = atomicAdd(work, 1);
            for (int r = 0; r < C; ++r) *cluster.map_shared_rank(&s_scene, r) = k;
        }
        cluster.sync();
        const int k = s_scene;
        if (k >= S.nscenes) return;
        const int sc = S.scene_order[k];
        const int c0 = S.scene_ofs[sc], c1 = S.scene_ofs[sc + 1];
        const int4 sl = S.scene_slots[sc];
        const int na = sl.y - sl.x;
        auto loc = [&](int s) { return s < sl.y ? s - sl.x : na + (s - sl.z); };
        const auto fetch = [&] {
            if constexpr (LEAN) return FetchClusterLean<ST>{spos, P.rest, sl};
            else return FetchCluster<ST>{spos, srest};
        }();
        // this block's chunk of the short (kind 0) or long lists of color ci: [beg, end)
        auto chunk = [&](int ci, int kind, int& beg, int& end) {
            const int4 rg = S.colors[ci];
            const int lo = kind ? rg.y : rg.x, hi = kind ? rg.z : rg.y;
            const int per = cluster_chunk(hi - lo, C);
            beg = min(hi, lo + rank * per);
            end = min(hi, beg + per);
        };
        auto rows = [&](int ci, int kind) { return S.ranges[2 * (ci * C + rank) + kind]; };
        // per chunk, the row where its records start in the shared arrays, less their global one
        if (!LEAN && threadIdx.x == 0) {
            int2 base = make_int2(0, 0);
            for (int ci = c0; ci < c1; ++ci)
                for (int k = 0; k < kKinds; ++k) {
                    const int4 r = rows(ci, k);
                    s_rec_base[2 * (ci - c0) + k] = make_int2(base.x - r.x, base.y - r.z);
                    base.x += r.y - r.x;
                    base.y += r.w - r.z;
                }
        }
        // stage: all the scene's states and rest positions, this block's records
        const int nloc = na + (sl.w - sl.z);
        for (int i = threadIdx.x; i < nloc; i += blockDim.x) {
            const int s = i < na ? sl.x + i : sl.z + (i - na);
            spos[i] = P.u[s];
            if (!LEAN) srest[i] = P.rest[s];
        }
        __syncthreads();
        for (int q = kKinds * c0; !LEAN && q < kKinds * c1; ++q) {
            const int ci = q / kKinds, k = q % kKinds;
            const int4 r = rows(ci, k);
            const int2 sb = s_rec_base[2 * (ci - c0) + k];
            const NbrRec<R>* gn = P.nbr + record_index(r.x, 0);
            const IncRec<R>* gi = P.inc + record_index(r.z, 0);
            NbrRec<R>* dn = snbr + (sb.x + r.x) * kSlice;
            IncRec<R>* di = sinc + (sb.y + r.z) * kSlice;
            for (int i = int(threadIdx.x); i < (r.y - r.x) * kSlice; i += blockDim.x) {
                NbrRec<R> n = gn[i];
                n.slot = loc(n.slot);
                dn[i] = n;
            }
            for (int i = int(threadIdx.x); i < (r.w - r.z) * kSlice; i += blockDim.x) di[i] = gi[i];
        }
        cluster.sync();  // every copy staged before any block writes into another's
        for (int it = 0; it < S.iterations; ++it) {
            const int friction = it >= S.friction_start ? 1 : 0;
            for (int ci = c0; ci < c1; ++ci) {
                auto solve = [&](auto lanes, auto multi, int kind, int cap) {
                    int beg, end;
                    chunk(ci, kind, beg, end);
                    const int2 sb = LEAN ? make_int2(0, 0) : s_rec_base[2 * (ci - c0) + kind];
                    const NbrRec<R>* nbr = LEAN ? P.nbr : snbr + ptrdiff_t(sb.x) * kSlice;
                    const IncRec<R>* inc = LEAN ? P.inc : sinc + ptrdiff_t(sb.y) * kSlice;
                    cluster_range<lanes.value, multi.value, LEAN, ST, R>(P, c, cluster, C, beg, end, sl, spos, srest, nbr, inc,
                                                                         stage, cap, S.stage.warp_bytes, fetch, friction);
                };
                solve(IntC<L>{}, IntC<0>{}, 0, S.stage.cap);
                if constexpr (LONG) solve(IntC<32>{}, IntC<1>{}, 1, S.stage.cap_long);
                cluster.sync();  // this color's states in every copy before the next color
            }
        }
        // the owned vertices back to global memory
        for (int q = kKinds * c0; q < kKinds * c1; ++q) {
            int beg, end;
            chunk(q / kKinds, q % kKinds, beg, end);
            for (int v = beg + int(threadIdx.x); v < end; v += blockDim.x) P.u[v] = spos[v - sl.x];
        }
        cluster.sync();  // no block stages the next scene while another still reads this one
    }
}

}  // namespace dev
}  // namespace gaia
