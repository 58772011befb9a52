// Device code of the GB300 VBD step.
//
// Precision modes (template parameters ST = state trait, R = compute type; see vbd_state.cuh):
//   fp32  <StF32, float>  : everything FP32
//   mixed <StDF,  float>  : displacements / inertia targets stored as double-float
//                           pairs; every per-incidence force and Hessian term, their
//                           accumulation and the 3x3 solve in FP32 (FP64 retry for
//                           ill-conditioned blocks). No FP64 instruction runs per
//                           incidence.
//   fp64  <StF64, double> : everything FP64 (the plain FP64 baseline)
//
// The state is the displacement u = x - X from the FP32 rest positions X, and
// the elastic terms are written in the displacement gradient G = F - I. Near
// rest, the reference's P = mu F + lambda (J - a) cof F is a difference of
// O(mu) terms (lambda (1 - a) = -mu), which costs FP32 three digits at strains
// of 1e-3; in G the same stress is mu (G - Cg) + lambda dJ (I + Cg) with
// Cg = cof(F) - I and dJ = det F - 1, built from small quantities only.
//
// Data layout in HBM (built once on the host, see vbd_engine.cu):
//   * vertices are renumbered into "slots": the solvable vertices of merged
//     color 0, then color 1, ..., then all fixed vertices. Per-slot arrays are
//     therefore contiguous per color and every per-vertex access of a color
//     sweep is coalesced.
//   * u[s]     = displacement and mass (ST::U: 16 B FP32, 32 B double-float or FP64)
//     rest[s]  = (X, Y, Z, unused)  float4, rest position
//     y[s]     = inertia target, as a displacement (ST::U)
//     xprev[s] = displacement at the start of the substep (ST::U)
//     vel[s]   = velocity (ST::V: FP32, or FP64 in the fp64 mode)
//   * per solvable vertex, in slot order, its one-ring and its incident tets:
//       NbrRec (8 B FP32, 16 B FP64): slot of a neighbour n and K_n = sum over the tets that
//         hold both vertices of A m_o . m_n (A = rest volume, m = rows of dF/dx, from the
//         FP64 DmInv), the material-free edge weight of the linear part of the force;
//       IncRec (8 B FP32, 16 B FP64): per incident tet the positions of its three other
//         vertices in the vertex's neighbour list (8 bits each, in the order whose rows have
//         determinant det DmInv, and the nearest one's again) and w = 1 / (6 A) = det DmInv.
//     The records of eight consecutive vertices are interleaved in rows (record k of a vertex
//     lies kSlice places after its record k - 1), so that lanes on neighbouring vertices read
//     neighbouring records. vrec[s] = (first rows, numbers and place in the row, see
//     record_index.hpp). Lists of more than kSegNbrs neighbours are cut into segments, the
//     further ones in vmore.
//
// Per vertex the Neo-Hookean block is evaluated in closed form from differences of rest
// positions, r = X_n - X_o, and of displacements, e = u_n - u_o. With (0, 1, 2) the tet's
// other vertices, N = (r1 - r0) x (r2 - r0) six times the rest area vector of the face
// opposite o over its height, D the same of the deformed face and C = D - N,
//   A m_o = -N / 6,  A cof(F) m_o = -D / 6,  6 A (det F - 1) = D . (r0 + e0) - N . r0
// so that, with G = F - I and G m_o = sum_n (m_n . m_o) e_n, the force and Hessian of
//   P = mu (G - (cof F - I)) + lambda (J - 1) cof F
// summed over the tets of o are
//   f = -mu sum_n K_n e_n - mu/6 sum_t C_t + lambda/6 sum_t (w S D)_t,  S = N.e0 + C.(r0 + e0)
//   H = lambda/6 sum_t (w D D^T)_t - mu sum_n K_n I
// (the same terms as the reference's contraction of its 9x9 d2E/dF2 with the vertex row of
// dF/dx, VBDPhysicsCompute.cu:2035-2232, VBD_NeoHookean.cpp:379-581: det F is affine in x_o,
// so the (J - a) d2J/dF2 term contracts to zero). Every difference is formed from small
// quantities: C = a x de + db x b' with a, b' edges and db, de differences of displacements.
//
// Where a tet is rotated, G is not small, and the parts of S, and the sums of K_n e_n and C,
// are large and cancel. In FP32 they keep what the stored rows of dF/dx gave:
//   * position 0 is the vertex opposite the longest edge of the face, so that the cross products
//     are of the two shorter edges, and S is taken at the vertex nearest to o (the fourth
//     position of IncRec): |N| |e| is then smallest against the tet's volume;
//   * S is two dot products with their rounding errors, sum K_n e_n a float pair over the
//     neighbours and over the lanes;
//   * the K_n are rounded so that the first moment of their rounding errors, sum dK_n r_n,
//     (nearly) vanishes, and with it their part in any linear motion e = A r.
// Error of a vertex's step from the elastic force against FP64, on a body of random tets,
// relative to the rows' (1.0): rotated by 0.3 rad 0.92, flattened to a tenth and rotated by
// 2 rad 0.92, as with stored rows 0.87 and 0.89 (tests/test_gpu_rotated_ring.py); without any of
// these 1.60 and 2.02. The 100^3 twist takes 9.4 ms a step with them, 8.1 without (the choice of the
// positions and the rounding of K_n, which cost nothing, alone: 1.07 and 1.49).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "cloth_dev.cuh"
#include "record_index.hpp"
#include "vbd_state.cuh"

namespace gaia {
namespace dev {

template <typename R>
struct MeshMat {
    R mu, lmbd, kh, kd, exp_damp, const_damp;
    int32_t init_type, pad;
};

template <typename R>
struct Consts {
    R dt, inv_dt, dt2inv;
    R kb, fr_mu, fr_epsU;
    R kc;  // collisionStiffness of the tet-mesh v-f contact
    R step, step_gd;
    double dt_d;
    double g[3];
    double lo[3], hi[3];
    float dt_f, g_f[3], lo_f[3], hi_f[3];  // the same constants for FP32 state arithmetic
    int32_t plane, assoc_grav;
    int32_t spin_limit;  // polls of a bounded wait before it gives up (kMbarSpinLimit unless a test lowers it)
};

// The FP64 or FP32 copy of a constant, matching the state scalar type.
template <typename Sc>
__device__ __forceinline__ Sc pick(double d, float f);
template <>
__device__ __forceinline__ float pick<float>(double, float f) { return f; }
template <>
__device__ __forceinline__ double pick<double>(double d, float) { return d; }

// Programmatic dependent launch: let the next grid in the stream start its
// prologue now, and wait for the previous grid's results (no-ops when the
// kernel was not launched as a programmatic dependent).
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Counter slots in device memory. CNT_TIMEOUT: blocks whose bounded wait on staged
// records (or on a grid barrier) ran out and that skipped their vertices; CNT_DRAIN: of
// those, blocks whose final drain wait ran out too.
enum { CNT_FP64_SOLVES = 0, CNT_FAILED_SOLVES = 1, CNT_NONFINITE = 2, CNT_TIMEOUT = 3, CNT_DRAIN = 4, CNT_N = 8 };

// One-ring and incidence records (see the top of the file), each one vector load.
template <typename R>
struct NbrRec;
template <>
struct alignas(8) NbrRec<float> {
    int32_t slot;
    float k;
};
template <>
struct alignas(16) NbrRec<double> {
    int32_t slot, pad;
    double k;
};
template <typename R>
struct IncRec;
template <>
struct alignas(8) IncRec<float> {
    uint32_t idx;
    float w;
};
template <>
struct alignas(16) IncRec<double> {
    uint32_t idx, pad;
    double w;
};

template <typename ST, typename R>
struct Ptrs {
    typename ST::U* u;
    const float4* rest;
    typename ST::U* y;
    typename ST::U* xprev;
    typename ST::V* vel;
    typename ST::V* vprev;
    const int4* vrec;          // per slot: first rows of its records and their numbers
    const int2* vmore;         // per slot its further segments [x, y) in segs; null: there are none
    const int4* segs;          // the further segments, as vrec
    const NbrRec<R>* nbr;
    const IncRec<R>* inc;
    const int32_t* slot_mesh;
    const MeshMat<R>* mats;
    unsigned long long* counters;
    int32_t nactive, nslots;
    // tet-mesh contact records (tet_cd.hpp; null when contact detection is off)
    const uint8_t* col_info;
    const int4* col_own;
    const int32_t* col_rel;
    const double2* mesh_fric;      // per mesh: frictionDynamic, frictionEpsV
    typename ST::U* snap;          // 2 per slot: states of the vertices with contact records as they
                                   // were after the previous iteration's solve of their color
    // mesh frames (null when off): per mesh the shift that the substep's initial step takes
    // out of every state of the mesh and the frame offset F (FP64); per slot the reference
    // position X + F as a float pair, which the world-box test uses in place of X
    const float4* frame_shift;
    const double4* frame_F;
    float4* rest_fh;
    float4* rest_fl;
};


struct DeformerDev {
    int32_t type;              // 0 rotator, 1 translator
    double axis[3], omega, end_time, speed[3];
};

struct DeformVerts {
    const int32_t* slot;
    const int32_t* def;        // deformer index
    const double* a;           // root (rotator) or original position (translator), 3 per vertex
    const double* b;           // root-relative point (rotator), 3 per vertex
    const DeformerDev* defs;
    int32_t n;
};

// ---------------------------------------------------------------------------
// small math
// ---------------------------------------------------------------------------
// Symmetric 3x3 solve by LDL^T (the same algorithm as the oracle's
// solve3x3_ldlt), with one reciprocal per pivot instead of two divisions (three IEEE
// divisions instead of six on the vertex's serial path; in FP64 a division is a dozen
// instructions of a pipe that issues one every 16 cycles). H = {h00, h01, h02, h11, h12, h22}.
template <typename R>
__device__ __forceinline__ bool ldlt3(const R* H, const R* b, R* x, R rel_tol) {
    const R scale = fmax(fabs(H[0]), fmax(fabs(H[3]), fabs(H[5])));
    if (!(scale > R(0))) return false;
    const R tol = rel_tol * scale;
    const R d0 = H[0];
    if (!(d0 > tol)) return false;
    const R r0 = R(1) / d0;
    const R l10 = H[1] * r0, l20 = H[2] * r0;
    const R d1 = H[3] - l10 * H[1];
    if (!(d1 > tol)) return false;
    const R r1 = R(1) / d1;
    const R l21 = (H[4] - l20 * H[1]) * r1;
    const R d2 = H[5] - l20 * H[2] - l21 * l21 * d1;
    if (!(d2 > tol)) return false;
    const R r2 = R(1) / d2;
    const R z0 = b[0];
    const R z1 = b[1] - l10 * z0;
    const R z2 = b[2] - l20 * z0 - l21 * z1;
    x[2] = z2 * r2;
    x[1] = z1 * r1 - l21 * x[2];
    x[0] = z0 * r0 - l10 * x[1] - l20 * x[2];
    return isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]);
}

// Relative pivot thresholds of the 3x3 LDL^T: an FP32 factorisation, the FP64 retry of an
// FP32-accumulated block, and an FP64 block. The retry's entries carry the rounding of
// their FP32 accumulation (a few 1e-7 of the largest diagonal after 10-30 incidences), so
// a pivot below kRetryPivot of it is rounding noise, not information: such a block is
// treated as singular (the gradient step) instead of being solved into a wild step.
constexpr float kFp32Pivot = 1e-5f;
constexpr double kRetryPivot = 2e-6;
constexpr double kFp64Pivot = 1e-12;

// FP32 solve with FP64 retry for ill-conditioned blocks; FP64 solve directly.
template <typename R>
__device__ __forceinline__ bool solve3(const R* H, const R* b, R* x, unsigned long long* counters);
template <>
__device__ __forceinline__ bool solve3<float>(const float* H, const float* b, float* x, unsigned long long* counters) {
    if (ldlt3<float>(H, b, x, kFp32Pivot)) return true;
    double Hd[6], bd[3], xd[3];
#pragma unroll
    for (int i = 0; i < 6; ++i) Hd[i] = H[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) bd[i] = b[i];
    atomicAdd(&counters[CNT_FP64_SOLVES], 1ull);
    if (!ldlt3<double>(Hd, bd, xd, kRetryPivot)) return false;
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i] = float(xd[i]);
    return true;
}
template <>
__device__ __forceinline__ bool solve3<double>(const double* H, const double* b, double* x, unsigned long long*) {
    return ldlt3<double>(H, b, x, kFp64Pivot);
}

// How records are read: streamed (once per launch), kept in the caches (every iteration by
// the persistent sweeps) or from shared memory.
enum RecRead { kRecStream = 0, kRecKept = 1, kRecShared = 2 };
template <int RR, typename T>
__device__ __forceinline__ T ld_rec(const T* p) {
    if constexpr (RR == kRecShared) {
        return *p;
    } else {
        T t;
        if constexpr (sizeof(T) == 8) {
            const int2 q = RR == kRecStream ? __ldcs(reinterpret_cast<const int2*>(p)) : __ldg(reinterpret_cast<const int2*>(p));
            memcpy(&t, &q, sizeof(t));
        } else {
            const int4 q = RR == kRecStream ? __ldcs(reinterpret_cast<const int4*>(p)) : __ldg(reinterpret_cast<const int4*>(p));
            memcpy(&t, &q, sizeof(t));
        }
        return t;
    }
}

// Accumulator of one vertex: force (3), lambda-part of the Hessian (6, upper
// triangle), and S = sum A mu |m_o|^2 (the isotropic part). FP32: k + l, sum K e over the
// neighbours as a float pair (before finish_acc).
template <typename R>
struct Acc {
    R f0, f1, f2, h00, h01, h02, h11, h12, h22, S;
    R k0, k1, k2, l0, l1, l2;
};

// Where a vertex's one-ring comes from. Global memory: either copied into the staging area
// asynchronously (past L1: the lines were written by earlier launches, earlier in the same
// kernel by the same block before a block barrier, or by other blocks before a grid barrier),
// or loaded into registers: Plain loads (states written by earlier launches or by the same
// block), or through L2 only (Grid: written by other blocks of the same launch). Never through
// the read-only path: the compiler may move such loads above the wait for the previous color.
enum StateRead { kStatePlain = 0, kStateGrid = 1 };
template <typename ST, int MODE>
struct FetchGlobal {
    const typename ST::U* u;
    const float4* rest;
    __device__ __forceinline__ void operator()(int s, typename ST::U& q, float4& X) const {
        if constexpr (MODE == kStateGrid) q = ST::ldcg(u, s);
        else q = ST::ld(u, s);
        X = __ldg(rest + s);
    }
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
// This thread's copies have landed (and are visible to it).
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A warp solves W = 32 / L vertices, L lanes each: lane i works on vertex i % W, as its
// sub-lane i / W. The lanes of a quarter warp are then on different vertices (up to L = 4),
// so that their accesses to shared memory fall into different banks, and the lanes on
// sub-lane 0, which run the vertex tails, are neighbours on neighbouring vertices.
template <int L>
struct Lanes {
    static constexpr int kW = 32 / L;
    __device__ __forceinline__ static int vertex() { return int(threadIdx.x) & (kW - 1); }   // within the warp
    __device__ __forceinline__ static int sub() { return (int(threadIdx.x) & 31) / kW; }
};

// A vertex's staged one-ring in shared memory: per neighbour e = u_n - u_o and r = X_n - X_o
// in the compute type, in 16-byte parts (each a plane of the warp's area, the entries of its W
// vertices interleaved; `cap` entries per vertex): FP32 {e, r.x} {r.y, r.z, -, -}, FP64
// {e.x, e.y} {e.z, r.x} {r.y, r.z}. The same parts first hold the neighbour as it lies in
// global memory (its state in ST::kNbParts parts, then its rest position) where it is copied
// asynchronously; the lane that copied an entry turns it into differences in place.
template <int W, typename ST, typename R>
struct Stage {
    static constexpr int kRaw = ST::kNbParts + 1;
    static constexpr int kParts = sizeof(R) == 8 ? 3 : kRaw;  // 16-byte parts per neighbour
    float4* p;
    int plane;
    __device__ __forceinline__ Stage(unsigned char* q, int cap, int v)
        : p(reinterpret_cast<float4*>(q) + v), plane(cap * W) {}
    __device__ __forceinline__ float4* part(int i, int k) const { return p + i * W + k * plane; }
    __device__ __forceinline__ void put(int i, const R* e, const R* r) const {
        if constexpr (sizeof(R) == 4) {
            *part(i, 0) = make_float4(e[0], e[1], e[2], r[0]);
            *reinterpret_cast<float2*>(part(i, 1)) = make_float2(r[1], r[2]);
        } else {
            *reinterpret_cast<double2*>(part(i, 0)) = make_double2(e[0], e[1]);
            *reinterpret_cast<double2*>(part(i, 1)) = make_double2(e[2], r[0]);
            *reinterpret_cast<double2*>(part(i, 2)) = make_double2(r[1], r[2]);
        }
    }
    __device__ __forceinline__ void get(int i, R* e, R* r) const {
        if constexpr (sizeof(R) == 4) {
            const float4 a = *part(i, 0);
            const float2 b = *reinterpret_cast<const float2*>(part(i, 1));
            e[0] = a.x; e[1] = a.y; e[2] = a.z;
            r[0] = a.w; r[1] = b.x; r[2] = b.y;
        } else {
            const double2 a = *reinterpret_cast<const double2*>(part(i, 0));
            const double2 b = *reinterpret_cast<const double2*>(part(i, 1));
            const double2 c = *reinterpret_cast<const double2*>(part(i, 2));
            e[0] = a.x; e[1] = a.y; e[2] = b.x;
            r[0] = b.y; r[1] = c.x; r[2] = c.y;
        }
    }
    // the neighbour in global slot s into entry i, asynchronously, and back out of it
    __device__ __forceinline__ void copy(int i, const typename ST::U* u, const float4* rest, int s) const {
        const float4* q = reinterpret_cast<const float4*>(u + s);
#pragma unroll
        for (int k = 0; k < ST::kNbParts; ++k) cp_async16(part(i, k), q + k);
        cp_async16(part(i, ST::kNbParts), rest + s);
    }
    __device__ __forceinline__ void raw(int i, typename ST::U& q, float4& X) const {
        float4 w[sizeof(typename ST::U) / 16] = {};
#pragma unroll
        for (int k = 0; k < ST::kNbParts; ++k) w[k] = *part(i, k);
        memcpy(&q, w, sizeof(q));
        X = *part(i, ST::kNbParts);
    }
};

// The staging area of this lane's vertex: the warps' areas (warp_bytes each) follow each other,
// `cap` entries per vertex.
template <int L, typename ST, typename R>
__device__ __forceinline__ Stage<32 / L, ST, R> warp_stage(unsigned char* smem, int cap, size_t warp_bytes) {
    using S = Stage<32 / L, ST, R>;
    return S(smem + size_t(threadIdx.x >> 5) * warp_bytes, cap, Lanes<L>::vertex());
}
template <int L, typename ST, typename R>
__device__ __forceinline__ Stage<32 / L, ST, R> warp_stage(unsigned char* smem, int cap) {
    return warp_stage<L, ST, R>(smem, cap, size_t(cap * (32 / L)) * (16 * Stage<32 / L, ST, R>::kParts));
}

// k + l += x y: l takes the rounding errors of product and sum (two-sum of k and fl(x y), the
// product's own error coming in with the last term).
__device__ __forceinline__ void pair_fma(float x, float y, float& k, float& l) {
    const float s = __fadd_rn(k, __fmul_rn(x, y));
    const float b = __fsub_rn(s, k);
    l = __fadd_rn(l, __fadd_rn(__fsub_rn(k, __fsub_rn(s, b)), __fmaf_rn(x, y, -b)));
    k = s;
}

// Two floats in a 64-bit register pair, operated on at once.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// N.e + C.p, which cancel where the tet is rotated: FP32 as two dot products, each a float pair
// (as pair_fma), the two in one packed sequence. Packed and scalar, the same operations, us a frame:
// 24 cubes, double-float, 1062 and 1105; collision drop, FP32, 2010 and 2100; 47^3 twist,
// double-float, 2076 and 2098; 100^3 twist and 200 cubes, FP32, 1% slower packed.
template <typename R>
__device__ __forceinline__ R volume_change(const R* N, const R* e, const R* C, const R* p) {
    if constexpr (sizeof(R) == 4) {
        F2 x = pack2(N[0], C[0]), y = pack2(e[0], p[0]);
        F2 s = mul2(x, y);
        F2 er = fma2(x, y, sub2(pack2(0.f, 0.f), s));
#pragma unroll
        for (int c = 1; c < 3; ++c) {
            x = pack2(N[c], C[c]);
            y = pack2(e[c], p[c]);
            const F2 t = add2(s, mul2(x, y));
            const F2 nb = sub2(s, t);
            er = add2(er, add2(sub2(s, add2(t, nb)), fma2(x, y, nb)));
            s = t;
        }
        float s0, s1, e0, e1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(s.v));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(e0), "=f"(e1) : "l"(er.v));
        return __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(e0, e1));
    } else {
        return (N[0] * e[0] + N[1] * e[1] + N[2] * e[2]) + (C[0] * p[0] + C[1] * p[1] + C[2] * p[2]);
    }
}

// One tet from its three other vertices' differences: C into cs, w S D into t, w D D^T into the
// accumulator's Hessian (unscaled, see finish_acc). es, rs: the vertex at the shortest rest edge.
template <typename R>
__device__ __forceinline__ void incidence(const R* e0, const R* e1, const R* e2, const R* r0, const R* r1, const R* r2,
                                          const R* es, const R* rs, R w, R* cs, R* t, Acc<R>& acc) {
    const R a[3] = {r1[0] - r0[0], r1[1] - r0[1], r1[2] - r0[2]};
    const R b[3] = {r2[0] - r0[0], r2[1] - r0[1], r2[2] - r0[2]};
    const R al[3] = {e1[0] - e0[0], e1[1] - e0[1], e1[2] - e0[2]};
    const R be[3] = {e2[0] - e0[0], e2[1] - e0[1], e2[2] - e0[2]};
    const R bd[3] = {b[0] + be[0], b[1] + be[1], b[2] + be[2]};
    // C = a x be + al x bd, N = a x b
    const R C0 = a[1] * be[2] - a[2] * be[1] + al[1] * bd[2] - al[2] * bd[1];
    const R C1 = a[2] * be[0] - a[0] * be[2] + al[2] * bd[0] - al[0] * bd[2];
    const R C2 = a[0] * be[1] - a[1] * be[0] + al[0] * bd[1] - al[1] * bd[0];
    const R N0 = a[1] * b[2] - a[2] * b[1], N1 = a[2] * b[0] - a[0] * b[2], N2 = a[0] * b[1] - a[1] * b[0];
    const R D0 = N0 + C0, D1 = N1 + C1, D2 = N2 + C2;
    const R N[3] = {N0, N1, N2}, C[3] = {C0, C1, C2}, p[3] = {rs[0] + es[0], rs[1] + es[1], rs[2] + es[2]};
    const R S = volume_change(N, es, C, p);
    const R w0 = w * D0, w1 = w * D1, w2 = w * D2;
    cs[0] += C0; cs[1] += C1; cs[2] += C2;
    t[0] += S * w0; t[1] += S * w1; t[2] += S * w2;
    acc.h00 += w0 * D0;
    acc.h01 += w0 * D1;
    acc.h02 += w0 * D2;
    acc.h11 += w1 * D1;
    acc.h12 += w1 * D2;
    acc.h22 += w2 * D2;
}

// The first records of a lane's share of a segment, loaded ahead of the state reads (they are
// static data): its first NB neighbours (sub, sub + L, ...) and its first two incidences.
// Record k of the segment is kSlice * k places after its first.
template <typename R, int NB>
struct SegRecs {
    NbrRec<R> n[NB];
    IncRec<R> i0, i1;
    const NbrRec<R>* np;  // the segment's records
    const IncRec<R>* ip;
    int nn, ni;           // their numbers (0 for a lane without a vertex)
};
template <int L, int RR, typename R, int NB>
__device__ __forceinline__ void preload(SegRecs<R, NB>& s, const NbrRec<R>* nbr, const IncRec<R>* inc, int4 seg,
                                        int sub) {
    s.np = nbr + record_index(seg.x, place_of(seg.z));
    s.ip = inc + record_index(seg.y, place_of(seg.z));
    s.nn = nbrs_of(seg.z);
    s.ni = seg.w;
#pragma unroll
    for (int j = 0; j < NB; ++j)
        if (sub + j * L < s.nn) s.n[j] = ld_rec<RR>(s.np + kSlice * (sub + j * L));
    if (sub < s.ni) s.i0 = ld_rec<RR>(s.ip + kSlice * sub);
    if (sub + L < s.ni) s.i1 = ld_rec<RR>(s.ip + kSlice * (sub + L));
}

// Neighbour records a lane holds at a time. ASYNC: the one-ring is copied into the staging area
// asynchronously, all of a vertex's neighbours (6 or 18 on a 5-tet lattice, about 14 on other
// meshes) in flight at once without occupying registers, at the price of a second pass over
// shared memory. Otherwise they are loaded into registers, two per lane at a time (one in
// the wide groups of small colors, which have one neighbour per lane).
template <int L, bool ASYNC>
struct NbrBatch {
    static constexpr int kN = L >= 16 ? 1 : (!ASYNC ? 2 : (L == 8 ? 3 : (L == 4 ? 5 : 9)));
};

// One lane's share of one segment: stages the segment's one-ring (neighbours sub, sub + L,
// ...; a narrow group reads each record twice, for the slot and then for K) in shared memory,
// adding the linear force on the way, then runs its incidences (sub,
// sub + L, ...) on the staged differences. Every lane
// of the warp calls it (lanes without a vertex with empty lists). Each neighbour state is
// read once per vertex instead of once per incidence, and the incidence loop has no
// dependent global load.
template <int L, int RR, bool ASYNC, typename ST, typename R, int NB, typename Fetch>
__device__ __forceinline__ void accumulate_segment(SegRecs<R, NB>& s, int sub, const Stage<32 / L, ST, R>& st, const Fetch& fetch,
                                                   const typename ST::U& uo, const float4& Xo, R mu, R lmbd,
                                                   Acc<R>& acc) {
    using U = typename ST::U;
    R kf[3] = {R(0), R(0), R(0)}, cs[3] = {R(0), R(0), R(0)}, t[3] = {R(0), R(0), R(0)};
    auto take = [&](int k, const U& q, const float4& X, R K) {
        R e[3];
        ST::diff(q, uo, e);
        const R r[3] = {R(X.x) - R(Xo.x), R(X.y) - R(Xo.y), R(X.z) - R(Xo.z)};
        st.put(k, e, r);
        if constexpr (sizeof(R) == 4) {
            pair_fma(K, e[0], acc.k0, acc.l0);
            pair_fma(K, e[1], acc.k1, acc.l1);
            pair_fma(K, e[2], acc.k2, acc.l2);
        } else {
            kf[0] += K * e[0];
            kf[1] += K * e[1];
            kf[2] += K * e[2];
        }
        acc.S += K;
    };
    if constexpr (ASYNC) {
        for (int k = sub; k < s.nn; k += NB * L) {
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (k + j * L < s.nn) st.copy(k + j * L, fetch.u, fetch.rest, s.n[j].slot);
            if (k + NB * L < s.nn) {
#pragma unroll
                for (int j = 0; j < NB; ++j)
                    if (k + (NB + j) * L < s.nn) s.n[j] = ld_rec<RR>(s.np + kSlice * (k + (NB + j) * L));
            }
        }
        cp_async_wait();
        for (int k = sub; k < s.nn; k += L) {
            U q;
            float4 X;
            st.raw(k, q, X);
            take(k, q, X, ld_rec<RR == kRecShared ? kRecShared : kRecKept>(s.np + kSlice * k).k);
        }
    } else {
        for (int k = sub; k < s.nn; k += NB * L) {
            U q[NB];
            float4 X[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (k + j * L < s.nn) fetch(s.n[j].slot, q[j], X[j]);
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                if (k + j * L >= s.nn) break;
                take(k + j * L, q[j], X[j], s.n[j].k);
                if (k + (j + NB) * L < s.nn) s.n[j] = ld_rec<RR>(s.np + kSlice * (k + (j + NB) * L));
            }
        }
    }
    __syncwarp();
    for (int k = sub; k < s.ni; k += L) {
        const IncRec<R> cur = s.i0;
        s.i0 = s.i1;
        if (k + 2 * L < s.ni) s.i1 = ld_rec<RR>(s.ip + kSlice * (k + 2 * L));
        R e0[3], e1[3], e2[3], r0[3], r1[3], r2[3];
        st.get(int(cur.idx & 255u), e0, r0);
        st.get(int((cur.idx >> 8) & 255u), e1, r1);
        st.get(int((cur.idx >> 16) & 255u), e2, r2);
        if constexpr (sizeof(R) == 4) {
            R es[3], rs[3];
            st.get(int(cur.idx >> 24), es, rs);
            incidence(e0, e1, e2, r0, r1, r2, es, rs, cur.w, cs, t, acc);
        } else {
            incidence(e0, e1, e2, r0, r1, r2, e0, r0, cur.w, cs, t, acc);
        }
    }
    const R m6 = mu * R(1.0 / 6.0), l6 = lmbd * R(1.0 / 6.0);
    acc.f0 += l6 * t[0] - m6 * cs[0] - mu * kf[0];
    acc.f1 += l6 * t[1] - m6 * cs[1] - mu * kf[1];
    acc.f2 += l6 * t[2] - m6 * cs[2] - mu * kf[2];
}

// The remaining segments of a vertex with more than kSegNbrs neighbours. Only the 32-lane
// solves of the long lists (MULTI) hold this loop: it costs registers.
template <int L, int RR, bool ASYNC, typename ST, typename R, int NB, typename Fetch>
__device__ __forceinline__ void accumulate_more(SegRecs<R, NB>& rec, const Ptrs<ST, R>& P, const NbrRec<R>* nbr,
                                                const IncRec<R>* inc, int2 more, int sub, const Stage<32 / L, ST, R>& st,
                                                const Fetch& fetch, const typename ST::U& uo, const float4& Xo, R mu,
                                                R lmbd, Acc<R>& acc) {
    static_assert(L == 32, "one vertex per warp");
    for (int i = more.x; i < more.y; ++i) {
        __syncwarp();
        preload<L, RR>(rec, nbr, inc, P.segs[i], sub);
        accumulate_segment<L, RR, ASYNC, ST>(rec, sub, st, fetch, uo, Xo, mu, lmbd, acc);
    }
}

// The accumulated sums in the units of the force and the Hessian (after the lane reduction).
template <typename R>
__device__ __forceinline__ void finish_acc(Acc<R>& a, R mu, R lmbd) {
    const R l6 = lmbd * R(1.0 / 6.0);
    a.h00 *= l6; a.h01 *= l6; a.h02 *= l6; a.h11 *= l6; a.h12 *= l6; a.h22 *= l6;
    a.S *= -mu;
    if constexpr (sizeof(R) == 4) {
        a.f0 -= mu * (a.k0 + a.l0);
        a.f1 -= mu * (a.k1 + a.l1);
        a.f2 -= mu * (a.k2 + a.l2);
    }
}

// One halving step of the reduce-scatter below: of n values, this lane keeps the lower or the
// upper half (rounded up; a missing one counts as zero) and adds its partner's share of it.
template <int N>
__device__ __forceinline__ void halve(double* v, int off, bool upper) {
    constexpr int H = (N + 1) / 2;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const double lo = v[i], hi = i + H < N ? v[i + H] : 0.0;
        const double got = __shfl_xor_sync(0xffffffffu, upper ? lo : hi, off);
        v[i] = (upper ? hi : lo) + got;
    }
}

// One halving step of N float pairs (k, l), as halve.
template <int N>
__device__ __forceinline__ void halve_pairs(float* k, float* l, int off, bool upper) {
    constexpr int H = (N + 1) / 2;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const float khi = i + H < N ? k[i + H] : 0.f, lhi = i + H < N ? l[i + H] : 0.f;
        const float ko = __shfl_xor_sync(0xffffffffu, upper ? k[i] : khi, off);
        const float lo = __shfl_xor_sync(0xffffffffu, upper ? l[i] : lhi, off);
        float s, e;
        two_sum(upper ? khi : k[i], ko, s, e);
        k[i] = s;
        l[i] = __fadd_rn(__fadd_rn(upper ? lhi : l[i], lo), e);
    }
}

// The three pairs of the accumulator over the L lanes of a vertex, rounded once, on sub-lane 0 (in
// k0, k1, k2): a lane holds two of them after the first step and one after the second.
template <int L>
__device__ __forceinline__ void reduce_pairs(Acc<float>& a) {
    constexpr int W = 32 / L;
    float k[3] = {a.k0, a.k1, a.k2}, l[3] = {a.l0, a.l1, a.l2};
    const int sub = Lanes<L>::sub(), vw = Lanes<L>::vertex();
    halve_pairs<3>(k, l, 16, (sub & (L / 2)) != 0);
    if constexpr (L >= 4) halve_pairs<2>(k, l, 8, (sub & (L / 4)) != 0);
#pragma unroll
    for (int off = 4; off >= W; off >>= 1) {
        const float ko = __shfl_xor_sync(0xffffffffu, k[0], off), lo = __shfl_xor_sync(0xffffffffu, l[0], off);
        float s, e;
        two_sum(k[0], ko, s, e);
        k[0] = s;
        l[0] = __fadd_rn(__fadd_rn(l[0], lo), e);
    }
    const float t = __fadd_rn(k[0], l[0]);
    a.k0 = t;
    a.k1 = L >= 4 ? __shfl_sync(0xffffffffu, t, (L / 4) * W + vw) : __fadd_rn(k[1], l[1]);
    a.k2 = __shfl_sync(0xffffffffu, t, (L / 2) * W + vw);
    a.l0 = a.l1 = a.l2 = 0.f;
}

// Sums over the L lanes of a vertex; valid on sub-lane 0.
template <int L, typename R>
__device__ __forceinline__ void reduce_group(Acc<R>& a) {
    constexpr int W = 32 / L;
    if constexpr (sizeof(R) == 8 && L >= 8) {
        // FP64 in wide groups: the adds of a butterfly over all ten sums (50 per lane at L = 32, as
        // many as two thirds of an incidence) cost more than the loop, as the FP64 pipe takes 16 cycles a warp
        // instruction. Each step halves the sums a lane holds (5, 3, 2, 1, 1 adds), and sub-lane 0
        // collects them at the end.
        double v[10] = {a.f0, a.f1, a.f2, a.h00, a.h01, a.h02, a.h11, a.h12, a.h22, a.S};
        const int sub = Lanes<L>::sub(), vw = Lanes<L>::vertex();
        // top bits of sub choose the halves: 10 -> 5 -> 3 -> 2 (-> 1)
        halve<10>(v, 16, (sub & (L / 2)) != 0);
        halve<5>(v, 8, (sub & (L / 4)) != 0);
        halve<3>(v, 4, (sub & (L / 8)) != 0);
        constexpr int kLeft = L >= 16 ? 1 : 2;  // sums held per lane
        if constexpr (L >= 16) halve<2>(v, 2, (sub & (L / 16)) != 0);
        if constexpr (L >= 32) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        // sum k sits on the lane whose choices lead to it: k = 5 b0 + 3 b1 + 2 b2 + b3
        double out[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) {
            const int b0 = k >= 5, k1 = k - 5 * b0, b1 = k1 >= 3, k2 = k1 - 3 * b1, b2 = k2 >= 2, k3 = k2 - 2 * b2;
            int src = b0 * (L / 2) + b1 * (L / 4) + b2 * (L / 8);
            if (kLeft == 1) src += k3 * (L / 16);
            out[k] = __shfl_sync(0xffffffffu, kLeft == 1 ? v[0] : v[k3], src * W + vw);
        }
        a = Acc<R>{out[0], out[1], out[2], out[3], out[4], out[5], out[6], out[7], out[8], out[9]};
    } else {
#pragma unroll
        for (int off = 16; off >= W; off >>= 1) {
            a.f0 += __shfl_xor_sync(0xffffffffu, a.f0, off);
            a.f1 += __shfl_xor_sync(0xffffffffu, a.f1, off);
            a.f2 += __shfl_xor_sync(0xffffffffu, a.f2, off);
            a.h00 += __shfl_xor_sync(0xffffffffu, a.h00, off);
            a.h01 += __shfl_xor_sync(0xffffffffu, a.h01, off);
            a.h02 += __shfl_xor_sync(0xffffffffu, a.h02, off);
            a.h11 += __shfl_xor_sync(0xffffffffu, a.h11, off);
            a.h12 += __shfl_xor_sync(0xffffffffu, a.h12, off);
            a.h22 += __shfl_xor_sync(0xffffffffu, a.h22, off);
            a.S += __shfl_xor_sync(0xffffffffu, a.S, off);
        }
        if constexpr (sizeof(R) == 4) reduce_pairs<L>(a);
    }
}

// IPC-style lagged friction (VBD_GeneralCompute.h:10-66; VBDPhysics.cpp:2563-2592)
// for an axis-aligned contact normal along `d`: tangents e_{d+1}, e_{d+2}.
template <typename R>
__device__ __forceinline__ void axis_friction(int d, const R* dx, R mu, R lambda, R epsU, R* f, R* H) {
    int t0 = (d + 1) % 3, t1 = (d + 2) % 3;
    R u0 = dx[t0], u1 = dx[t1];
    R un = sqrt(u0 * u0 + u1 * u1);
    if (!(un > R(0))) return;
    R f1 = un > epsU ? R(1) / un : (-un / epsU + R(2)) / epsU;
    R s = mu * lambda * f1;
    f[t0] -= s * u0;
    f[t1] -= s * u1;
    // H += s * (e_t0 e_t0^T + e_t1 e_t1^T): diagonal entries of the two tangents
    H[t0 == 0 ? 0 : (t0 == 1 ? 3 : 5)] += s;
    H[t1 == 0 ? 0 : (t1 == 1 ? 3 : 5)] += s;
}

// ---------------------------------------------------------------------------
// Per-color block solve. One group of L lanes per vertex of the color range
// [beg, end). PROBE = write force/Hessian of the single vertex `beg` to
// probe_out instead of moving it.
// ---------------------------------------------------------------------------
template <typename ST, typename R, bool PROBE>
__device__ __forceinline__ bool vertex_tail(const Ptrs<ST, R>& P, const Consts<R>& c, int v, const typename ST::U& uo,
                                            const float4& Xo, const float3& Fo, const MeshMat<R>& mat,
                                            const Acc<R>& acc, int friction, double* probe_out,
                                            const R* con, typename ST::U* unew = nullptr);

// ---------------------------------------------------------------------------
// Tet-mesh vertex-face contact (VBDPhysicsCompute.cu:1731-1773, 1812-1930)
// ---------------------------------------------------------------------------
template <typename R>
struct V3T;
template <>
struct V3T<float> {
    using type = float3;
};
template <>
struct V3T<double> {
    using type = double3;
};

// accumlateCollisionForceAndHessianPerCollision_v2: the contact of vertex sp with its
// recorded face, at the current positions, on the contact vertex of index `order`
// (3 = sp itself, 0..2 = a face vertex). Positions are taken relative to sp's: q - p =
// (X_q - X_p) + (u_q - u_p). Penalty k * depth along the face normal (interior closest
// point) or the closest-point direction oriented like the face normal, lagged IPC
// friction in the frame (edge AB, AB x n); scaled by b = 1 (sp) or -barycentric.
template <typename ST, typename R, typename Get>
__device__ __forceinline__ void contact_term(const Ptrs<ST, R>& P, const Consts<R>& c, const Get& state, int sp,
                                             int order, R* f, R* H) {
    using U = typename ST::U;
    using V = typename V3T<R>::type;
    const int4 fo = P.col_own[sp];
    const int fs[3] = {fo.x, fo.y, fo.z};
    const U up = state(sp);
    U uf[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) uf[k] = state(fs[k]);
    const float4 Xp = P.rest[sp];
    V q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 Xq = P.rest[fs[k]];
        R d[3];
        ST::diff(uf[k], up, d);
        q[k] = V{R(Xq.x) - R(Xp.x) + d[0], R(Xq.y) - R(Xp.y) + d[1], R(Xq.z) - R(Xp.z) + d[2]};
    }
    const V o{R(0), R(0), R(0)};
    V bary, cp;
    const int type = cloth::closest_point_triangle<V, R>(o, q[0], q[1], q[2], bary, cp);
    V fn = cloth::cross(cloth::sub(q[1], q[0]), cloth::sub(q[2], q[0]));
    const R fl = sqrt(cloth::dot(fn, fn));
    fn = V{fn.x / fl, fn.y / fl, fn.z / fl};
    const V diff = cp;
    V n;
    if (type == cloth::AtInterior) {
        n = fn;
    } else {
        const R inv = R(1) / sqrt(cloth::dot(diff, diff));
        n = cloth::mul(inv, diff);
        if (cloth::dot(n, fn) < R(0)) n = V{-n.x, -n.y, -n.z};
    }
    const R depth = cloth::dot(diff, n);
    if (!(depth > R(0))) return;
    const R bw[4] = {-bary.x, -bary.y, -bary.z, R(1)};
    const R b = bw[order];
    const R lambda = depth * c.kc;
    const R nn[3] = {n.x, n.y, n.z};
    const R s1 = b * lambda, s2 = b * b * c.kc;
    f[0] += s1 * nn[0]; f[1] += s1 * nn[1]; f[2] += s1 * nn[2];
    H[0] += s2 * nn[0] * nn[0]; H[1] += s2 * nn[0] * nn[1]; H[2] += s2 * nn[0] * nn[2];
    H[3] += s2 * nn[1] * nn[1]; H[4] += s2 * nn[1] * nn[2]; H[5] += s2 * nn[2] * nn[2];
    // relative tangential displacement over the substep: dx_p - sum_k bary_k dx_k
    R dx[3];
    ST::diff(up, P.xprev[sp], dx);
    const R bk[3] = {bary.x, bary.y, bary.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        R dk[3];
        ST::diff(uf[k], P.xprev[fs[k]], dk);
        dx[0] -= bk[k] * dk[0];
        dx[1] -= bk[k] * dk[1];
        dx[2] -= bk[k] * dk[2];
    }
    V t0 = cloth::sub(q[1], q[0]);
    const R l0 = sqrt(cloth::dot(t0, t0));
    t0 = V{t0.x / l0, t0.y / l0, t0.z / l0};
    V t1 = cloth::cross(t0, n);
    const R l1 = sqrt(cloth::dot(t1, t1));
    t1 = V{t1.x / l1, t1.y / l1, t1.z / l1};
    const R ta[3] = {t0.x, t0.y, t0.z}, tb[3] = {t1.x, t1.y, t1.z};
    const R u0 = ta[0] * dx[0] + ta[1] * dx[1] + ta[2] * dx[2];
    const R u1 = tb[0] * dx[0] + tb[1] * dx[1] + tb[2] * dx[2];
    const double2 fp = P.mesh_fric[P.slot_mesh[sp]], ff = P.mesh_fric[fo.w];
    const R mu = (R(fp.x) + R(ff.x)) * R(0.5);
    const R epsU = (R(fp.y) + R(ff.y)) * R(0.5) * c.dt;
    cloth::friction<R>(mu, lambda, ta, tb, u0, u1, epsU, b, f, H);
}

// Flags of a solve launch: friction on, and which half of the contact snapshots this iteration
// writes (it reads the other one).
enum { kSolveFriction = 1, kSolveParity = 2 };

// accumulateCollisionForceAndHessian (VBDPhysicsCompute.cu:1731-1773) of a vertex with contact
// records (info != 0): its own contact and its relations, at most five terms, one per lane of
// its group where the group is wide enough, summed into con (force 3, Hessian 6), which the
// solve adds between inertia and boundary. The vertices of the running color [beg, end) enter
// as they were before this launch (their snapshots: a contact partner can share the vertex's
// color and be updated by this very launch), all others as they are, which is the reference's
// Jacobi-within-color update (positionsNew, VBDPhysicsCompute.cu:803-908). Evaluated by a
// kernel of its own before each color, one thread per vertex, the terms of a vertex ran one
// after another and every color paid a second launch: 14 us per color on four small bodies in
// contact, 7.5 us with the terms here. Every lane of the warp calls it.
template <int L, typename ST, typename R>
__device__ __forceinline__ void contact_sums(const Ptrs<ST, R>& P, const Consts<R>& c, int v, int info, int sub, int beg,
                                          int end, int flags, R* con) {
    using U = typename ST::U;
    const U* before = P.snap + ((flags & kSolveParity) ? 0 : size_t(P.nslots));
    const auto state = [&](int s) { return s >= beg && s < end ? before[s] : P.u[s]; };
    for (int j = sub; j < 5; j += L) {
        if (j == 0) {
            if (info & 8) contact_term<ST, R>(P, c, state, v, 3, con, con + 3);
        } else if (j - 1 < (info & 7)) {
            const int e = P.col_rel[4 * v + j - 1];
            contact_term<ST, R>(P, c, state, e >> 2, e & 3, con, con + 3);
        }
    }
#pragma unroll
    for (int off = 16; off >= 32 / L; off >>= 1)
#pragma unroll
        for (int k = 0; k < 9; ++k) con[k] += __shfl_xor_sync(0xffffffffu, con[k], off);
}

// The same as a call: in the narrow groups of large colors few warps take it, and the solve of
// the others keeps its registers.
template <int L, typename ST, typename R>
__device__ __noinline__ void contact_sums_call(const Ptrs<ST, R>& P, const Consts<R>& c, int v, int info, int sub,
                                               int beg, int end, int flags, R* con) {
    contact_sums<L, ST, R>(P, c, v, info, sub, beg, end, flags, con);
}

// The snapshots of the vertices with contact records that the first solve of each color after
// a detection reads: the current states, into half `half`.
template <typename ST>
__global__ void k_contact_snapshot(const typename ST::U* u, typename ST::U* snap, int32_t nslots, int half,
                                   const int32_t* list, const int32_t* nlist) {
    const int n = *nlist;
    for (int i = int(blockIdx.x * blockDim.x + threadIdx.x); i < n; i += int(gridDim.x * blockDim.x)) {
        const int v = list[i];
        snap[size_t(half) * nslots + v] = u[v];
    }
}

// The vertex tail's own inputs into L1 while the incidence loop runs: they do not change during
// a sweep, and loaded only in the tail their latency would follow the lane reduction on the
// critical path. Wide groups (few vertices, bound by that path) prefetch what only the vertices
// at a wall read, too; the others save its 48 bytes per vertex.
template <int L, typename ST, typename R>
__device__ __forceinline__ void prefetch_tail(const Ptrs<ST, R>& P, int v) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(P.y + v));
    if constexpr (L >= 16) {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(P.xprev + v));
        if (P.rest_fh) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.rest_fh + v));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.rest_fl + v));
        }
    }
}

// The mesh frame's offset of a vertex, rounded to FP32 (zero without frames).
template <typename ST, typename R>
__device__ __forceinline__ float3 frame_offset(const Ptrs<ST, R>& P, int v) {
    if (!P.frame_F) return make_float3(0.f, 0.f, 0.f);
    const double4 f = P.frame_F[P.slot_mesh[v]];
    return make_float3(float(f.x), float(f.y), float(f.z));
}

// Whether the vertex can touch the world box: false only where an FP32 estimate of its
// position is inside by more than the estimate can be off, so that the exact test (which
// reads the start-of-substep state and, in a mesh frame, X + F as a float pair: 48 bytes
// more per vertex) runs for the few vertices at the walls. The estimate adds three floats
// (and rounds the frame offset): its error is below 2^-21 of the sum of their magnitudes.
// A position that is not finite counts as near.
template <typename ST, typename R>
__device__ __forceinline__ bool near_box(const Consts<R>& c, const typename ST::U& uo, const float4& Xo,
                                         const float3& Fo) {
    const float4 u = ST::head(uo);
    const float X[3] = {Xo.x, Xo.y, Xo.z}, F[3] = {Fo.x, Fo.y, Fo.z}, U3[3] = {u.x, u.y, u.z};
    bool inside = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float x = (X[d] + F[d]) + U3[d];
        const float m = 4.8e-7f * ((fabsf(X[d]) + fabsf(F[d])) + (fabsf(U3[d]) + fabsf(x)));
        inside = inside && x - m > c.lo_f[d] + 2.4e-7f * fabsf(c.lo_f[d]) && x + m < c.hi_f[d] - 2.4e-7f * fabsf(c.hi_f[d]);
    }
    return !inside;
}

// Bulk prefetch into L2 (no shared memory, no completion to wait for): addr and bytes
// 16-byte aligned.
__device__ __forceinline__ void bulk_prefetch_l2(const void* addr, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(addr), "r"(bytes) : "memory");
}

// The record rows of the vertices [v0, v1): whole slices, from the slice of v0 to the end of
// the longest list that the slice of v1 - 1 can hold (max_nbr, max_inc per vertex of the
// color; the arrays are padded by as much).
struct RecTile {
    int n0, n1, i0, i1;
};
template <typename ST, typename R>
__device__ __forceinline__ RecTile rec_tile(const Ptrs<ST, R>& P, int v0, int v1, int max_nbr, int max_inc) {
    const int4 r0 = P.vrec[v0], r1 = P.vrec[v1 - 1];
    return RecTile{r0.x, r1.x + max_nbr, r0.y, r1.y + max_inc};
}

// What the warp `pf` warps on (one resident wave later) will load first, into L2: its records
// (from their vrec, which this warp loaded ahead), rest positions and tail inputs, and the
// vrec of the warp as far on again. Every link of a vertex's load chain (vrec, records,
// neighbours) is then an L2 round trip instead of a DRAM one.
template <int L, typename ST, typename R>
__device__ __forceinline__ void prefetch_vertices(const Ptrs<ST, R>& P, int v, int end, int pf, int4 ahead) {
    const int va = v + pf * Lanes<L>::kW;  // this lane's vertex in that warp
    if (va >= end) return;
    if (Lanes<L>::vertex() % kSlice == 0 && Lanes<L>::sub() == 0) {
        // one lane per slice: the longest list is at most a little longer than its first vertex's
        bulk_prefetch_l2(P.nbr + record_index(ahead.x, 0), uint32_t(max(nbrs_of(ahead.z), 1)) * uint32_t(kSlice * sizeof(NbrRec<R>)));
        bulk_prefetch_l2(P.inc + record_index(ahead.y, 0), uint32_t(max(ahead.w, 1)) * uint32_t(kSlice * sizeof(IncRec<R>)));
    }
    if (Lanes<L>::sub() == L - 1) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P.rest + va));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P.y + va));
        if (va + pf * Lanes<L>::kW < end) asm volatile("prefetch.global.L2 [%0];" ::"l"(P.vrec + va + pf * Lanes<L>::kW));
    }
}

template <int L, bool PROBE, bool CONTACT, typename ST, typename R>
__device__ __forceinline__ void finish_vertex(const Ptrs<ST, R>& P, const Consts<R>& c, int v, bool valid, int sub,
                                              const typename ST::U& uo, const float4& Xo, const float3& Fo,
                                              const MeshMat<R>& mat, Acc<R>& acc, int info, int beg, int end, int flags,
                                              double* probe_out);

// Minimum resident blocks of 256 threads: caps FP32-compute kernels at 64
// registers (32 warps per SM, no spills); the FP64 kernel keeps its registers, as do
// the wide groups, whose colors are too small to fill the GPU.
template <int L, typename R>
struct SolveOcc {
    static constexpr int kMinBlocks = sizeof(R) == 8 || L >= 16 ? 2 : 4;
};

// [beg, end): the color or the part of it that this launch solves; color: all of it.
// DEEP (variant 4): asynchronous one-ring copies (narrow groups). MULTI: vertices of several
// segments among them. pf > 0: prefetch distance in warps.
// max_nbr: the longest neighbour list of the launch, the staging entries per vertex.
template <int L, typename ST, typename R, bool PROBE, bool DEEP, bool MULTI, bool CONTACT>
__global__ void __launch_bounds__(256, SolveOcc<L, R>::kMinBlocks)
    k_solve(Ptrs<ST, R> P, Consts<R> c, int beg, int end, int2 color, int flags, double* probe_out, int pf, int max_nbr) {
    using U = typename ST::U;
    constexpr bool kAsync = DEEP && L < 16;
    constexpr int NB = NbrBatch<L, kAsync>::kN;
    constexpr int RR = kAsync ? kRecKept : kRecStream;  // neighbour records are read twice
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_launch_dependents();
    const int sub = Lanes<L>::sub();
    const int v = beg + int((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * Lanes<L>::kW + Lanes<L>::vertex();
    const bool valid = v < end;
    Acc<R> acc = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    U uo{};
    MeshMat<R> mat{};
    float4 Xo = make_float4(0.f, 0.f, 0.f, 0.f);
    // prologue on static data (records, rest position, materials): overlaps the previous
    // color's tail when launched as a programmatic dependent
    int4 seg = make_int4(0, 0, 0, 0);
    if (valid) {
        seg = P.vrec[v];
        Xo = __ldg(P.rest + v);
        mat = P.mats[P.slot_mesh[v]];
    }
    SegRecs<R, NB> rec;
    const Stage<32 / L, ST, R> st = warp_stage<L, ST, R>(smem, max_nbr);
    if (valid && sub == 0 && !PROBE) prefetch_tail<L>(P, v);
    float3 Fo = make_float3(0.f, 0.f, 0.f);
    if constexpr (L >= 16)
        if (valid && sub == 0) Fo = frame_offset(P, v);
    preload<L, RR>(rec, P.nbr, P.inc, seg, sub);
    constexpr bool kPrefetch = sizeof(R) == 4 && !PROBE && !DEEP && L < 16;
    int4 ahead = make_int4(0, 0, 0, 0);
    if constexpr (kPrefetch)
        if (pf > 0 && v + pf * Lanes<L>::kW < end && sub == 0) ahead = P.vrec[v + pf * Lanes<L>::kW];
    pdl_wait();
    int info = 0;
    if (valid) {
        uo = P.u[v];
        if constexpr (CONTACT) info = P.col_info[v];
    }
    const U uon = ST::nb(uo);
    const FetchGlobal<ST, kStatePlain> fetch{P.u, P.rest};
    accumulate_segment<L, RR, kAsync, ST>(rec, sub, st, fetch, uon, Xo, mat.mu, mat.lmbd, acc);
    if constexpr (kPrefetch)
        if (pf > 0) prefetch_vertices<L>(P, v, end, pf, ahead);
    if constexpr (MULTI)
        if (valid)
            accumulate_more<L, RR, kAsync, ST>(rec, P, P.nbr, P.inc, P.vmore[v], sub, st, fetch, uon, Xo, mat.mu, mat.lmbd, acc);
    reduce_group<L, R>(acc);
    if constexpr (L < 16)
        if (valid && sub == 0) Fo = frame_offset(P, v);
    finish_vertex<L, PROBE, CONTACT>(P, c, v, valid, sub, uo, Xo, Fo, mat, acc, info, color.x, color.y, flags, probe_out);
}

// ---- per-vertex tail (lane 0 of a vertex group): damping, inertia, ground and
// friction, 3x3 solve, update ------------------------------------------------------
// con: the vertex's contact sums (null: none). The new state goes to P.u[v], or to *unew when
// given; returns whether the vertex moved.
template <typename ST, typename R, bool PROBE>
__device__ __forceinline__ bool vertex_tail(const Ptrs<ST, R>& P, const Consts<R>& c, int v, const typename ST::U& uo,
                                            const float4& Xo, const float3& Fo, const MeshMat<R>& mat,
                                            const Acc<R>& acc, int friction, double* probe_out,
                                            const R* con, typename ST::U* unew) {
    using U = typename ST::U;
    using Sc = typename ST::Sc;
    R f[3] = {acc.f0, acc.f1, acc.f2};
    R H[6] = {acc.h00 + acc.S, acc.h01, acc.h02, acc.h11 + acc.S, acc.h12, acc.h22 + acc.S};
    if (mat.kh > R(0) || mat.kd > R(0)) {
        R dx[3];
        ST::diff(uo, P.xprev[v], dx);
        // damping Hessian (k_h H_lambda + k_d S I) / dt (VBD_NeoHookean.cpp:562-574)
        R D[6] = {mat.kh * acc.h00 + mat.kd * acc.S, mat.kh * acc.h01, mat.kh * acc.h02,
                  mat.kh * acc.h11 + mat.kd * acc.S, mat.kh * acc.h12, mat.kh * acc.h22 + mat.kd * acc.S};
#pragma unroll
        for (int i = 0; i < 6; ++i) D[i] *= c.inv_dt;
        f[0] -= D[0] * dx[0] + D[1] * dx[1] + D[2] * dx[2];
        f[1] -= D[1] * dx[0] + D[3] * dx[1] + D[4] * dx[2];
        f[2] -= D[2] * dx[0] + D[4] * dx[1] + D[5] * dx[2];
#pragma unroll
        for (int i = 0; i < 6; ++i) H[i] += D[i];
    }
    // inertia (VBD_GeneralCompute.h:68-85)
    {
        const U yv = P.y[v];
        R dy[3];
        ST::diff(yv, uo, dy);
        R w = R(ST::mass(uo)) * c.dt2inv;
        f[0] += w * dy[0];
        f[1] += w * dy[1];
        f[2] += w * dy[2];
        H[0] += w; H[3] += w; H[5] += w;
    }
    // tet-mesh contact (between inertia and boundary, VBDPhysicsCompute.cu:893-895)
    if (con) {
        f[0] += con[0]; f[1] += con[1]; f[2] += con[2];
#pragma unroll
        for (int i = 0; i < 6; ++i) H[i] += con[3 + i];
    }
    // plane ground / world box with friction on each violated axis (VBDPhysics.cpp:2858-2953)
    if (c.plane && near_box<ST, R>(c, uo, Xo, Fo)) {
        // x = X + u, or (X + F) + u in a mesh frame F, X + F held as a float pair per slot
        const bool framed = P.rest_fh != nullptr;
        const float4 X = framed ? P.rest_fh[v] : Xo;
        const float4 Xl = framed ? P.rest_fl[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float Xc[3] = {X.x, X.y, X.z}, Xlc[3] = {Xl.x, Xl.y, Xl.z};
        R dx[3];
        ST::diff(uo, P.xprev[v], dx);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            // below = lo - x, above = x - hi
            R below = framed ? ST::template sub_plane<R>(pick<Sc>(c.lo[d], c.lo_f[d]), Xc[d], Xlc[d], uo, d)
                             : ST::template sub_from<R>(pick<Sc>(c.lo[d], c.lo_f[d]), Xc[d], uo, d);
            R depth;
            if (below > R(0)) {
                depth = below;
                f[d] += depth * c.kb;
            } else {
                R above = framed ? -ST::template sub_plane<R>(pick<Sc>(c.hi[d], c.hi_f[d]), Xc[d], Xlc[d], uo, d)
                                 : -ST::template sub_from<R>(pick<Sc>(c.hi[d], c.hi_f[d]), Xc[d], uo, d);
                if (!(above > R(0))) continue;
                depth = above;
                f[d] -= depth * c.kb;
            }
            H[d == 0 ? 0 : (d == 1 ? 3 : 5)] += c.kb;
            if (friction) axis_friction<R>(d, dx, c.fr_mu, depth * c.kb, c.fr_epsU, f, H);
        }
    }
    if (PROBE) {
        probe_out[0] = f[0]; probe_out[1] = f[1]; probe_out[2] = f[2];
        probe_out[3] = H[0]; probe_out[4] = H[1]; probe_out[5] = H[2];
        probe_out[6] = H[1]; probe_out[7] = H[3]; probe_out[8] = H[4];
        probe_out[9] = H[2]; probe_out[10] = H[4]; probe_out[11] = H[5];
        return false;
    }
    // CMP_EPSILON2 gate (Types/Types.h:20-21; VBDPhysics.cpp:2432); a non-finite force (a
    // NaN or Inf position among the vertex's neighbours) is counted, as the reference's
    // CPU path stops on a NaN descent direction (VBDPhysics.cpp:2460-2464)
    const R fn2 = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
    if (!(fn2 > R(1e-5f * 1e-5f))) {
        if (!(fn2 <= R(1e-5f * 1e-5f))) atomicAdd(&P.counters[CNT_NONFINITE], 1ull);
        return false;
    }
    R d3[3];
    R step = c.step;
    if (!solve3<R>(H, f, d3, P.counters)) {
        // VBDPhysics.cpp:2452-2458: gradient step along the force
        atomicAdd(&P.counters[CNT_FAILED_SOLVES], 1ull);
        step = c.step_gd;
        d3[0] = f[0]; d3[1] = f[1]; d3[2] = f[2];
    }
    const Sc s0 = Sc(step * d3[0]), s1 = Sc(step * d3[1]), s2 = Sc(step * d3[2]);
    if (!(isfinite(s0) && isfinite(s1) && isfinite(s2))) {
        atomicAdd(&P.counters[CNT_NONFINITE], 1ull);
        return false;
    }
    if (unew) *unew = ST::add(uo, s0, s1, s2);
    else P.u[v] = ST::add(uo, s0, s1, s2);
    return true;
}

// The end of a color launch for one vertex group: contact sums (CONTACT: scenes with contact
// detection), the tail on sub-lane 0 and the vertex's contact snapshot for the next iteration.
// Every lane of the warp calls it, with the reduced sums.
template <int L, bool PROBE, bool CONTACT, typename ST, typename R>
__device__ __forceinline__ void finish_vertex(const Ptrs<ST, R>& P, const Consts<R>& c, int v, bool valid, int sub,
                                              const typename ST::U& uo, const float4& Xo, const float3& Fo,
                                              const MeshMat<R>& mat, Acc<R>& acc, int info, int beg, int end, int flags,
                                              double* probe_out) {
    if constexpr (CONTACT) {
        R con[9] = {R(0), R(0), R(0), R(0), R(0), R(0), R(0), R(0), R(0)};
        const bool some = __any_sync(0xffffffffu, info != 0);
        if (some) {
            if constexpr (L >= 16) contact_sums<L, ST, R>(P, c, v, info, sub, beg, end, flags, con);
            else contact_sums_call<L, ST, R>(P, c, v, info, sub, beg, end, flags, con);
        }
        if (!valid || sub != 0) return;
        finish_acc(acc, mat.mu, mat.lmbd);
        typename ST::U un = uo;
        const bool moved = vertex_tail<ST, R, PROBE>(P, c, v, uo, Xo, Fo, mat, acc, flags & kSolveFriction, probe_out,
                                                     info ? con : nullptr, &un);
        if (PROBE) return;
        if (moved) P.u[v] = un;
        if (info) P.snap[((flags & kSolveParity) ? size_t(P.nslots) : 0) + v] = moved ? un : uo;
    } else {
        if (!valid || sub != 0) return;
        finish_acc(acc, mat.mu, mat.lmbd);
        vertex_tail<ST, R, PROBE>(P, c, v, uo, Xo, Fo, mat, acc, flags & kSolveFriction, probe_out, nullptr);
    }
}

// ---------------------------------------------------------------------------
// TMA-staged solve (FP32 compute). Each block owns vpb = blockDim / L
// consecutive vertices of the color; their neighbour and their incidence
// records are one contiguous range each. Thread 0 stages the ranges into shared
// memory with two bulk copies (cp.async.bulk) completing on an mbarrier, issued
// before the programmatic-dependency wait: a block's whole record range is in
// flight at once, overlapping the previous color's tail, at no register cost.
// Neighbour positions are gathered as in k_solve. tile_nbr and tile_inc bound the
// records of any block of this launch (the host sizes the dynamic shared memory
// from them). Vertices of one segment only.
// ---------------------------------------------------------------------------
constexpr int kMbarSpinLimit = 1 << 20;
// Polls of the final drain wait of a block whose first wait ran out, each after a 1 us
// sleep: about two seconds in all, far beyond the time any issued copy takes to land.
constexpr int kDrainPolls = 1 << 21;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait on an mbarrier phase: at most `limit` polls; false if the phase did not
// complete within them.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
    for (int i = 0; i < limit; ++i)
        if (mbar_test(bar, parity)) return true;
    return false;
}

// The wait of a block that gave up: the phase completes when every byte its copies
// declared (expect_tx = exactly the bytes issued) has landed, so this waits, bounded and
// with sleeps, until no copy of the block is left writing into its shared memory.
__device__ __forceinline__ bool mbar_drain(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kDrainPolls; ++i) {
        if (mbar_test(bar, parity)) return true;
        __nanosleep(1000);
    }
    return false;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// The copies of a record range (whole slices: 16-byte aligned) on mbarrier `bar` by one thread.
template <typename ST>
__device__ __forceinline__ void issue_tile(const Ptrs<ST, float>& P, const RecTile& t, NbrRec<float>* s_nbr,
                                           IncRec<float>* s_inc, uint32_t bar) {
    const uint32_t nb = uint32_t(t.n1 - t.n0) * uint32_t(8 * kSlice), ib = uint32_t(t.i1 - t.i0) * uint32_t(8 * kSlice);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(nb + ib) : "memory");
    if (nb) bulk_g2s(s_nbr, P.nbr + record_index(t.n0, 0), nb, bar);
    if (ib) bulk_g2s(s_inc, P.inc + record_index(t.i0, 0), ib, bar);
}

template <int L, bool CONTACT, typename ST>
__global__ void __launch_bounds__(256, 4)
    k_solve_tma(Ptrs<ST, float> P, Consts<float> c, int beg, int end, int2 color, int flags, int max_nbr, int max_inc,
                int tile_nbr, int tile_inc) {
    using U = typename ST::U;
    constexpr int NB = NbrBatch<L, false>::kN;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t bar = smem_u32(smem);
    NbrRec<float>* s_nbr = reinterpret_cast<NbrRec<float>*>(smem + 16);
    IncRec<float>* s_inc = reinterpret_cast<IncRec<float>*>(smem + 16 + 8 * size_t(tile_nbr));
    unsigned char* s_stage = smem + 16 + 8 * (size_t(tile_nbr) + size_t(tile_inc));
    pdl_launch_dependents();
    const int vpb = blockDim.x / L;
    const int v0 = beg + blockIdx.x * vpb;
    const int v1 = min(end, v0 + vpb);
    const RecTile tile = rec_tile(P, v0, v1, max_nbr, max_inc);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) issue_tile(P, tile, s_nbr, s_inc, bar);
    const int sub = Lanes<L>::sub();
    const int v = v0 + int(threadIdx.x >> 5) * Lanes<L>::kW + Lanes<L>::vertex();
    const bool valid = v < v1;
    MeshMat<float> mat{};
    float4 Xo = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 seg = make_int4(0, 0, 0, 0);
    if (valid) {
        seg = P.vrec[v];
        seg.x -= tile.n0;
        seg.y -= tile.i0;
        Xo = __ldg(P.rest + v);
        mat = P.mats[P.slot_mesh[v]];
        if (sub == 0) prefetch_tail<L>(P, v);
    }
    const Stage<32 / L, ST, float> st = warp_stage<L, ST, float>(s_stage, max_nbr);
    pdl_wait();
    U uo{};
    int info = 0;
    if (valid) {
        uo = P.u[v];
        if constexpr (CONTACT) info = P.col_info[v];
    }
    const U uon = ST::nb(uo);
    // the block goes on only if every thread saw the records land within the limit
    const bool ok = __syncthreads_and(mbar_wait(bar, 0, c.spin_limit)) != 0;
    if (!ok) {
        // the records did not land within the limit: the block skips its vertices (none
        // moves) and records it, which the host reports as a device-timeout status; thread
        // 0 then drains the copies so that none is left writing into this block's shared
        // memory after it exits
        if (threadIdx.x == 0) {
            atomicAdd(&P.counters[CNT_TIMEOUT], 1ull);
            if (!mbar_drain(bar, 0)) atomicAdd(&P.counters[CNT_DRAIN], 1ull);
        }
        return;
    }
    Acc<float> acc = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    SegRecs<float, NB> rec;
    preload<L, kRecShared>(rec, s_nbr, s_inc, seg, sub);
    accumulate_segment<L, kRecShared, false, ST>(rec, sub, st, FetchGlobal<ST, kStatePlain>{P.u, P.rest}, uon, Xo, mat.mu, mat.lmbd, acc);
    reduce_group<L, float>(acc);
    const float3 Fo = valid && sub == 0 ? frame_offset(P, v) : make_float3(0.f, 0.f, 0.f);
    finish_vertex<L, false, CONTACT>(P, c, v, valid, sub, uo, Xo, Fo, mat, acc, info, color.x, color.y, flags, nullptr);
}

// ---------------------------------------------------------------------------
// Double-buffered TMA pipeline (FP32 compute). A persistent grid walks the color's tiles
// of vpt = blockDim / L consecutive vertices (tile t of block b: t = b, b + grid, ...). The
// records of a tile are one contiguous range per array; thread 0 stages the next tile's
// ranges into the other shared-memory buffer (two cp.async.bulk copies on that buffer's
// mbarrier) while the block computes the current one, so the record stream of the whole
// color is in flight ahead of the warps without occupying their registers. Bounded waits as
// in k_solve_tma: a block whose wait runs out counts a timeout, drains every copy it issued
// and returns. tile_nbr and tile_inc bound the records of any tile (the host sizes the buffers
// from them). Vertices of one segment only.
// ---------------------------------------------------------------------------
template <int L, bool CONTACT, typename ST>
__global__ void __launch_bounds__(256)
    k_solve_pipe(Ptrs<ST, float> P, Consts<float> c, int beg, int end, int2 color, int flags, int max_nbr, int max_inc,
                 int tile_nbr, int tile_inc) {
    using U = typename ST::U;
    constexpr int NB = NbrBatch<L, false>::kN;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t bar0 = smem_u32(smem);
    const size_t buf_bytes = 8 * (size_t(tile_nbr) + size_t(tile_inc));
    auto s_nbr = [&](int b) { return reinterpret_cast<NbrRec<float>*>(smem + 16 + size_t(b) * buf_bytes); };
    auto s_inc = [&](int b) { return reinterpret_cast<IncRec<float>*>(smem + 16 + size_t(b) * buf_bytes + 8 * size_t(tile_nbr)); };
    unsigned char* s_stage = smem + 16 + 2 * buf_bytes;
    const int vpt = int(blockDim.x) / L;
    const int ntiles = (end - beg + vpt - 1) / vpt;
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto tile_of = [&](int t) { return rec_tile(P, beg + t * vpt, min(end, beg + (t + 1) * vpt), max_nbr, max_inc); };
    // thread 0: the records of tile t into buffer b (records are static: no ordering with
    // the previous color needed)
    auto issue = [&](int t, int b) { issue_tile(P, tile_of(t), s_nbr(b), s_inc(b), bar0 + 8u * uint32_t(b)); };
    if (threadIdx.x == 0 && int(blockIdx.x) < ntiles) issue(int(blockIdx.x), 0);
    pdl_wait();
    const int sub = Lanes<L>::sub();
    const Stage<32 / L, ST, float> st = warp_stage<L, ST, float>(s_stage, max_nbr);
    int k = 0;
    for (int t = int(blockIdx.x); t < ntiles; t += int(gridDim.x), ++k) {
        const int b = k & 1;
        const uint32_t parity = uint32_t(k >> 1) & 1u;
        const int tn = t + int(gridDim.x);
        // the next tile into the other buffer (released by the barrier that ended the last tile)
        if (threadIdx.x == 0 && tn < ntiles) issue(tn, b ^ 1);
        const RecTile tile = tile_of(t);
        const int v0 = beg + t * vpt, v1 = min(end, v0 + vpt);
        const int v = v0 + int(threadIdx.x >> 5) * Lanes<L>::kW + Lanes<L>::vertex();
        const bool valid = v < v1;
        MeshMat<float> mat{};
        float4 Xo = make_float4(0.f, 0.f, 0.f, 0.f);
        int4 seg = make_int4(0, 0, 0, 0);
        U uo{};
        int info = 0;
        if (valid) {
            seg = P.vrec[v];
            seg.x -= tile.n0;
            seg.y -= tile.i0;
            Xo = __ldg(P.rest + v);
            mat = P.mats[P.slot_mesh[v]];
            if (sub == 0) prefetch_tail<L>(P, v);
            uo = P.u[v];
            if constexpr (CONTACT) info = P.col_info[v];
        }
        const U uon = ST::nb(uo);
        const bool ok = __syncthreads_and(mbar_wait(bar0 + 8u * uint32_t(b), parity, c.spin_limit)) != 0;
        if (!ok) {
            // this tile's records did not land within the limit: skip the block's remaining
            // tiles (their vertices do not move), count it, and drain every copy issued (this
            // tile's and, if issued, the next one's) before the block exits
            if (threadIdx.x == 0) {
                atomicAdd(&P.counters[CNT_TIMEOUT], 1ull);
                bool drained = mbar_drain(bar0 + 8u * uint32_t(b), parity);
                if (tn < ntiles) drained = mbar_drain(bar0 + 8u * uint32_t(b ^ 1), uint32_t((k + 1) >> 1) & 1u) && drained;
                if (!drained) atomicAdd(&P.counters[CNT_DRAIN], 1ull);
            }
            return;
        }
        Acc<float> acc = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        SegRecs<float, NB> rec;
        preload<L, kRecShared>(rec, s_nbr(b), s_inc(b), seg, sub);
        accumulate_segment<L, kRecShared, false, ST>(rec, sub, st, FetchGlobal<ST, kStatePlain>{P.u, P.rest}, uon, Xo, mat.mu, mat.lmbd, acc);
        reduce_group<L, float>(acc);
        const float3 Fo = valid && sub == 0 ? frame_offset(P, v) : make_float3(0.f, 0.f, 0.f);
        finish_vertex<L, false, CONTACT>(P, c, v, valid, sub, uo, Xo, Fo, mat, acc, info, color.x, color.y, flags, nullptr);
        __syncthreads();  // every read of buffer b done before the next iteration refills it
    }
}

// ---------------------------------------------------------------------------
// Persistent scene-major sweep: every iteration of a substep in one launch. Each block
// takes whole scenes (meshes) from a work counter, in the order `scene_order` (largest
// first), and runs all `iterations` of that scene: per iteration its colors in sequence,
// each color's vertices over the block's vertex groups, a block barrier between colors.
// Meshes do not interact (no contact records in this mode), so per mesh the sequence
// of color updates, and every vertex's arithmetic, equal the merged color-major sweep's;
// a scene's records and states stay in the block's L1 / the L2 across its iterations,
// and no launch or device-wide barrier separates colors. Layout: the slots of a mesh
// are contiguous and color-major within it; colors[scene_ofs[m] .. scene_ofs[m + 1])
// are mesh m's color slot ranges in sweep order. MAXB bounds the block size (and so the
// registers a thread may use: 256 leaves the compiler all it needs, 1024 caps it at 64).
// ---------------------------------------------------------------------------

// One vertex group's solve inside a persistent sweep, its state and its neighbours' read with
// Fetch. Every lane of the warp calls it; v is the group's vertex when valid. cap: staged
// neighbours per vertex.
template <int L, bool MULTI, typename ST, typename R, typename Fetch>
__device__ __forceinline__ void solve_in_sweep(const Ptrs<ST, R>& P, const Consts<R>& c, int v, bool valid, int sub,
                                               unsigned char* smem, int cap, int warp_bytes, const Fetch& fetch,
                                               const typename ST::U& uo, int friction) {
    using U = typename ST::U;
    constexpr bool kAsync = L < 16;
    constexpr int NB = NbrBatch<L, kAsync>::kN;
    Acc<R> acc = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    MeshMat<R> mat{};
    float4 Xo = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 seg = make_int4(0, 0, 0, 0);
    if (valid) {
        seg = __ldg(P.vrec + v);
        Xo = __ldg(P.rest + v);
        mat = P.mats[P.slot_mesh[v]];
    }
    SegRecs<R, NB> rec;
    const Stage<32 / L, ST, R> st = warp_stage<L, ST, R>(smem, cap, size_t(warp_bytes));
    preload<L, kRecKept>(rec, P.nbr, P.inc, seg, sub);
    if (valid && sub == 0) prefetch_tail<L>(P, v);
    const U uon = ST::nb(uo);
    accumulate_segment<L, kRecKept, kAsync, ST>(rec, sub, st, fetch, uon, Xo, mat.mu, mat.lmbd, acc);
    if constexpr (MULTI)
        if (valid)
            accumulate_more<L, kRecKept, kAsync, ST>(rec, P, P.nbr, P.inc, P.vmore[v], sub, st, fetch, uon, Xo, mat.mu, mat.lmbd, acc);
    __syncwarp();  // the staging area is written again by the warp's next vertices
    reduce_group<L, R>(acc);
    if (valid && sub == 0) {
        finish_acc(acc, mat.mu, mat.lmbd);
        vertex_tail<ST, R, false>(P, c, v, uo, Xo, frame_offset(P, v), mat, acc, friction, nullptr, nullptr);
    }
}

// The staging areas of a persistent sweep: entries per vertex of the short lists (L lanes per
// vertex) and of the long ones (a warp per vertex), and the bytes per warp that hold either.
struct SweepStage {
    int32_t cap, cap_long, warp_bytes;
};

// The vertices [beg, end) of one color in turn over `warps` warps, this one being number `w`.
template <int L, bool MULTI, bool GRID, typename ST, typename R, typename Fetch>
__device__ __forceinline__ void sweep_range(const Ptrs<ST, R>& P, const Consts<R>& c, int beg, int end, int w, int warps,
                                            unsigned char* smem, int cap, int warp_bytes, const Fetch& fetch,
                                            int friction) {
    const int g = w * Lanes<L>::kW + Lanes<L>::vertex();
    for (int base = beg; base < end; base += warps * Lanes<L>::kW) {
        const int v = base + g;
        const bool valid = v < end;
        typename ST::U uo{};
        if (valid) uo = GRID ? ST::ldcg_own(P.u, v) : ST::ld_own(P.u, v);
        solve_in_sweep<L, MULTI, ST, R>(P, c, v, valid, Lanes<L>::sub(), smem, cap, warp_bytes, fetch, uo, friction);
    }
}

// colors: (first slot, first slot of the vertices with long lists, end). LONG: there are such.
template <int L, bool LONG, typename ST, typename R, int MAXB>
__global__ void __launch_bounds__(MAXB) k_sweep_scenes(Ptrs<ST, R> P, Consts<R> c, const int4* colors,
                                                       const int32_t* scene_ofs, const int32_t* scene_order,
                                                       int32_t nscenes, int32_t iterations, int32_t friction_start,
                                                       int32_t* work, SweepStage S) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_scene;
    const int w = int(threadIdx.x >> 5), warps = int(blockDim.x >> 5);
    const FetchGlobal<ST, kStatePlain> fetch{P.u, P.rest};
    for (;;) {
        if (threadIdx.x == 0) s_scene = atomicAdd(work, 1);
        __syncthreads();
        const int k = s_scene;
        __syncthreads();  // every thread has read s_scene before it is written again
        if (k >= nscenes) return;
        const int sc = scene_order[k];
        const int c0 = scene_ofs[sc], c1 = scene_ofs[sc + 1];
        for (int it = 0; it < iterations; ++it) {
            const int friction = it >= friction_start ? 1 : 0;
            for (int ci = c0; ci < c1; ++ci) {
                const int4 rg = colors[ci];
                sweep_range<L, false, false, ST, R>(P, c, rg.x, rg.y, w, warps, smem, S.cap, S.warp_bytes, fetch, friction);
                if constexpr (LONG)
                    sweep_range<32, true, false, ST, R>(P, c, rg.y, rg.z, w, warps, smem, S.cap_long, S.warp_bytes, fetch,
                                                        friction);
                __syncthreads();  // this color's updates before the next color reads them
            }
        }
    }
}

// Mesh frames, at the start of every substep: per mesh, the FP32 head of its reference
// vertex's state becomes the shift that k_initial_step takes out of every state of the mesh
// (exactly in the double-float modes; the FP32 mode rounds u - s, which is small where the
// mesh moves as a whole), and the frame offset F accumulates it in FP64. A mesh that falls
// or slides as a body then keeps states of the size of its deformation and of one substep's
// motion, and every FP32 difference and update of the solve rounds at that scale instead of
// at the scale of the distance travelled.
template <typename ST>
__global__ void k_frame_update(const typename ST::U* u, const int32_t* ref, double4* F, float4* shift,
                               int32_t nmesh) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmesh) return;
    const int r = ref[m];
    const float4 sh = r >= 0 ? ST::head(u[r]) : make_float4(0.f, 0.f, 0.f, 0.f);
    double4 f = F[m];
    f.x += double(sh.x);
    f.y += double(sh.y);
    f.z += double(sh.z);
    F[m] = f;
    shift[m] = sh;
}

// Initial step of a substep over all slots: VBD_BaseMaterial.h:201-259 and
// VBD_BaseMaterial.cpp:7-31 (initialization types 0..4). Displacements: every
// update is linear in x, so it reads as in positions.
template <typename ST, typename R>
__global__ void k_initial_step(Ptrs<ST, R> P, Consts<R> c) {
    using U = typename ST::U;
    using V = typename ST::V;
    using Sc = typename ST::Sc;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.nslots) return;
    const Sc dt = pick<Sc>(c.dt_d, c.dt_f);
    const int mesh = P.slot_mesh[s];
    U x = P.u[s];
    // mesh frames: the substep starts in the frame moved by this substep's shift (x, and the
    // start-of-substep state, inertia target and initial guess derived from it)
    if (P.frame_shift) {
        const float4 sh = P.frame_shift[mesh];
        x = ST::shift(x, sh.x, sh.y, sh.z);
        // X + F of this slot for the world-box test, as a float pair
        const float4 X = P.rest[s];
        const double4 F = P.frame_F[mesh];
        const double xf[3] = {double(X.x) + F.x, double(X.y) + F.y, double(X.z) + F.z};
        float4 h, l;
        h.x = float(xf[0]); l.x = float(xf[0] - double(h.x));
        h.y = float(xf[1]); l.y = float(xf[1] - double(h.y));
        h.z = float(xf[2]); l.z = float(xf[2] - double(h.z));
        h.w = 0.f; l.w = 0.f;
        P.rest_fh[s] = h;
        P.rest_fl[s] = l;
    }
    V v = P.vel[s];
    P.xprev[s] = x;
    const bool fixed = s >= P.nactive;
    const int init_type = P.mats[mesh].init_type;
    if (init_type == 2 || init_type == 4) P.vprev[s] = v;
    const V vp = v;
    if (c.assoc_grav) {
        v.x += dt * pick<Sc>(c.g[0], c.g_f[0]);
        v.y += dt * pick<Sc>(c.g[1], c.g_f[1]);
        v.z += dt * pick<Sc>(c.g[2], c.g_f[2]);
    }
    if (fixed) { v.x = 0; v.y = 0; v.z = 0; }
    const U yv = ST::add(x, dt * v.x, dt * v.y, dt * v.z);
    P.vel[s] = v;
    P.y[s] = yv;
    U xn;
    switch (init_type) {
        case 1: xn = x; break;
        case 2: xn = ST::add(x, dt * vp.x, dt * vp.y, dt * vp.z); break;
        case 3: xn = ST::add(x, Sc(0.5) * dt * v.x, Sc(0.5) * dt * v.y, Sc(0.5) * dt * v.z); break;
        case 4: {
            const Sc h = Sc(0.5) * dt * dt;
            xn = ST::add(x, dt * vp.x + h * pick<Sc>(c.g[0], c.g_f[0]), dt * vp.y + h * pick<Sc>(c.g[1], c.g_f[1]), dt * vp.z + h * pick<Sc>(c.g[2], c.g_f[2]));
            break;
        }
        default: xn = yv; break;
    }
    P.u[s] = xn;
}

// A state to time solves on: every solved vertex moved by up to a hundredth of the distance to
// its first neighbour (at rest no vertex has a force, and the solves end at the force test).
template <typename ST, typename R>
__global__ void k_perturb(Ptrs<ST, R> P) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.nactive) return;
    const int4 seg = P.vrec[s];
    if (nbrs_of(seg.z) == 0) return;
    const float4 a = P.rest[s], b = P.rest[P.nbr[record_index(seg.x, place_of(seg.z))].slot];
    const float d = sqrtf((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y) + (a.z - b.z) * (a.z - b.z));
    using Sc = typename ST::Sc;
    uint32_t h = uint32_t(s) * 2654435761u;
    Sc m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        h = (h ^ (h >> 15)) * 2246822519u + 374761393u;
        m[c] = Sc(0.01f * d) * (Sc(h >> 8) * Sc(1.0 / 8388608.0) - Sc(1));
    }
    P.u[s] = ST::add(P.u[s], m[0], m[1], m[2]);
}

// Deformers (VBD/VBDDeformer.h:45-172). Rotator: p = root + R(theta) rootP with
// theta = omega * t; Translator: p = orig + speed * t. t = time after this substep's
// advance, clamped to the end time. Per selected vertex, in FP64 (a few thousand
// boundary vertices per substep).
template <typename ST>
__global__ void k_deformers(typename ST::U* u, const float4* rest, DeformVerts D, const double* time, double dt) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= D.n) return;
    const DeformerDev d = D.defs[D.def[k]];
    double t = time[0] + dt;
    if (t >= d.end_time && d.end_time > 0) t = d.end_time;
    int s = D.slot[k];
    const float4 X = rest[s];
    const double* a = D.a + 3 * size_t(k);
    double p[3];
    if (d.type == 0) {
        const double* b = D.b + 3 * size_t(k);
        double th = t * d.omega, co = cos(th), si = sin(th), C = 1 - co;
        double ux = d.axis[0], uy = d.axis[1], uz = d.axis[2];
        double Rm[9] = {co + ux * ux * C, ux * uy * C - uz * si, ux * uz * C + uy * si,
                        uy * ux * C + uz * si, co + uy * uy * C, uy * uz * C - ux * si,
                        uz * ux * C - uy * si, uz * uy * C + ux * si, co + uz * uz * C};
        p[0] = a[0] + (Rm[0] * b[0] + Rm[1] * b[1] + Rm[2] * b[2]);
        p[1] = a[1] + (Rm[3] * b[0] + Rm[4] * b[1] + Rm[5] * b[2]);
        p[2] = a[2] + (Rm[6] * b[0] + Rm[7] * b[1] + Rm[8] * b[2]);
    } else {
        p[0] = d.speed[0] * t + a[0];
        p[1] = d.speed[1] * t + a[1];
        p[2] = d.speed[2] * t + a[2];
    }
    double du[3] = {p[0] - double(X.x), p[1] - double(X.y), p[2] - double(X.z)};
    u[s] = ST::from_d(du, ST::mass(u[s]));
}

// Velocity update with the CPU path's damping (VBDPhysics.cpp:2486-2561);
// fixed vertices get zero velocity. Thread 0 advances the substep clock.
template <typename ST, typename R>
__global__ void k_velocity(Ptrs<ST, R> P, Consts<R> c, double* time) {
    using V = typename ST::V;
    using Sc = typename ST::Sc;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) time[0] += c.dt_d;
    if (s >= P.nslots) return;
    V v{0, 0, 0, 0};
    if (s < P.nactive) {
        const Sc dt = pick<Sc>(c.dt_d, c.dt_f);
        Sc d[3];
        ST::diff(P.u[s], P.xprev[s], d);
        v.x = d[0] / dt;
        v.y = d[1] / dt;
        v.z = d[2] / dt;
        const MeshMat<R> mat = P.mats[P.slot_mesh[s]];
        Sc vm = sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
        if (vm > Sc(1e-6f)) {
            Sc vn = vm * Sc(mat.exp_damp) - Sc(mat.const_damp);
            vn = vn > Sc(1e-6f) ? vn : Sc(0);
            Sc sc = vn / vm;
            v.x *= sc; v.y *= sc; v.z *= sc;
        } else {
            v.x *= Sc(0); v.y *= Sc(0); v.z *= Sc(0);
        }
    }
    P.vel[s] = v;
}

// Chebyshev over-relaxation of the iterate (VBDPhysicsCompute.cu:910-944):
// x = pp + omega (x - pp), then pp = the iterate before this iteration's sweep.
template <typename ST>
__global__ void k_accel_apply(typename ST::U* u, typename ST::U* prevprev, const typename ST::U* prev_iter,
                              int32_t nactive, double omega, const uint8_t* col_info) {
    using Sc = typename ST::Sc;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nactive) return;
    // vertices in contact are not extrapolated (VBDPhysicsCompute.cu:928, activeCollisionMask)
    if (col_info && col_info[s]) {
        prevprev[s] = prev_iter[s];
        return;
    }
    const typename ST::U x = u[s], pp = prevprev[s];
    Sc d[3];
    ST::diff(x, pp, d);
    const Sc om = Sc(omega);
    typename ST::U r = ST::add(pp, om * d[0], om * d[1], om * d[2]);
    r.w = x.w;
    u[s] = r;
    prevprev[s] = prev_iter[s];
}

// FP32 positions for contact detection: xf[s] = X + u (now), xf[nslots + s] = X + xprev
// (start of the substep), each rounded once from FP64.
template <typename ST>
__global__ void k_gather_xf(const typename ST::U* u, const typename ST::U* xprev, const float4* rest, float4* xf,
                            int32_t nslots) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    const float4 X = rest[s];
    double a[3], b[3];
    ST::to_d(u[s], a);
    ST::to_d(xprev[s], b);
    xf[s] = make_float4(float(double(X.x) + a[0]), float(double(X.y) + a[1]), float(double(X.z) + a[2]), 0.f);
    xf[nslots + s] = make_float4(float(double(X.x) + b[0]), float(double(X.y) + b[1]), float(double(X.z) + b[2]), 0.f);
}

// ---------------------------------------------------------------------------
// Host-order state <-> slots (positions = X + u).
// ---------------------------------------------------------------------------
// Mesh frames (frame non-null): positions = X + F[mesh] + u, F per mesh in FP64.
__device__ __forceinline__ double4 frame_of(const double4* frame, const int32_t* slot_mesh, int s) {
    return frame ? frame[slot_mesh[s]] : make_double4(0.0, 0.0, 0.0, 0.0);
}

template <typename ST>
__global__ void k_scatter_state(typename ST::U* u, const float4* rest, typename ST::V* vel, const float* x,
                                const float* v, const int32_t* slot_of, int32_t n, const double4* frame,
                                const int32_t* slot_mesh) {
    using Sc = typename ST::Sc;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s = slot_of[i];
    if (x) {
        const float4 X = rest[s];
        const double4 F = frame_of(frame, slot_mesh, s);
        double du[3] = {double(x[3 * size_t(i)]) - double(X.x) - F.x,
                        double(x[3 * size_t(i) + 1]) - double(X.y) - F.y,
                        double(x[3 * size_t(i) + 2]) - double(X.z) - F.z};
        u[s] = ST::from_d(du, ST::mass(u[s]));
    }
    if (v) {
        typename ST::V w{Sc(v[3 * size_t(i)]), Sc(v[3 * size_t(i) + 1]), Sc(v[3 * size_t(i) + 2]), Sc(0)};
        vel[s] = w;
    }
}

template <typename ST>
__global__ void k_gather_positions(const typename ST::U* u, const float4* rest, float* out32, double* out64,
                                   const int32_t* slot_of, int32_t n, const double4* frame,
                                   const int32_t* slot_mesh) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s = slot_of[i];
    double p[3];
    ST::to_d(u[s], p);
    const float4 X = rest[s];
    const double4 F = frame_of(frame, slot_mesh, s);
    p[0] += double(X.x) + F.x;
    p[1] += double(X.y) + F.y;
    p[2] += double(X.z) + F.z;
    if (out32) {
        out32[3 * size_t(i)] = float(p[0]);
        out32[3 * size_t(i) + 1] = float(p[1]);
        out32[3 * size_t(i) + 2] = float(p[2]);
    } else {
        out64[3 * size_t(i)] = p[0];
        out64[3 * size_t(i) + 1] = p[1];
        out64[3 * size_t(i) + 2] = p[2];
    }
}

template <typename V>
__global__ void k_gather_velocities(const V* vel, float* out32, double* out64, const int32_t* slot_of, int32_t n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V v = vel[slot_of[i]];
    if (out32) {
        out32[3 * size_t(i)] = float(v.x);
        out32[3 * size_t(i) + 1] = float(v.y);
        out32[3 * size_t(i) + 2] = float(v.z);
    } else {
        out64[3 * size_t(i)] = double(v.x);
        out64[3 * size_t(i) + 1] = double(v.y);
        out64[3 * size_t(i) + 2] = double(v.z);
    }
}

template <typename ST>
__global__ void k_scatter_positions_f64(typename ST::U* u, const float4* rest, const double* in,
                                        const int32_t* slot_of, int32_t n, const double4* frame,
                                        const int32_t* slot_mesh) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int s = slot_of[i];
    const float4 X = rest[s];
    const double4 F = frame_of(frame, slot_mesh, s);
    double du[3] = {in[3 * size_t(i)] - double(X.x) - F.x, in[3 * size_t(i) + 1] - double(X.y) - F.y,
                    in[3 * size_t(i) + 2] - double(X.z) - F.z};
    u[s] = ST::from_d(du, ST::mass(u[s]));
}

template <typename ST>
__global__ void k_scatter_velocities_f64(typename ST::V* vel, const double* in, const int32_t* slot_of, int32_t n) {
    using Sc = typename ST::Sc;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vel[slot_of[i]] = typename ST::V{Sc(in[3 * size_t(i)]), Sc(in[3 * size_t(i) + 1]), Sc(in[3 * size_t(i) + 2]), Sc(0)};
}

}  // namespace dev
}  // namespace gaia
