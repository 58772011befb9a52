// GB300 VBD engine (the class template behind every handle of libgaia_vbd.so).
//
// One handle = one scene on one GPU: device buffers in the slot layout
// described in vbd_kernels.cuh, one CUDA stream, and three CUDA graphs per
// substep (initial step + deformers | all color sweeps of all iterations |
// velocity update). The graphs replace the reference's per-iteration graph
// (VBDPhysics.cpp:1546-1570) and its host<->device syncs per substep.
//
// Each precision mode instantiates the template in a translation unit of its own
// (vbd_engine_<mode>.cu, through the make_engine_* factories), so that they compile in
// parallel; the C ABI (vbd_engine.cu) holds only the base class.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <memory>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/gaia_vbd.h"
#include "host_threads.hpp"
#include "launch_shape.hpp"
#include "scene.hpp"
#include "state_io.hpp"
#include "tet_cd.hpp"
#include "vbd_cluster.cuh"
#include "vbd_convergence.cuh"
#include "vbd_grid.cuh"
#include "vbd_kernels.cuh"

namespace gaia {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

// A bounded device-side wait ran out (GAIA_VBD_E_DEVICE_TIMEOUT).
struct DeviceTimeout : std::runtime_error {
    using std::runtime_error::runtime_error;
};

#define GAIA_CUDA(call)                                                                                  \
    do {                                                                                                 \
        cudaError_t e__ = (call);                                                                        \
        if (e__ != cudaSuccess)                                                                          \
            throw CudaError(std::string(#call) + ": " + cudaGetErrorString(e__) + " (" + __FILE__ + ":" + \
                            std::to_string(__LINE__) + ")");                                             \
    } while (0)

namespace {

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    void alloc(size_t count, size_t* total) {
        if (p) cudaFree(p);
        p = nullptr;
        n = count;
        if (count) {
            GAIA_CUDA(cudaMalloc(&p, count * sizeof(T)));
            if (total) *total += count * sizeof(T);
        }
    }
    void upload(const std::vector<T>& h, size_t* total, cudaStream_t st) {
        alloc(h.size(), total);
        if (!h.empty()) GAIA_CUDA(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    }
};

inline int div_up(int64_t a, int64_t b) { return int((a + b - 1) / b); }

}  // namespace

enum { kSweepMerged = 0, kSweepScenes = 1, kSweepCluster = 2, kSweepGrid = 3 };
constexpr int kVariantDeep = 4;  // solve variant: k_solve with asynchronous one-ring copies
constexpr int kVariantGrid = 5;  // solve variant: k_sweep_grid
constexpr int kVariantPrefetch = 6;  // solve variant: k_solve with the next wave's records prefetched into L2
constexpr int kVariantPipe = 7;      // solve variant: k_solve_pipe, double-buffered TMA tiles on a persistent grid

class EngineBase {
public:
    virtual ~EngineBase() {}
    virtual int mode() const = 0;
    virtual double tuned_ms() const = 0;
    virtual double measure_sweep_ms() = 0;
    virtual void run_steps(int n) = 0;
    virtual void run_steps_timed(int n, float* total_ms, float* sweep_ms) = 0;
    virtual void autotune() = 0;
    virtual void reset() = 0;
    virtual void get_positions(int mesh, double* out) = 0;
    virtual void set_positions(int mesh, const double* in) = 0;
    virtual void get_velocities(int mesh, double* out) = 0;
    virtual void set_velocities(int mesh, const double* in) = 0;
    virtual void set_state_f32(const float* x, const float* v) = 0;
    virtual void get_positions_f32(float* x) = 0;
    virtual void get_velocities_f32(float* v) = 0;
    virtual double energy() = 0;
    virtual void convergence(double* out4) = 0;
    virtual void convergence_log(std::vector<double>& rows) = 0;
    virtual void vertex_force_hessian(int mesh, int v, int friction, double* f3, double* h9) = 0;
    virtual void stats(gaia_vbd_stats* s) = 0;
    virtual void sync() = 0;
    virtual void color_config(int g, int32_t* L, int32_t* B, int32_t* variant, float* ms) const = 0;
    virtual double get_time() = 0;
    virtual void set_time(double t) = 0;
    // tet-mesh contact
    virtual void set_prev_positions(int mesh, const double* in) = 0;
    virtual int collide() = 0;
    virtual void contacts(std::vector<int32_t>& rows) = 0;
};

template <typename ST, typename R>
class Engine : public EngineBase {
    using S4 = typename ST::U;   // per-vertex displacement state
    using V4 = typename ST::V;   // per-vertex velocity
    using Sc = typename ST::Sc;

public:
    // cluster mode: a cluster size whose blocks hold every scene (states and owned records)
    struct ClusterFit {
        int C;
        int32_t pos_cap, nbr_cap, inc_cap;
        size_t bytes;  // without the staging areas
        bool lean;     // only the states in shared memory
    };

    // mode: kSweepMerged (one launch per merged color and iteration), kSweepScenes (one
    // persistent launch per substep running every scene's iterations, scene-major slots),
    // kSweepCluster (the same on thread-block clusters with the scene in shared memory) or
    // kSweepGrid (one cooperative launch per substep over the merged colors, a bounded grid
    // barrier between colors)
    Engine(const Scene& s, int mode) : sc_(s), mode_(mode) {
        GAIA_CUDA(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
        GAIA_CUDA(cudaEventCreate(&ev_a_));
        GAIA_CUDA(cudaEventCreate(&ev_b_));
        GAIA_CUDA(cudaEventCreate(&ev_c_));
        build_layout();
        upload();
        setup_contact();
        setup_frames();
        lanes_ = sc_.p.lanesPerVertex;
        block_ = sc_.p.blockSize;
        if (lanes_ != 0 && lanes_ != 2 && lanes_ != 4 && lanes_ != 8 && lanes_ != 16 && lanes_ != 32)
            throw std::runtime_error("lanesPerVertex must be 2, 4, 8, 16 or 32");
        if (block_ != 0 && (block_ < 64 || block_ > 256 || block_ % 32))
            throw std::runtime_error("blockSize must be a multiple of 32 in [64, 256]");
        use_pdl_ = sc_.p.usePDL;
        small_color_ = sc_.p.smallColorVertices;
        variant_fixed_ = sc_.p.solveVariant;
        if (variant_fixed_ != -1 && variant_fixed_ != 0 && variant_fixed_ != 1 && variant_fixed_ != kVariantDeep &&
            variant_fixed_ != kVariantPrefetch && variant_fixed_ != kVariantPipe)
            throw std::runtime_error("solveVariant must be -1 (autotune), 0 (registers), 1 (TMA-staged), 4 (one-ring "
                                     "copied asynchronously), 6 (registers, next wave's data prefetched into L2) or "
                                     "7 (double-buffered TMA tiles on a persistent grid)");
        // the FP64 engine has neither the TMA variants nor the record prefetch
        if ((variant_fixed_ == 1 || variant_fixed_ == kVariantPrefetch || variant_fixed_ == kVariantPipe) &&
            sizeof(R) != 4)
            variant_fixed_ = 0;
        if (variant_fixed_ >= 0) variant_ = variant_fixed_;
        if (mode_ == kSweepScenes) {
            setup_scenes();
            if ((lanes_ == 0 || block_ == 0) && sc_.p.autotune) autotune_scenes();
            finalize_scenes();
        } else if (mode_ == kSweepCluster) {
            setup_scenes();
            setup_cluster();
            if ((lanes_ == 0 || block_ == 0 || sc_.p.clusterSize == 0) && sc_.p.autotune) autotune_cluster();
            finalize_cluster();
        } else if (mode_ == kSweepGrid) {
            setup_grid();
            if ((lanes_ == 0 || block_ == 0) && sc_.p.autotune) autotune_grid();
            finalize_grid();
        } else {
            if ((lanes_ == 0 || block_ == 0 || variant_fixed_ < 0) && sc_.p.autotune) autotune_impl();
            finalize_cfg();
        }
        if (sc_.p.evaluateConvergence) setup_conv();
        capture();
    }

    int mode() const override { return mode_; }

    void color_config(int g, int32_t* L, int32_t* B, int32_t* variant, float* ms) const override {
        if (g < 0 || size_t(g) >= ccfg_.size()) throw std::invalid_argument("color index out of range");
        if (L) *L = ccfg_[g].L;
        if (B) *B = ccfg_[g].B;
        if (variant) *variant = ccfg_[g].variant;
        if (ms) *ms = ccfg_[g].ms;
    }

    ~Engine() override {
        destroy_graphs();
        if (ev_a_) cudaEventDestroy(ev_a_);
        if (ev_b_) cudaEventDestroy(ev_b_);
        if (ev_c_) cudaEventDestroy(ev_c_);
        if (st_) cudaStreamDestroy(st_);
    }

    // ---- layout ---------------------------------------------------------------
    void build_layout() {
        const auto& meshes = sc_.meshes;
        nmesh_ = int(meshes.size());
        mesh_off_.assign(nmesh_ + 1, 0);
        for (int m = 0; m < nmesh_; ++m) mesh_off_[m + 1] = mesh_off_[m] + meshes[m].nv;
        nslots_ = mesh_off_[nmesh_];
        if (nslots_ > int64_t(INT32_MAX) / 2) throw std::runtime_error("scene too large for 32-bit vertex indices");
        slot_of_.assign(nslots_, -1);
        int32_t slot = 0;
        group_beg_.clear();
        group_mid_.clear();
        group_end_.clear();
        find_long_lists();
        deal_ofs_.assign(1, 0);
        scene_colors_.clear();
        scene_ofs_.assign(1, 0);
        if (mode_ == kSweepScenes || mode_ == kSweepCluster) {
            // scene-major: mesh by mesh, within a mesh its vertices of merged color 0, 1, ...
            std::vector<std::vector<std::vector<int32_t>>> per(size_t(nmesh_),
                                                               std::vector<std::vector<int32_t>>(sc_.groups.size()));
            for (size_t gi = 0; gi < sc_.groups.size(); ++gi) {
                const auto& g = sc_.groups[gi];
                for (size_t i = 0; i + 1 < g.size(); i += 2) {
                    const int m = g[i], v = g[i + 1];
                    if (!meshes[m].fixed[v]) per[size_t(m)][gi].push_back(v);
                }
            }
            for (int m = 0; m < nmesh_; ++m) {
                for (auto& verts : per[size_t(m)]) {
                    if (verts.empty()) continue;
                    const int32_t beg = slot;
                    for (int32_t v : verts)
                        deal_ofs_.push_back(deal_ofs_.back() + meshes[m].nbr_ofs[v + 1] - meshes[m].nbr_ofs[v]);
                    for (int32_t v : verts)
                        if (!is_long(m, v)) slot_of_[mesh_off_[m] + v] = slot++;
                    const int32_t mid = slot;
                    for (int32_t v : verts)
                        if (is_long(m, v)) slot_of_[mesh_off_[m] + v] = slot++;
                    scene_colors_.push_back(make_int4(beg, mid, slot, 0));
                }
                scene_ofs_.push_back(int32_t(scene_colors_.size()));
            }
        } else {
            for (auto& g : sc_.groups) {
                group_beg_.push_back(slot);
                for (int part = 0; part < 2; ++part) {
                    for (size_t i = 0; i + 1 < g.size(); i += 2) {
                        int m = g[i], v = g[i + 1];
                        if (!meshes[m].fixed[v] && is_long(m, v) == (part == 1)) slot_of_[mesh_off_[m] + v] = slot++;
                    }
                    (part ? group_end_ : group_mid_).push_back(slot);
                }
            }
        }
        nactive_ = slot;
        for (int64_t gi = 0; gi < nslots_; ++gi)
            if (slot_of_[gi] < 0) slot_of_[gi] = slot++;
        if (slot != nslots_) throw std::runtime_error("internal: slot assignment incomplete");
        orig_of_.assign(nslots_, 0);
        for (int64_t gi = 0; gi < nslots_; ++gi) orig_of_[slot_of_[gi]] = int32_t(gi);
        slot_mesh_.assign(nslots_, 0);
        for (int m = 0; m < nmesh_; ++m)
            for (int v = 0; v < meshes[m].nv; ++v) slot_mesh_[slot_of_[mesh_off_[m] + v]] = m;

        build_records();
        // per-slot state
        h_pos_.resize(nslots_);
        h_vel_.resize(nslots_);
        h_rest_.resize(nslots_);
        for (int m = 0; m < nmesh_; ++m) {
            const TetMesh& M = meshes[m];
            for (int v = 0; v < M.nv; ++v) {
                int32_t s = slot_of_[mesh_off_[m] + v];
                h_rest_[s] = make_float4(M.X[3 * size_t(v)], M.X[3 * size_t(v) + 1], M.X[3 * size_t(v) + 2], 0.f);
                const double zero[3] = {0.0, 0.0, 0.0};
                h_pos_[s] = ST::from_d(zero, M.mass[v]);  // displacement from rest, mass
                h_vel_[s] = V4{Sc(M.V[3 * size_t(v)]), Sc(M.V[3 * size_t(v) + 1]), Sc(M.V[3 * size_t(v) + 2]), Sc(0)};
            }
        }
        // materials
        h_mats_.resize(nmesh_);
        for (int m = 0; m < nmesh_; ++m) {
            const ObjectParams& o = sc_.objs[m];
            dev::MeshMat<R> mm{};
            mm.mu = R(o.miu);
            mm.lmbd = R(o.lmbd);
            mm.kh = R(o.dampingHydrostatic);
            mm.kd = R(o.dampingDeviatoric);
            mm.exp_damp = R(std::pow(o.exponentialVelDamping, sc_.p.dt));  // VBDPhysics.cpp:794-807
            mm.const_damp = R(o.constantVelDamping * sc_.p.dt);
            mm.init_type = o.initializationType;
            h_mats_[m] = mm;
        }
        // deformers
        for (size_t di = 0; di < sc_.defs.size(); ++di) {
            const DeformerParams& d = sc_.defs[di];
            dev::DeformerDev dd{};
            dd.type = d.type;
            for (int k = 0; k < 3; ++k) {
                dd.axis[k] = d.axis[k];
                dd.speed[k] = d.speed[k];
            }
            dd.omega = d.angularVelocity;
            dd.end_time = d.endTime;
            h_defs_.push_back(dd);
            for (size_t k = 0; k < d.selectedMeshes.size(); ++k) {
                int m = d.selectedMeshes[k];
                for (int32_t v : d.selectedVertices[k]) {
                    const float* X = &meshes[m].X[3 * size_t(v)];
                    double P[3] = {X[0], X[1], X[2]};
                    h_def_slot_.push_back(slot_of_[mesh_off_[m] + v]);
                    h_def_idx_.push_back(int32_t(di));
                    if (d.type == 0) {
                        double OP[3] = {P[0] - d.center[0], P[1] - d.center[1], P[2] - d.center[2]};
                        double dot = OP[0] * d.axis[0] + OP[1] * d.axis[1] + OP[2] * d.axis[2];
                        for (int c = 0; c < 3; ++c) {
                            double root = dot * d.axis[c];
                            h_def_a_.push_back(root);
                            h_def_b_.push_back(P[c] - root);
                        }
                    } else {
                        for (int c = 0; c < 3; ++c) {
                            h_def_a_.push_back(P[c]);
                            h_def_b_.push_back(0.0);
                        }
                    }
                }
            }
        }
        // constants
        const PhysicsParams& p = sc_.p;
        c_.dt = R(p.dt);
        c_.inv_dt = R(1.0 / p.dt);
        c_.dt2inv = R(p.dtSqrReciprocal);
        c_.dt_d = p.dt;
        c_.dt_f = float(p.dt);
        for (int k = 0; k < 3; ++k) {
            c_.g[k] = p.gravity[k];
            c_.lo[k] = p.worldLo[k];
            c_.hi[k] = p.worldHi[k];
            c_.g_f[k] = float(p.gravity[k]);
            c_.lo_f[k] = float(p.worldLo[k]);
            c_.hi_f[k] = float(p.worldHi[k]);
        }
        c_.kb = R(p.boundaryCollisionStiffness);
        c_.kc = R(p.collisionStiffness);
        c_.fr_mu = R(p.boundaryFrictionDynamic);
        c_.fr_epsU = R(p.boundaryFrictionEpsV * p.dt);
        c_.step = R(p.stepSize);
        c_.step_gd = R(p.stepSizeGD);
        c_.plane = p.usePlaneGround ? 1 : 0;
        c_.assoc_grav = p.associateGravityWithInertia ? 1 : 0;
        c_.spin_limit = p.waitPollLimit >= 0 ? p.waitPollLimit : dev::kMbarSpinLimit;
    }

    // Vertices with long neighbour lists come last in their color and are solved a warp per
    // vertex, in a launch of their own where the others take fewer lanes: the staging areas of a
    // launch are sized by its longest list, and only that form holds lists of more than kSegNbrs.
    // Long is more than 32 neighbours (a tet mesh has about 14, a 5-tet lattice up to 18), or 64
    // or kSegNbrs where more than a 32nd of the vertices would be long. Vertices of up to
    // kFewTets tets are not counted out: 42 tets hold at most 126 neighbours, and about 23 where
    // they share faces. A step of a 40^3 lattice at 4 lanes (FP32, 10 iterations) takes 1.15 times
    // as long with one hub of 202 neighbours beside it; when such a vertex changed the whole scene
    // over to a warp per vertex, 1.57 times.
    static constexpr int kFewTets = 42;
    void find_long_lists() {
        const auto& meshes = sc_.meshes;
        std::vector<std::vector<uint8_t>> over(meshes.size());  // 1: > 32, 2: > 64, 3: > kSegNbrs neighbours
        int64_t count[4] = {0, 0, 0, 0}, active = 0;
        std::vector<int32_t> nb;
        for (size_t m = 0; m < meshes.size(); ++m) {
            const TetMesh& M = meshes[m];
            for (int32_t v = 0; v < M.nv; ++v) {
                if (M.fixed[v]) continue;
                ++active;
                if (M.nbr_ofs[v + 1] - M.nbr_ofs[v] <= kFewTets) continue;
                nb.clear();
                for (int q = M.nbr_ofs[v]; q < M.nbr_ofs[v + 1]; ++q)
                    for (int j = 0; j < 4; ++j)
                        if (j != M.nbr_order[q]) nb.push_back(M.tets[4 * size_t(M.nbr_tet[q]) + j]);
                std::sort(nb.begin(), nb.end());
                const int64_t n = std::unique(nb.begin(), nb.end()) - nb.begin();
                const int k = n > dev::kSegNbrs ? 3 : (n > 64 ? 2 : (n > 32 ? 1 : 0));
                if (!k) continue;
                if (over[m].empty()) over[m].assign(size_t(M.nv), 0);
                over[m][size_t(v)] = uint8_t(k);
                ++count[k];
            }
        }
        int line = 1;
        if (32 * (count[1] + count[2] + count[3]) > active) line = 32 * (count[2] + count[3]) > active ? 3 : 2;
        any_long_ = false;
        for (auto& o : over)
            for (auto& k : o) {
                k = k >= line ? 1 : 0;
                any_long_ = any_long_ || k;
            }
        long_ = std::move(over);
    }
    bool is_long(int m, int v) const { return !long_[size_t(m)].empty() && long_[size_t(m)][size_t(v)]; }

    // One-ring and incidence records of the active slots (layout in vbd_kernels.cuh), the host
    // threads taking contiguous ranges of slices; a color (of the merged sweep, or of one
    // scene) starts a slice, and so do its long lists. Neighbours are listed by slot, so that the k-th neighbours of
    // consecutive vertices of a regular mesh are consecutive too; incidences keep the mesh's
    // ascending tet order, and a segment closes when the next tet's vertices would take it
    // past kSegNbrs neighbours.
    void build_records() {
        const auto& meshes = sc_.meshes;
        inc_ofs_.assign(size_t(nactive_) + 1, 0);
        int64_t total = 0;
        for (int32_t s = 0; s < nactive_; ++s) {
            const int m = slot_mesh_[s], v = orig_of_[s] - int32_t(mesh_off_[m]);
            total += meshes[m].nbr_ofs[v + 1] - meshes[m].nbr_ofs[v];
            inc_ofs_[s + 1] = checked_count(total);
        }
        ninc_ = int32_t(total);
        std::vector<int2> slices;  // slot ranges
        auto cut = [&](int beg, int end) {
            for (int v = beg; v < end; v += dev::kSlice) slices.push_back(make_int2(v, std::min(end, v + dev::kSlice)));
        };
        if (mode_ == kSweepScenes || mode_ == kSweepCluster)
            for (int4 c : scene_colors_) {
                cut(c.x, c.y);
                cut(c.y, c.z);
            }
        else
            for (size_t g = 0; g < group_beg_.size(); ++g) {
                cut(group_beg_[g], group_mid_[g]);
                cut(group_mid_[g], group_end_[g]);
            }
        struct Seg {
            int32_t slot;                // its vertex
            int4 r;                      // as vrec
        };
        struct Part {                    // of one host thread
            std::vector<dev::NbrRec<R>> nbr;
            std::vector<dev::IncRec<R>> inc;
            std::vector<Seg> more;       // further segments
        };
        const int nt = std::max(1, std::min<int>(int(std::thread::hardware_concurrency()), int(ninc_ / 65536) + 1));
        std::vector<Part> part{size_t(nt)};
        vrec_.assign(size_t(nactive_), make_int4(0, 0, 0, 0));
        auto range = [&](int k) { return size_t(int64_t(slices.size()) * k / nt); };
        auto work = [&](int k) {
            Part& out = part[size_t(k)];
            std::vector<dev::NbrRec<R>> nbr;
            std::vector<dev::IncRec<R>> inc;
            // the lists of one segment into place: every kSlice-th record from the segment's first
            auto place = [&](int4 seg) {
                const int at = dev::place_of(seg.z);
                for (size_t i = 0; i < nbr.size(); ++i) out.nbr[dev::record_index(seg.x + int(i), at)] = nbr[i];
                for (size_t i = 0; i < inc.size(); ++i) out.inc[dev::record_index(seg.y + int(i), at)] = inc[i];
            };
            std::vector<std::vector<dev::NbrRec<R>>> ln(dev::kSlice);
            std::vector<std::vector<dev::IncRec<R>>> li(dev::kSlice);
            for (size_t sl = range(k); sl < range(k + 1); ++sl) {
                const int2 rg = slices[sl];
                size_t mn = 0, mi = 0;
                std::vector<Seg> extra;
                std::vector<std::pair<std::vector<dev::NbrRec<R>>, std::vector<dev::IncRec<R>>>> extra_lists;
                for (int32_t s = rg.x; s < rg.y; ++s) {
                    bool first = true;
                    segments_of(s, nbr, inc, [&] {
                        if (first) {
                            ln[size_t(s - rg.x)] = nbr;
                            li[size_t(s - rg.x)] = inc;
                            mn = std::max(mn, nbr.size());
                            mi = std::max(mi, inc.size());
                        } else {
                            extra.push_back({s, make_int4(0, 0, dev::pack_nbrs(int(nbr.size()), 0), int(inc.size()))});
                            extra_lists.emplace_back(nbr, inc);
                        }
                        first = false;
                    });
                }
                // rows of this part so far
                const int nb = checked_count(int64_t(out.nbr.size() / dev::kSlice));
                const int ib = checked_count(int64_t(out.inc.size() / dev::kSlice));
                size_t en = 0, ei = 0;
                for (auto& e : extra_lists) {
                    en += e.first.size();
                    ei += e.second.size();
                }
                out.nbr.resize(out.nbr.size() + dev::kSlice * (mn + en));
                out.inc.resize(out.inc.size() + dev::kSlice * (mi + ei));
                for (int32_t s = rg.x; s < rg.y; ++s) {
                    nbr = ln[size_t(s - rg.x)];
                    inc = li[size_t(s - rg.x)];
                    vrec_[size_t(s)] = make_int4(nb, ib, dev::pack_nbrs(int(nbr.size()), s - rg.x), int(inc.size()));
                    place(vrec_[size_t(s)]);
                }
                int n1 = nb + int(mn), i1 = ib + int(mi);
                for (size_t e = 0; e < extra.size(); ++e) {
                    nbr = extra_lists[e].first;
                    inc = extra_lists[e].second;
                    extra[e].r.x = n1;
                    extra[e].r.y = i1;
                    place(extra[e].r);
                    n1 += int(nbr.size());
                    i1 += int(inc.size());
                    out.more.push_back(extra[e]);
                }
            }
        };
        run_parts(nt, work);
        size_t nn = 0, ni = 0;
        for (auto& q : part) {
            nn += q.nbr.size();
            ni += q.inc.size();
        }
        nbr_end_ = checked_count(int64_t(nn / dev::kSlice));
        inc_end_ = checked_count(int64_t(ni / dev::kSlice));
        // the parts end to end, padded for the copies of whole slices that run past the last list
        max_nbr_all_ = max_nbr_short_ = max_inc_all_ = 2;
        h_nbr_.clear();
        h_inc_.clear();
        h_nbr_.reserve(nn + size_t(dev::kSlice) * 1024);
        h_inc_.reserve(ni + size_t(dev::kSlice) * 1024);
        segs_.clear();
        std::vector<Seg> more;
        for (int k = 0; k < nt; ++k) {
            Part& q = part[size_t(k)];
            const int n0 = int(h_nbr_.size() / dev::kSlice), i0 = int(h_inc_.size() / dev::kSlice);
            if (range(k) < range(k + 1))
                for (int32_t s = slices[range(k)].x; s < slices[range(k + 1) - 1].y; ++s) {
                    vrec_[size_t(s)].x += n0;
                    vrec_[size_t(s)].y += i0;
                }
            for (Seg& e : q.more) {
                e.r.x += n0;
                e.r.y += i0;
                more.push_back(e);
            }
            h_nbr_.insert(h_nbr_.end(), q.nbr.begin(), q.nbr.end());
            h_inc_.insert(h_inc_.end(), q.inc.begin(), q.inc.end());
        }
        for (int32_t q = 0; q < nactive_; ++q) {
            const int4 r = vrec_[size_t(q)];
            const int n = (dev::nbrs_of(r.z) + 1) & ~1;
            max_nbr_all_ = std::max(max_nbr_all_, n);
            if (!long_slot(q)) max_nbr_short_ = std::max(max_nbr_short_, n);
            max_inc_all_ = std::max(max_inc_all_, r.w);
        }
        for (const Seg& e : more) max_nbr_all_ = std::max(max_nbr_all_, (dev::nbrs_of(e.r.z) + 1) & ~1);
        h_nbr_.resize(h_nbr_.size() + size_t(dev::kSlice) * max_nbr_all_, dev::NbrRec<R>{});
        h_inc_.resize(h_inc_.size() + size_t(dev::kSlice) * max_inc_all_, dev::IncRec<R>{});
        multi_seg_ = !more.empty();
        vmore_.clear();
        if (any_long_) {  // (the sweeps read it for every long list)
            vmore_.assign(size_t(nactive_), make_int2(0, 0));
            std::stable_sort(more.begin(), more.end(), [](const Seg& a, const Seg& b) { return a.slot < b.slot; });
            for (size_t i = 0; i < more.size(); ++i) {
                int2& q = vmore_[size_t(more[i].slot)];
                if (q.y == 0) q.x = int(i);
                q.y = int(i) + 1;
                segs_.push_back(more[i].r);
            }
        }
    }

    // The edge weights of one segment in the compute type. FP32: each rounded to the one of its
    // two neighbouring floats that keeps sum (k - K) r small (r the rest edges), largest first:
    // the weights of a rigid or linear motion e = A r then sum as the FP64 ones do, although the
    // terms of a flat one-ring are far larger than their sum.
    static void round_weights(int n, const double* K, const double (*r)[3], R* k) {
        for (int i = 0; i < n; ++i) k[i] = R(K[i]);
        if (sizeof(R) != 4 || n < 2) return;
        double d0[dev::kSegNbrs][3], d1[dev::kSegNbrs][3], key[dev::kSegNbrs], s[3] = {0, 0, 0};
        R alt[dev::kSegNbrs];
        int order[dev::kSegNbrs];
        for (int i = 0; i < n; ++i) {
            const R inf = std::numeric_limits<R>::infinity();
            alt[i] = std::nextafter(k[i], double(k[i]) < K[i] ? inf : -inf);
            key[i] = 0.0;
            for (int c = 0; c < 3; ++c) {
                d0[i][c] = (double(k[i]) - K[i]) * r[i][c];
                d1[i][c] = (double(alt[i]) - K[i]) * r[i][c];
                key[i] += (d1[i][c] - d0[i][c]) * (d1[i][c] - d0[i][c]);
            }
            order[i] = i;
        }
        std::sort(order, order + n, [&](int a, int b) { return key[a] != key[b] ? key[a] > key[b] : a < b; });
        auto norm = [](const double* a, const double* b, const double* c) {
            double q = 0.0;
            for (int j = 0; j < 3; ++j) q += (a[j] - b[j] + c[j]) * (a[j] - b[j] + c[j]);
            return q;
        };
        const double zero[3] = {0, 0, 0};
        for (int q = 0; q < n; ++q) {
            const int i = order[q];
            if (norm(s, zero, d1[i]) < norm(s, zero, d0[i])) {
                std::swap(k[i], alt[i]);
                std::swap(d0[i], d1[i]);
            }
            for (int c = 0; c < 3; ++c) s[c] += d0[i][c];
        }
        for (int pass = 0; pass < 2; ++pass)
            for (int q = 0; q < n; ++q) {
                const int i = order[q];
                if (!(norm(s, d0[i], d1[i]) < 0.99 * norm(s, zero, zero))) continue;
                for (int c = 0; c < 3; ++c) s[c] += d1[i][c] - d0[i][c];
                std::swap(k[i], alt[i]);
                std::swap(d0[i], d1[i]);
            }
    }

    // The segments of slot s one after another in nbr and inc (done() is called after each).
    template <typename Fn>
    void segments_of(int32_t s, std::vector<dev::NbrRec<R>>& nbr, std::vector<dev::IncRec<R>>& inc, Fn&& done) const {
        const int m = slot_mesh_[s];
        const TetMesh& M = sc_.meshes[m];
        const int v = orig_of_[s] - int32_t(mesh_off_[m]);
        int32_t slots[dev::kSegNbrs];
        double K[dev::kSegNbrs], rest[dev::kSegNbrs][3];
        R k[dev::kSegNbrs];
        const float* Xo = &M.X[3 * size_t(v)];
        int n = 0;
        inc.clear();
        auto close = [&] {
            // by slot: rank of each neighbour, records in that order, positions renamed
            int order[dev::kSegNbrs];
            uint32_t rank[dev::kSegNbrs];
            for (int i = 0; i < n; ++i) order[i] = i;
            std::sort(order, order + n, [&](int a, int b) { return slots[a] < slots[b]; });
            round_weights(n, K, rest, k);
            nbr.resize(size_t(n));
            for (int i = 0; i < n; ++i) {
                rank[order[i]] = uint32_t(i);
                nbr[size_t(i)] = dev::NbrRec<R>{};
                nbr[size_t(i)].slot = slots[order[i]];
                nbr[size_t(i)].k = k[order[i]];
            }
            for (auto& q : inc)
                q.idx = rank[q.idx & 255u] | rank[(q.idx >> 8) & 255u] << 8 | rank[(q.idx >> 16) & 255u] << 16 |
                        rank[q.idx >> 24] << 24;
            done();
            n = 0;
            inc.clear();
        };
        for (int q = M.nbr_ofs[v]; q < M.nbr_ofs[v + 1]; ++q) {
            const int t = M.nbr_tet[q], o = M.nbr_order[q];
            const double* Di = &M.dminv[9 * size_t(t)];
            double row[4][3];
            for (int c = 0; c < 3; ++c) {
                row[0][c] = -(Di[3 * c] + Di[3 * c + 1] + Di[3 * c + 2]);
                for (int j = 1; j < 4; ++j) row[j][c] = Di[3 * c + (j - 1)];
            }
            int others[3], w = 0;
            for (int j = 0; j < 4; ++j)
                if (j != o) others[w++] = j;
            if (o & 1) std::swap(others[0], others[1]);  // keeps det of the rows = det(DmInv)
            // The face normals are taken at the vertex opposite the face's longest edge, the volume
            // change at the vertex nearest to o: the parts that cancel in a rotated tet are then
            // smallest (a rotation of the three vertices keeps the determinant's sign).
            std::array<double, 3> r[3];
            for (int i = 0; i < 3; ++i)
                for (int c = 0; c < 3; ++c)
                    r[i][c] = double(M.X[3 * size_t(M.tets[4 * size_t(t) + others[i]]) + c]) - double(Xo[c]);
            auto edge2 = [&](int i, int j) {
                double q = 0.0;
                for (int c = 0; c < 3; ++c) q += (r[i][c] - r[j][c]) * (r[i][c] - r[j][c]);
                return q;
            };
            int first = 0, near = 0;
            for (int i = 1; i < 3; ++i) {
                if (edge2((i + 1) % 3, (i + 2) % 3) > edge2((first + 1) % 3, (first + 2) % 3)) first = i;
                auto len2 = [&](int j) { return r[j][0] * r[j][0] + r[j][1] * r[j][1] + r[j][2] * r[j][2]; };
                if (len2(i) < len2(near)) near = i;
            }
            std::rotate(others, others + first, others + 3);
            std::rotate(r, r + first, r + 3);
            near = (near - first + 3) % 3;
            int32_t sl[3];
            int at[3], fresh = 0;
            auto find = [&](int32_t x) {
                for (int i = 0; i < n; ++i)
                    if (slots[i] == x) return i;
                return -1;
            };
            for (int i = 0; i < 3; ++i) {
                sl[i] = slot_of_[mesh_off_[m] + M.tets[4 * size_t(t) + others[i]]];
                fresh += find(sl[i]) < 0 ? 1 : 0;
            }
            if (n + fresh > dev::kSegNbrs) close();
            for (int i = 0; i < 3; ++i) {
                at[i] = find(sl[i]);
                if (at[i] < 0) {
                    at[i] = n;
                    slots[n] = sl[i];
                    for (int c = 0; c < 3; ++c) rest[n][c] = r[i][c];
                    K[n++] = 0.0;
                }
                const double* a = row[o];
                const double* b = row[others[i]];
                K[at[i]] += M.vol[t] * (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]);
            }
            dev::IncRec<R> rec{};
            rec.idx = uint32_t(at[0]) | uint32_t(at[1]) << 8 | uint32_t(at[2]) << 16 | uint32_t(at[near]) << 24;
            rec.w = R(1.0 / (6.0 * M.vol[t]));
            inc.push_back(rec);
        }
        close();
    }

    // Longest lists in the slot range [beg, end): neighbours (even: the staging entries per
    // vertex) and incidences.
    int2 max_lists(int beg, int end) {
        const auto key = std::make_pair(beg, end);
        auto it = lists_cache_.find(key);
        if (it != lists_cache_.end()) return it->second;
        int2 m = make_int2(2, 1);
        for (int v = beg; v < end; ++v) {
            m.x = std::max(m.x, (dev::nbrs_of(vrec_[size_t(v)].z) + 1) & ~1);
            m.y = std::max(m.y, vrec_[size_t(v)].w);
            if (several_segments(v)) m.x = dev::kSegNbrs;
        }
        if (end - beg > 1) lists_cache_[key] = m;  // (a single vertex is a probed one: any of the scene's)
        return m;
    }
    bool several_segments(int slot) const { return multi_seg_ && vmore_[size_t(slot)].y > vmore_[size_t(slot)].x; }
    bool long_slot(int slot) const {
        const int m = slot_mesh_[size_t(slot)];
        return is_long(m, orig_of_[size_t(slot)] - int32_t(mesh_off_[m]));
    }
    // Bytes of the staging areas of a block of B threads.
    static size_t stage_bytes(int cap, int L, int B) {
        return size_t(B / L) * size_t(cap) * (16 * dev::Stage<1, ST, R>::kParts);
    }
    // The same for a persistent sweep: L lanes per vertex, a warp per vertex for the long lists.
    dev::SweepStage sweep_stage(int L) const {
        dev::SweepStage S;
        S.cap = max_nbr_short_;
        S.cap_long = any_long_ ? max_nbr_all_ : 0;
        S.warp_bytes = int(std::max(stage_bytes(S.cap, L, 32), stage_bytes(S.cap_long, 32, 32)));
        return S;
    }
    size_t sweep_stage_bytes(int L, int B) const { return size_t(B / 32) * size_t(sweep_stage(L).warp_bytes); }
    int fit_sweep_lanes(int L, int B) const {
        while (L < 32 && sweep_stage_bytes(L, B) > kTmaSmemMax) L *= 2;
        return L;
    }
    // Fewest lanes per vertex, at least L, whose staging fits the shared memory of a block.
    int fit_lanes(int L, int B, int beg, int end) {
        while (L < 32 && stage_bytes(max_lists(beg, end).x, L, B) > kTmaSmemMax) L *= 2;
        return L;
    }
    // The limit of a kernel's dynamic shared memory, raised once for every launch: a captured
    // launch must not depend on what a later one asks for. The 48 KB that need no raise hold
    // the kernel's static shared memory too.
    template <typename K>
    static void allow_smem(K kern, size_t bytes) {
        if (bytes > 40 * 1024)
            GAIA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTmaSmemMax)));
    }

    void upload() {
        bytes_ = 0;
        d_pos_.upload(h_pos_, &bytes_, st_);
        d_rest_.upload(h_rest_, &bytes_, st_);
        d_vel_.upload(h_vel_, &bytes_, st_);
        d_y_.upload(h_pos_, &bytes_, st_);
        d_xprev_.upload(h_pos_, &bytes_, st_);
        d_vprev_.upload(h_vel_, &bytes_, st_);
        d_inc_ofs_.upload(inc_ofs_, &bytes_, st_);
        d_vrec_.upload(vrec_, &bytes_, st_);
        d_vmore_.upload(vmore_, &bytes_, st_);
        d_segs_.upload(segs_, &bytes_, st_);
        d_nbr_.upload(h_nbr_, &bytes_, st_);
        d_inc_.upload(h_inc_, &bytes_, st_);
        d_slot_mesh_.upload(slot_mesh_, &bytes_, st_);
        d_mats_.upload(h_mats_, &bytes_, st_);
        d_slot_of_.upload(slot_of_, &bytes_, st_);
        d_counters_.alloc(dev::CNT_N, &bytes_);
        GAIA_CUDA(cudaMemsetAsync(d_counters_.p, 0, dev::CNT_N * sizeof(unsigned long long), st_));
        d_time_.alloc(1, &bytes_);
        GAIA_CUDA(cudaMemsetAsync(d_time_.p, 0, sizeof(double), st_));
        d_def_slot_.upload(h_def_slot_, &bytes_, st_);
        d_def_idx_.upload(h_def_idx_, &bytes_, st_);
        d_def_a_.upload(h_def_a_, &bytes_, st_);
        d_def_b_.upload(h_def_b_, &bytes_, st_);
        d_defs_.upload(h_defs_, &bytes_, st_);
        if (sc_.p.useAccelerator) {
            d_acc_pp_.alloc(nslots_, &bytes_);
            d_acc_prev_.alloc(nslots_, &bytes_);
        }
        d_stage_f32_.alloc(6 * size_t(nslots_), &bytes_);
        d_stage_f64_.alloc(3 * size_t(nslots_), &bytes_);
        d_probe_.alloc(12, &bytes_);
        GAIA_CUDA(cudaStreamSynchronize(st_));
        // keep host copies small: records are device-only from here on
        std::vector<dev::NbrRec<R>>().swap(h_nbr_);
        std::vector<dev::IncRec<R>>().swap(h_inc_);
    }

    dev::Ptrs<ST, R> ptrs() const {
        dev::Ptrs<ST, R> P;
        P.u = d_pos_.p;
        P.rest = d_rest_.p;
        P.y = d_y_.p;
        P.xprev = d_xprev_.p;
        P.vel = d_vel_.p;
        P.vprev = d_vprev_.p;
        P.vrec = d_vrec_.p;
        P.vmore = d_vmore_.p;
        P.segs = d_segs_.p;
        P.nbr = d_nbr_.p;
        P.inc = d_inc_.p;
        P.slot_mesh = d_slot_mesh_.p;
        P.mats = d_mats_.p;
        P.counters = d_counters_.p;
        P.nactive = nactive_;
        P.nslots = int32_t(nslots_);
        const tetcd::Records rc = cd_.records();
        P.col_info = rc.info;
        P.col_own = rc.own;
        P.col_rel = rc.rel;
        P.mesh_fric = d_mesh_fric_.p;
        P.snap = d_snap_.p;
        P.frame_shift = frames_ ? d_frame_shift_.p : nullptr;
        P.frame_F = frames_ ? d_frame_F_.p : nullptr;
        P.rest_fh = frames_ ? d_rest_fh_.p : nullptr;
        P.rest_fl = frames_ ? d_rest_fl_.p : nullptr;
        return P;
    }

    // ---- mesh frames --------------------------------------------------------------------
    // FP32-compute engines keep each mesh's states relative to a frame offset F that follows
    // the mesh (k_frame_update, once per substep). Off with contact detection (contacts
    // couple meshes, whose frames differ) and with deformers (they set absolute positions).
    void setup_frames() {
        frames_ = sizeof(R) == 4 && sc_.p.meshFrames && !cd_.enabled() && h_def_slot_.empty() && nmesh_ > 0;
        if (!frames_) return;
        std::vector<int32_t> ref(size_t(nmesh_), -1);
        for (int m = 0; m < nmesh_; ++m)
            for (int v = 0; v < sc_.meshes[m].nv; ++v)
                if (!sc_.meshes[m].fixed[v]) {
                    ref[size_t(m)] = slot_of_[mesh_off_[m] + v];
                    break;
                }
        d_frame_ref_.upload(ref, &bytes_, st_);
        d_frame_F_.alloc(nmesh_, &bytes_);
        d_frame_shift_.alloc(nmesh_, &bytes_);
        d_rest_fh_.alloc(nslots_, &bytes_);
        d_rest_fl_.alloc(nslots_, &bytes_);
        reset_frames();
    }

    // F = 0, no shift, X + F = X
    void reset_frames() {
        if (!frames_) return;
        GAIA_CUDA(cudaMemsetAsync(d_frame_F_.p, 0, nmesh_ * sizeof(double4), st_));
        GAIA_CUDA(cudaMemsetAsync(d_frame_shift_.p, 0, nmesh_ * sizeof(float4), st_));
        GAIA_CUDA(cudaMemcpyAsync(d_rest_fh_.p, d_rest_.p, nslots_ * sizeof(float4), cudaMemcpyDeviceToDevice, st_));
        GAIA_CUDA(cudaMemsetAsync(d_rest_fl_.p, 0, nslots_ * sizeof(float4), st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    const double4* frame_ptr() const { return frames_ ? d_frame_F_.p : nullptr; }

    // ---- tet-mesh contact -----------------------------------------------------------
    // Surface faces / vertices, surface rings and tets of all meshes in slot terms for
    // the detector, the detector itself, and the first hierarchies.
    void setup_contact() {
        const PhysicsParams& p = sc_.p;
        tetcd::Params prm;
        prm.ccd = p.allowCCD;
        prm.dcd = p.allowDCD;
        prm.handle_self = p.handleSelfCollision;
        prm.check_feasible = p.checkFeasibleRegion;
        prm.feasible_eps = float(p.feasibleRegionEpsilon);
        prm.off_height = float(p.collisionOffHeight);
        prm.check_traverse = p.checkTetTraverse;
        prm.traverse_non_self = p.tetrahedralTraverseForNonSelfIntersection;
        prm.stop_after_passing = p.stopTraversingAfterPassingQueryPoint;
        prm.shift_to_center = p.shiftQueryPointToCenter;
        prm.static_traverse = p.useStaticTraverse;
        prm.center_shift = float(p.centerShiftLevel);
        prm.ray_eps = float(p.rayTriIntersectionEPSILON);
        prm.max_search_mult = float(p.maxSearchDistanceMultiplier);
        tetcd::Topo t;
        t.nslots = int32_t(nslots_);
        t.face_ofs.assign(nmesh_ + 1, 0);
        std::vector<std::vector<int32_t>> ring(static_cast<size_t>(nslots_));
        for (int m = 0; m < nmesh_; ++m) {
            const TetMesh& M = sc_.meshes[m];
            auto slot = [&](int32_t v) { return slot_of_[mesh_off_[m] + v]; };
            const int32_t f0 = int32_t(t.faces.size());
            const size_t nf = M.sfaces.size() / 3;
            t.face_ofs[m + 1] = f0 + int32_t(nf);
            for (size_t f = 0; f < nf; ++f) {
                t.faces.push_back(make_int4(slot(M.sfaces[3 * f]), slot(M.sfaces[3 * f + 1]), slot(M.sfaces[3 * f + 2]), m));
                int32_t nb[3];
                for (int k = 0; k < 3; ++k) nb[k] = M.sface_nbr[3 * f + k] < 0 ? -1 : f0 + M.sface_nbr[3 * f + k];
                t.face_nbr.push_back(make_int4(nb[0], nb[1], nb[2], 0));
            }
            for (int32_t v : M.sverts) t.verts.push_back(make_int2(slot(v), m));
            for (int32_t v = 0; v < M.nv; ++v)
                for (int32_t r = M.sring_ofs[v]; r < M.sring_ofs[v + 1]; ++r) ring[slot(v)].push_back(slot(M.sring[r]));
            const int32_t t0 = int32_t(t.tets.size());
            for (size_t f = 0; f < nf; ++f) t.face_tet.push_back(make_int2(t0 + M.sface_tet[2 * f], M.sface_tet[2 * f + 1]));
            for (int32_t k = 0; k < M.ntet; ++k) {
                const int32_t* tv = &M.tets[4 * size_t(k)];
                t.tets.push_back(make_int4(slot(tv[0]), slot(tv[1]), slot(tv[2]), slot(tv[3])));
                t.tet_mesh.push_back(m);
                int32_t nb[4];
                for (int j = 0; j < 4; ++j) nb[j] = M.tet_nbr[4 * size_t(k) + j] < 0 ? -1 : t0 + M.tet_nbr[4 * size_t(k) + j];
                t.tet_nbr.push_back(make_int4(nb[0], nb[1], nb[2], nb[3]));
            }
        }
        t.ring_ofs.assign(size_t(nslots_) + 1, 0);
        for (int64_t s = 0; s < nslots_; ++s) {
            t.ring.insert(t.ring.end(), ring[s].begin(), ring[s].end());
            t.ring_ofs[s + 1] = int32_t(t.ring.size());
        }
        cd_.init(t, prm, bytes_);
        if (!cd_.enabled()) return;
        std::vector<double2> fr(nmesh_);
        for (int m = 0; m < nmesh_; ++m) fr[m] = make_double2(sc_.objs[m].frictionDynamic, sc_.objs[m].frictionEpsV);
        d_mesh_fric_.upload(fr, &bytes_, st_);
        d_xf_.alloc(2 * size_t(nslots_), &bytes_);
        d_snap_.alloc(2 * size_t(nslots_), &bytes_);
        GAIA_CUDA(cudaMemsetAsync(d_snap_.p, 0, 2 * size_t(nslots_) * sizeof(S4), st_));
        enqueue_gather();
        cd_.build(d_xf_.p, st_);
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    void enqueue_gather() {
        dev::k_gather_xf<ST><<<div_up(nslots_, 256), 256, 0, st_>>>(d_pos_.p, d_xprev_.p, d_rest_.p, d_xf_.p, int32_t(nslots_));
        GAIA_CUDA(cudaGetLastError());
    }

    // One detection pass on the current and start-of-substep positions.
    void enqueue_detection(bool intermediate, bool rebuild) {
        if (!cd_.enabled()) return;
        enqueue_gather();
        cd_.enqueue(d_xf_.p, intermediate, rebuild, st_);
    }

    // Contact snapshots of the vertices with records for the iteration that follows a detection.
    void enqueue_contact_snapshot(int it) {
        const tetcd::Records rc = cd_.records();
        dev::k_contact_snapshot<ST><<<kContactBlocks, 128, 0, st_>>>(d_pos_.p, d_snap_.p, int32_t(nslots_),
                                                                    (it & 1) ? 0 : 1, rc.list, rc.nlist);
        GAIA_CUDA(cudaGetLastError());
    }

    // ---- kernels ----------------------------------------------------------------
    // Launch of one color's solve. pdl: launched as a programmatic dependent of
    // the previous kernel in the stream (its static-data prologue overlaps that
    // kernel's tail; k_solve waits on griddepcontrol before reading positions).
    template <bool PROBE, bool DEEP, int L, bool MULTI = false>
    void launch_solve_l(int B, int beg, int end, int2 color, int flags, double* probe, bool pdl, bool prefetch) {
        if (cd_.enabled()) launch_solve_c<PROBE, DEEP, L, MULTI, true>(B, beg, end, color, flags, probe, pdl, prefetch);
        else launch_solve_c<PROBE, DEEP, L, MULTI, false>(B, beg, end, color, flags, probe, pdl, prefetch);
    }
    template <bool PROBE, bool DEEP, int L, bool MULTI, bool CONTACT>
    void launch_solve_c(int B, int beg, int end, int2 color, int flags, double* probe, bool pdl, bool prefetch) {
        const int cap = max_lists(beg, end).x;
        const size_t smem = stage_bytes(cap, L, B);
        auto kern = dev::k_solve<L, ST, R, PROBE, DEEP, MULTI, CONTACT>;
        allow_smem(kern, smem);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(div_up(int64_t(end - beg) * L, B));
        cfg.blockDim = dim3(B);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st_;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = pdl ? attr : nullptr;
        cfg.numAttrs = pdl ? 1 : 0;
        // the prefetching variant fetches for the warps one resident wave ahead
        const int pf = prefetch ? std::max(1, blocks_per_sm(kern, B, smem)) * sm_count() * (B / 32) : 0;
        GAIA_CUDA(cudaLaunchKernelEx(&cfg, kern, ptrs(), c_, beg, end, color, flags, probe, pf, cap));
    }

    template <typename K>
    int blocks_per_sm(K kern, int B, size_t smem) {
        const auto key = std::make_tuple(reinterpret_cast<const void*>(kern), B, smem);
        auto it = occ_cache_.find(key);
        if (it != occ_cache_.end()) return it->second;
        int per_sm = 0;
        GAIA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, B, smem));
        return occ_cache_[key] = per_sm;
    }

    int sm_count() {
        if (sms_ == 0) {
            int dev = 0;
            GAIA_CUDA(cudaGetDevice(&dev));
            GAIA_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
        }
        return sms_;
    }

    // Largest neighbour and incidence record ranges of any block of vpb consecutive vertices
    // in [beg, end), as rec_tile (vbd_kernels.cuh) takes them.
    int2 max_records(int beg, int end, int vpb) {
        auto key = std::make_pair(beg, vpb);
        auto it = maxrec_cache_.find(key);
        if (it != maxrec_cache_.end()) return it->second;
        const int2 lists = max_lists(beg, end);
        int2 m = make_int2(0, 0);
        for (int v0 = beg; v0 < end; v0 += vpb) {
            const int4 r0 = vrec_[size_t(v0)], r1 = vrec_[size_t(std::min(end, v0 + vpb) - 1)];
            m.x = std::max(m.x, dev::kSlice * (r1.x + lists.x - r0.x));
            m.y = std::max(m.y, dev::kSlice * (r1.y + lists.y - r0.y));
        }
        maxrec_cache_[key] = m;
        return m;
    }

    // Shared memory of the TMA variants: `buffers` record tiles beside the staging areas.
    size_t tma_bytes(int L, int B, int beg, int end, int buffers) {
        const int2 mr = max_records(beg, end, B / L);
        return 16 + 8 * size_t(buffers) * (size_t(mr.x) + size_t(mr.y)) + stage_bytes(max_lists(beg, end).x, L, B);
    }

    template <int L>
    bool launch_solve_tma_l(int B, int beg, int end, int2 color, int flags, bool pdl) {
        if constexpr (sizeof(R) != 4) {
            return false;
        } else {
            const int vpb = B / L;
            const int2 mr = max_records(beg, end, vpb);
            const int2 lists = max_lists(beg, end);
            const size_t smem = tma_bytes(L, B, beg, end, 1);
            if (smem > kTmaSmemMax) return false;
            auto kern = cd_.enabled() ? dev::k_solve_tma<L, true, ST> : dev::k_solve_tma<L, false, ST>;
            allow_smem(kern, smem);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(div_up(end - beg, vpb));
            cfg.blockDim = dim3(B);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st_;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = pdl ? attr : nullptr;
            cfg.numAttrs = pdl ? 1 : 0;
            GAIA_CUDA(cudaLaunchKernelEx(&cfg, kern, ptrs(), c_, beg, end, color, flags, lists.x, lists.y, mr.x, mr.y));
            return true;
        }
    }

    // Double-buffered TMA pipeline on a persistent grid (FP32 compute, both tile buffers fit).
    template <int L>
    bool launch_solve_pipe_l(int B, int beg, int end, int2 color, int flags, bool pdl) {
        if constexpr (sizeof(R) != 4) {
            return false;
        } else {
            const int vpt = B / L;
            const int2 mr = max_records(beg, end, vpt);
            const int2 lists = max_lists(beg, end);
            const size_t smem = tma_bytes(L, B, beg, end, 2);
            if (smem > kTmaSmemMax) return false;
            auto kern = cd_.enabled() ? dev::k_solve_pipe<L, true, ST> : dev::k_solve_pipe<L, false, ST>;
            allow_smem(kern, smem);
            const int per_sm = blocks_per_sm(kern, B, smem);
            if (per_sm < 1) return false;
            const int ntiles = div_up(end - beg, vpt);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(unsigned(std::min(ntiles, per_sm * sm_count())));
            cfg.blockDim = dim3(B);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = st_;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = pdl ? attr : nullptr;
            cfg.numAttrs = pdl ? 1 : 0;
            GAIA_CUDA(cudaLaunchKernelEx(&cfg, kern, ptrs(), c_, beg, end, color, flags, lists.x, lists.y, mr.x, mr.y));
            return true;
        }
    }

    bool launch_solve_pipe(int L, int B, int beg, int end, int2 color, int flags, bool pdl) {
        switch (L) {
            case 2: return launch_solve_pipe_l<2>(B, beg, end, color, flags, pdl);
            case 4: return launch_solve_pipe_l<4>(B, beg, end, color, flags, pdl);
            case 8: return launch_solve_pipe_l<8>(B, beg, end, color, flags, pdl);
            case 16: return launch_solve_pipe_l<16>(B, beg, end, color, flags, pdl);
            default: return launch_solve_pipe_l<32>(B, beg, end, color, flags, pdl);
        }
    }

    // TMA-staged launch if this engine computes in FP32 and the block's records fit.
    bool launch_solve_tma(int L, int B, int beg, int end, int2 color, int flags, bool pdl) {
        switch (L) {
            case 2: return launch_solve_tma_l<2>(B, beg, end, color, flags, pdl);
            case 4: return launch_solve_tma_l<4>(B, beg, end, color, flags, pdl);
            case 8: return launch_solve_tma_l<8>(B, beg, end, color, flags, pdl);
            case 16: return launch_solve_tma_l<16>(B, beg, end, color, flags, pdl);
            default: return launch_solve_tma_l<32>(B, beg, end, color, flags, pdl);
        }
    }

    template <bool PROBE, bool DEEP>
    void launch_solve_reg(int L, int B, int beg, int end, int2 color, int flags, double* probe, bool pdl, bool prefetch) {
        B = std::min(B, 256);  // the probe of an engine whose schedule runs larger blocks
        switch (fit_lanes(L, B, beg, end)) {
            case 2: launch_solve_l<PROBE, DEEP, 2>(B, beg, end, color, flags, probe, pdl, prefetch); break;
            case 4: launch_solve_l<PROBE, DEEP, 4>(B, beg, end, color, flags, probe, pdl, prefetch); break;
            case 8: launch_solve_l<PROBE, DEEP, 8>(B, beg, end, color, flags, probe, pdl, prefetch); break;
            case 16: launch_solve_l<PROBE, false, 16>(B, beg, end, color, flags, probe, pdl, prefetch); break;
            default: launch_solve_l<PROBE, false, 32>(B, beg, end, color, flags, probe, pdl, prefetch); break;
        }
    }

    // Vertices of any list length, a warp each.
    template <bool PROBE>
    void launch_solve_wide(int B, int beg, int end, int2 color, int flags, double* probe, bool pdl) {
        B = std::min(B, 256);
        if (multi_seg_) launch_solve_l<PROBE, false, 32, true>(B, beg, end, color, flags, probe, pdl, false);
        else launch_solve_l<PROBE, false, 32>(B, beg, end, color, flags, probe, pdl, false);
    }

    // The vertices [beg, end), none of them with a long list, of a color.
    void launch_solve(int L, int B, int beg, int end, int2 color, int flags, bool pdl, int variant) {
        if (variant == 1 && launch_solve_tma(L, B, beg, end, color, flags, pdl)) return;
        if (variant == kVariantPipe && launch_solve_pipe(L, B, beg, end, color, flags, pdl)) return;
        if (variant == kVariantDeep) launch_solve_reg<false, true>(L, B, beg, end, color, flags, nullptr, pdl, false);
        else launch_solve_reg<false, false>(L, B, beg, end, color, flags, nullptr, pdl, variant == kVariantPrefetch);
    }

    // One color's solve. Its long lists take a launch of their own, unless all its vertices take a
    // warp each anyway: a launch more costs as much as a small color (about 2.5 us).
    void launch_color(size_t g, int L, int B, int flags, bool pdl, int variant) {
        const int beg = group_beg_[g], mid = group_mid_[g], end = group_end_[g];
        const int2 color = make_int2(beg, end);
        if (end <= beg) return;
        if (mid == end) {
            launch_solve(L, B, beg, end, color, flags, pdl, variant);
        } else if (mid == beg || (L == 32 && variant != 1 && variant != kVariantPipe)) {
            launch_solve_wide<false>(B, beg, end, color, flags, nullptr, pdl);
        } else {
            launch_solve(L, B, beg, mid, color, flags, pdl, variant);
            launch_solve_wide<false>(B, mid, end, color, flags, nullptr, use_pdl_);
        }
    }

    // Launch configuration of every merged color. Colors differ in size and in
    // vertex degree (on a 5-tet lattice the largest color holds the vertices with
    // 8 incident tets, the next ones those with 32), so the autotuner picks lanes
    // per vertex, block size and kernel variant per color.
    struct ColorCfg {
        int L = 4, B = 128, variant = 0;
        float ms = 0.f;
    };

    // One configuration for all colors; small colors, which cannot fill the GPU,
    // use one warp per vertex (one incidence per lane, the shortest load chain).
    void uniform_cfg(int L, int B, int variant) {
        ccfg_.assign(group_beg_.size(), ColorCfg{});
        for (size_t g = 0; g < group_beg_.size(); ++g) {
            const int n = group_end_[g] - group_beg_[g];
            ccfg_[g] = effective(g, ColorCfg{n <= small_color_ ? 32 : L, B, variant, 0.f});
        }
    }

    // The shape that a configuration of color g runs with: more lanes per vertex, or the register
    // variant, where its shared memory does not fit a block; a warp per vertex for long lists.
    ColorCfg effective(size_t g, ColorCfg c) {
        const int beg = group_beg_[g], mid = group_mid_[g];
        if (group_end_[g] <= beg) return c;
        if (mid <= beg) {
            c.L = 32;
            c.variant = 0;
            return c;
        }
        if (c.variant == 1 || c.variant == kVariantPipe) {
            if (sizeof(R) == 4 && tma_bytes(c.L, c.B, beg, mid, c.variant == 1 ? 1 : 2) <= kTmaSmemMax) return c;
            c.variant = 0;
        }
        c.L = fit_lanes(c.L, c.B, beg, mid);
        return c;
    }

    void enqueue_init(bool rebuild) {
        auto P = ptrs();
        if (frames_) {
            dev::k_frame_update<ST><<<div_up(nmesh_, 128), 128, 0, st_>>>(d_pos_.p, d_frame_ref_.p, d_frame_F_.p,
                                                                         d_frame_shift_.p, nmesh_);
            GAIA_CUDA(cudaGetLastError());
        }
        dev::k_initial_step<ST, R><<<div_up(nslots_, 256), 256, 0, st_>>>(P, c_);
        GAIA_CUDA(cudaGetLastError());
        // contacts: DCD on the start-of-substep positions, CCD on the trajectories to the
        // initial guess, before the deformers move their vertices (VBDPhysics.cpp:846-859)
        enqueue_detection(false, rebuild);
        if (!h_def_slot_.empty()) {
            dev::DeformVerts D;
            D.slot = d_def_slot_.p;
            D.def = d_def_idx_.p;
            D.a = d_def_a_.p;
            D.b = d_def_b_.p;
            D.defs = d_defs_.p;
            D.n = int32_t(h_def_slot_.size());
            dev::k_deformers<ST><<<div_up(D.n, 256), 256, 0, st_>>>(d_pos_.p, d_rest_.p, D, d_time_.p, sc_.p.dt);
            GAIA_CUDA(cudaGetLastError());
        }
        if (sc_.p.useAccelerator)
            GAIA_CUDA(cudaMemcpyAsync(d_acc_pp_.p, d_pos_.p, nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
    }

    // One iteration's color sweep: VBDPhysics.cpp:879-953 (graph of per-color kernels).
    void enqueue_iteration(int it, double* omega, bool accel) {
        int friction = it >= sc_.p.frictionStartIter ? 1 : 0;
        // intermediateCollisionDetection (VBDPhysics.cpp:878-884)
        const int ici = sc_.p.intermediateCollisionIterations;
        if (ici > 0 && it % ici == 0 && it) enqueue_detection(true, false);
        if (cd_.enabled() && (it == 0 || (ici > 0 && it % ici == 0))) enqueue_contact_snapshot(it);
        if (accel) {
            // getAcceleratorOmega (VBDPhysics.cpp:3558-3574)
            double rho = sc_.p.acceleratorRho;
            int order = it + 1;
            *omega = order == 1 ? 1.0 : (order == 2 ? 2.0 / (2.0 - rho * rho) : 4.0 / (4.0 - rho * rho * *omega));
            GAIA_CUDA(cudaMemcpyAsync(d_acc_prev_.p, d_pos_.p, nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
        }
        // programmatic launch only directly after another solve kernel in the stream (k_solve
        // reads no dynamic data before griddepcontrol.wait)
        const bool detected = cd_.enabled() && (it == 0 || (ici > 0 && it % ici == 0));
        bool after_solve = it > 0 && !accel && !detected;
        const int flags = (friction ? dev::kSolveFriction : 0) | ((it & 1) ? dev::kSolveParity : 0);
        for (size_t g = 0; g < group_beg_.size(); ++g) {
            const int n = group_end_[g] - group_beg_[g];
            if (n <= 0) continue;
            const ColorCfg& cc = ccfg_[g];
            launch_color(g, cc.L, cc.B, flags, use_pdl_ && after_solve, cc.variant);
            after_solve = true;
        }
        if (accel) {
            dev::k_accel_apply<ST><<<div_up(nactive_, 256), 256, 0, st_>>>(d_pos_.p, d_acc_pp_.p, d_acc_prev_.p, nactive_,
                                                                          *omega, cd_.records().info);
            GAIA_CUDA(cudaGetLastError());
        }
        // evaluateConvergence (VBDPhysics.cpp:948-951): a record after iterations 0, n, 2n, ...
        if (sc_.p.evaluateConvergence && it % sc_.p.evaluationSteps == 0) enqueue_conv(true);
    }

    void enqueue_velocity() {
        dev::k_velocity<ST, R><<<div_up(nslots_, 256), 256, 0, st_>>>(ptrs(), c_, d_time_.p);
        GAIA_CUDA(cudaGetLastError());
    }

    // ---- graphs -----------------------------------------------------------------
    void destroy_graphs() {
        for (auto* g : {&g_init_, &g_init_rb_, &g_sweep_, &g_vel_, &g_step_, &g_step_rb_})
            if (*g) {
                cudaGraphExecDestroy(*g);
                *g = nullptr;
            }
    }

    template <typename Fn>
    cudaGraphExec_t capture_one(Fn&& fn, int64_t* kernels = nullptr) {
        cudaGraph_t graph = nullptr;
        GAIA_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
        try {
            fn();
        } catch (...) {
            cudaStreamEndCapture(st_, &graph);
            if (graph) cudaGraphDestroy(graph);
            throw;
        }
        GAIA_CUDA(cudaStreamEndCapture(st_, &graph));
        if (kernels) {
            // kernel nodes of the captured work: the launches one replay makes
            size_t n = 0;
            GAIA_CUDA(cudaGraphGetNodes(graph, nullptr, &n));
            std::vector<cudaGraphNode_t> nodes(n);
            if (n) GAIA_CUDA(cudaGraphGetNodes(graph, nodes.data(), &n));
            int64_t k = 0;
            for (auto nd : nodes) {
                cudaGraphNodeType t;
                GAIA_CUDA(cudaGraphNodeGetType(nd, &t));
                k += t == cudaGraphNodeTypeKernel ? 1 : 0;
            }
            *kernels = k;
        }
        cudaGraphExec_t exec = nullptr;
        cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        GAIA_CUDA(e);
        return exec;
    }

    void capture() {
        destroy_graphs();
        int64_t k_init = 0, k_init_rb = 0, k_sweep = 0, k_vel = 0;
        g_init_ = capture_one([&] { enqueue_init(false); }, &k_init);
        g_init_rb_ = cd_.enabled() ? capture_one([&] { enqueue_init(true); }, &k_init_rb) : nullptr;
        g_sweep_ = capture_one([&] { enqueue_sweep(); }, &k_sweep);
        g_vel_ = capture_one([&] { enqueue_velocity(); }, &k_vel);
        // the whole substep as one graph (no gaps between the three): for untimed steps and
        // for timed steps whose sweep time is measured apart
        g_step_ = capture_one([&] {
            enqueue_init(false);
            enqueue_sweep();
            enqueue_velocity();
        });
        g_step_rb_ = cd_.enabled() ? capture_one([&] {
            enqueue_init(true);
            enqueue_sweep();
            enqueue_velocity();
        })
                                   : nullptr;
        const int64_t nsub = sc_.p.numSubsteps;
        launches_per_step_ = nsub * (k_init + k_sweep + k_vel) + (g_init_rb_ ? k_init_rb - k_init : 0);
        launches_per_substep_ = (launches_per_step_ + nsub - 1) / nsub;
    }

    // One substep's iterations (the sweep graph's content).
    void enqueue_sweep() {
        if (mode_ == kSweepScenes) {
            enqueue_scenes_sweep(scene_L_, scene_B_);
            return;
        }
        if (mode_ == kSweepCluster) {
            enqueue_cluster_sweep(scene_C_, scene_L_, scene_B_);
            return;
        }
        if (mode_ == kSweepGrid) {
            enqueue_grid_sweep(scene_L_, scene_B_);
            return;
        }
        // evaluateConvergence at iteration -1, on the initial guess (VBDPhysics.cpp:866-870)
        if (sc_.p.evaluateConvergence) enqueue_conv(true);
        double omega = 1.0;
        for (int it = 0; it < sc_.p.iterations; ++it) enqueue_iteration(it, &omega, sc_.p.useAccelerator);
    }

    // The face hierarchy of the contact detector is rebuilt at the first substep of a
    // step and refitted in the others.
    cudaGraphExec_t init_graph(int sub) const { return sub == 0 && g_init_rb_ ? g_init_rb_ : g_init_; }
    cudaGraphExec_t step_graph(int sub) const { return sub == 0 && g_step_rb_ ? g_step_rb_ : g_step_; }

    // The convergence log holds the records of the last step.
    void start_step_log() {
        if (sc_.p.evaluateConvergence) GAIA_CUDA(cudaMemsetAsync(d_conv_count_.p, 0, sizeof(int32_t), st_));
    }

    void run_steps(int n) override {
        stepped_ = true;
        for (int k = 0; k < n; ++k)
            for (int sub = 0; sub < sc_.p.numSubsteps; ++sub) {
                if (sub == 0) start_step_log();
                GAIA_CUDA(cudaGraphLaunch(step_graph(sub), st_));
            }
    }

    // Device time of n steps. Without sweep_ms the steps run as run_steps runs them (one
    // graph per substep) and are timed as a whole; with it the substep's initial step, sweep
    // and velocity update run as three graphs with events around every sweep, so that the
    // solve kernels are timed apart.
    void run_steps_timed(int n, float* total_ms, float* sweep_ms) override {
        if (!sweep_ms) {
            GAIA_CUDA(cudaEventRecord(ev_a_, st_));
            run_steps(n);
            GAIA_CUDA(cudaEventRecord(ev_b_, st_));
            GAIA_CUDA(cudaEventSynchronize(ev_b_));
            float tot = 0.f;
            GAIA_CUDA(cudaEventElapsedTime(&tot, ev_a_, ev_b_));
            if (total_ms) *total_ms = tot;
            return;
        }
        stepped_ = true;
        // per-substep sweep events: [start, end] pairs recorded around the sweep graph
        int nsub = n * sc_.p.numSubsteps;
        std::vector<cudaEvent_t> ev(2 * size_t(nsub));
        for (auto& e : ev) GAIA_CUDA(cudaEventCreate(&e));
        GAIA_CUDA(cudaEventRecord(ev_a_, st_));
        int q = 0;
        for (int k = 0; k < n; ++k)
            for (int sub = 0; sub < sc_.p.numSubsteps; ++sub, ++q) {
                if (sub == 0) start_step_log();
                GAIA_CUDA(cudaGraphLaunch(init_graph(sub), st_));
                GAIA_CUDA(cudaEventRecord(ev[2 * q], st_));
                GAIA_CUDA(cudaGraphLaunch(g_sweep_, st_));
                GAIA_CUDA(cudaEventRecord(ev[2 * q + 1], st_));
                GAIA_CUDA(cudaGraphLaunch(g_vel_, st_));
            }
        GAIA_CUDA(cudaEventRecord(ev_b_, st_));
        GAIA_CUDA(cudaEventSynchronize(ev_b_));
        float tot = 0.f, sw = 0.f;
        GAIA_CUDA(cudaEventElapsedTime(&tot, ev_a_, ev_b_));
        for (int i = 0; i < nsub; ++i) {
            float t = 0.f;
            GAIA_CUDA(cudaEventElapsedTime(&t, ev[2 * i], ev[2 * i + 1]));
            sw += t;
        }
        for (auto& e : ev) cudaEventDestroy(e);
        if (total_ms) *total_ms = tot;
        if (sweep_ms) *sweep_ms = sw;
    }

    // Time per launch of one color's solve over `reps` launches in a row.
    float time_color(size_t g, int L, int B, int variant, int reps) {
        launch_color(g, L, B, dev::kSolveFriction, false, variant);  // warm-up
        GAIA_CUDA(cudaEventRecord(ev_a_, st_));
        for (int r = 0; r < reps; ++r) launch_color(g, L, B, dev::kSolveFriction, use_pdl_, variant);
        GAIA_CUDA(cudaEventRecord(ev_b_, st_));
        GAIA_CUDA(cudaEventSynchronize(ev_b_));
        float ms = 0.f;
        GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
        return ms / reps;
    }

    // The state that solves are timed on, put back when it goes out of scope. Before the first step
    // that is the rest state with every vertex moved a little and, for the merged colors (walls):
    // the world box raised past the lowest vertices, and contact records on a few where detection
    // is on. At rest no vertex has a force, and the vertices at a wall or in contact are the ones
    // a launch waits for. Later it is the state as it stands.
    class TuneState {
    public:
        TuneState(Engine& e, bool walls) : e_(e), c_(e.c_) {
            const size_t bytes = size_t(e.nslots_) * sizeof(S4);
            save_.alloc(e.nslots_, nullptr);
            start_.alloc(e.nslots_, nullptr);
            GAIA_CUDA(cudaMemcpyAsync(save_.p, e.d_pos_.p, bytes, cudaMemcpyDeviceToDevice, e.st_));
            if (!e.stepped_) {
                dev::k_perturb<ST, R><<<div_up(e.nactive_, 256), 256, 0, e.st_>>>(e.ptrs());
                GAIA_CUDA(cudaGetLastError());
                if (walls) raise_floor();
                sampled_ = walls && e.cd_.enabled();
                if (sampled_) e.cd_.sample_records(e.st_);
            }
            GAIA_CUDA(cudaMemcpyAsync(start_.p, e.d_pos_.p, bytes, cudaMemcpyDeviceToDevice, e.st_));
        }
        ~TuneState() {
            e_.c_ = c_;
            (void)cudaMemcpyAsync(e_.d_pos_.p, save_.p, size_t(e_.nslots_) * sizeof(S4), cudaMemcpyDeviceToDevice, e_.st_);
            (void)cudaMemsetAsync(e_.d_counters_.p, 0, dev::CNT_N * sizeof(unsigned long long), e_.st_);
            if (sampled_) try {
                    e_.cd_.clear_records(e_.st_);
                } catch (...) {
                }
            (void)cudaStreamSynchronize(e_.st_);
        }
        TuneState(const TuneState&) = delete;
        TuneState& operator=(const TuneState&) = delete;
        const S4* state() const { return start_.p; }

    private:
        // The wall that gravity points to, a hundredth of the scene's height past the first vertices.
        void raise_floor() {
            if (!e_.c_.plane) return;
            int d = 0;
            for (int k = 1; k < 3; ++k)
                if (std::fabs(c_.g[k]) > std::fabs(c_.g[d])) d = k;
            auto comp = [d](const float4& x) { return d == 0 ? x.x : (d == 1 ? x.y : x.z); };
            float lo = std::numeric_limits<float>::infinity(), hi = -lo;
            for (int32_t s = 0; s < e_.nactive_; ++s) {
                lo = std::min(lo, comp(e_.h_rest_[size_t(s)]));
                hi = std::max(hi, comp(e_.h_rest_[size_t(s)]));
            }
            if (c_.g[d] > 0) {
                e_.c_.hi[d] = double(hi) - 0.01 * (double(hi) - lo);
                e_.c_.hi_f[d] = float(e_.c_.hi[d]);
            } else {
                e_.c_.lo[d] = double(lo) + 0.01 * (double(hi) - lo);
                e_.c_.lo_f[d] = float(e_.c_.lo[d]);
            }
        }
        Engine& e_;
        const dev::Consts<R> c_;
        DevBuf<S4> save_, start_;
        bool sampled_ = false;
    };

    // How much faster a shape has to be timed than one before it to take its place: more than the
    // timings of one shape differ, so that handles of a scene pick alike (lanes per vertex decide
    // the order of the sums, and so the last bits of the results).
    static constexpr float kFaster = 0.98f;

    // One substep's color launches of `iters` iterations, as the sweep's graph chains them.
    void enqueue_chain(const std::vector<ColorCfg>& cfg, int iters) {
        if (cd_.enabled()) enqueue_contact_snapshot(0);
        bool after_solve = false;
        for (int it = 0; it < iters; ++it)
            for (size_t g = 0; g < group_beg_.size(); ++g) {
                if (group_end_[g] <= group_beg_[g]) continue;
                launch_color(g, cfg[g].L, cfg[g].B, dev::kSolveFriction | ((it & 1) ? dev::kSolveParity : 0),
                             use_pdl_ && after_solve, cfg[g].variant);
                after_solve = true;
            }
    }
    // Time of one iteration of a chain, in a graph as in the step.
    float time_chain(const std::vector<ColorCfg>& cfg, int iters, const S4* save) {
        struct Exec {
            cudaGraphExec_t g = nullptr;
            ~Exec() {
                if (g) cudaGraphExecDestroy(g);
            }
        } exec;
        exec.g = capture_one([&] { enqueue_chain(cfg, iters); });
        float best = 1e30f;
        for (int r = 0; r < 3; ++r) {  // the first one warms up
            GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, save, nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
            GAIA_CUDA(cudaEventRecord(ev_a_, st_));
            GAIA_CUDA(cudaGraphLaunch(exec.g, st_));
            GAIA_CUDA(cudaEventRecord(ev_b_, st_));
            GAIA_CUDA(cudaEventSynchronize(ev_b_));
            float ms = 0.f;
            GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
            if (r) best = std::min(best, ms);
        }
        return best / float(iters);
    }

    // Autotuner: the shape (kernel variant, lanes per vertex, block size) of every color, by the
    // time of whole iterations in a graph on a state like a step's (TuneState): first one shape for
    // all colors, then, color kind by color kind, every other shape for that kind, kept where the
    // iteration gets faster. Timed by itself at rest, as it was, a color says little: a small one
    // costs its launch whatever the shape (4.7 us apart from a graph, 2 us in one), a large one finds
    // its records in the caches, and neither a wall nor a contact keeps a lane busy. Rules for what
    // that got wrong (a warp per vertex up to 1024 vertices, no two lanes with contact detection)
    // held only near the scenes they came from. 12^3 drop, double-float (432 vertices a color): a
    // frame of 320 us with 32 lanes, 295 with 16; 16^3 drop, FP32 (1024): a device step of 278 us
    // with 32, 219 with 16; 8 colliding bodies in FP64: a frame of 4800 us with 2 lanes, 3050 with
    // 8; 10^3 drop, FP32 (100): a device step of 190 us with 32, 205 with 16.
    // Fixed lanesPerVertex / blockSize / solveVariant parameters restrict the search.
    void autotune_impl() {
        if (nactive_ == 0 || group_beg_.empty()) return;
        TuneState tune(*this, true);
        // one block size in FP32 (64 and 128 threads measure the same, 256 slower)
        const std::vector<int> Bs = block_ ? std::vector<int>{block_} : (sizeof(R) == 4 ? std::vector<int>{128} : std::vector<int>{64, 128});
        // kernel variants: 0 register gathers, 4 asynchronous one-ring copies, 6 as 0 with the data of
        // the warps one resident wave ahead prefetched into L2 (FP32 compute only); 4 and 6 are 0 at
        // 16 and 32 lanes. The TMA variants 1 and 7 run on request only: with 8-byte records a
        // block's range is a few KB, and waiting for all of it costs more than the loads it saves
        // (100^3 twist, FP32, best shape: 47.3 us per color against 43.3 us for variant 0 and 41.2
        // us for 6).
        std::vector<int> variants = {0, kVariantDeep};
        if (sizeof(R) == 4) variants.push_back(kVariantPrefetch);
        if (variant_fixed_ >= 0) variants = {variant_fixed_};
        std::vector<ColorCfg> shapes;
        for (int var : variants)
            for (int L : {32, 16, 8, 4, 2}) {
                if (lanes_ && L != lanes_) continue;
                if (L >= 16 && variant_fixed_ < 0 && var != 0) continue;
                for (int B : Bs) shapes.push_back(ColorCfg{L, B, var, 0.f});
            }
        const size_t ng = group_beg_.size();
        auto same = [](const ColorCfg& a, const ColorCfg& b) { return a.L == b.L && a.B == b.B && a.variant == b.variant; };
        // colors of a kind: about as many vertices, with lists as long
        std::map<std::tuple<int, int, int>, std::vector<size_t>> kinds;
        for (size_t g = 0; g < ng; ++g) {
            const int n = group_end_[g] - group_beg_[g];
            if (n <= 0 || group_mid_[g] <= group_beg_[g]) continue;
            const int2 lists = max_lists(group_beg_[g], group_mid_[g]);
            kinds[std::make_tuple(-int(std::lround(2.0 * std::log2(double(n)))), lists.x, lists.y)].push_back(g);
        }
        int iters = 2, narrow_var = -1, narrow = 0, last_var = -1;
        float last = 0.f;
        std::vector<ColorCfg> best;
        float tbest = 1e30f;
        for (ColorCfg& c : shapes) {
            std::vector<ColorCfg> cfg(ng);
            for (size_t g = 0; g < ng; ++g) cfg[g] = effective(g, c);
            if (best.empty()) {  // enough iterations for the events' resolution, about 40 launches at most
                const float t = time_chain(cfg, iters, tune.state());
                iters = std::max(1, std::min(std::max(2, 40 / int(ng)), int(std::ceil(0.2f / t))));
            }
            // narrower groups only take longer from here on
            if (c.variant == narrow_var && c.L < narrow) continue;
            const float t = time_chain(cfg, iters, tune.state());
            if (t > 1.5f * tbest && c.variant == last_var && t > last) {
                narrow_var = c.variant;
                narrow = c.L;
            }
            last_var = c.variant;
            last = t;
            c.ms = t;
            if (t < kFaster * tbest) {
                tbest = t;
                best = cfg;
            }
        }
        // the four kinds of the largest colors; a shape that takes twice the time for all colors is
        // no better for one
        const float limit = 2.f * tbest;
        int left = 4;
        for (auto& kind : kinds) {
            if (left-- == 0) break;
            for (const ColorCfg& c : shapes) {
                if (c.ms == 0.f || c.ms > limit) continue;
                std::vector<ColorCfg> cfg = best;
                bool other = false;
                for (size_t g : kind.second) {
                    cfg[g] = effective(g, c);
                    other = other || !same(cfg[g], best[g]);
                }
                if (!other) continue;
                const float t = time_chain(cfg, iters, tune.state());
                if (t < kFaster * tbest) {
                    tbest = t;
                    best = cfg;
                }
            }
        }
        ccfg_ = best;
        // one launch of each color, as reported
        for (size_t g = 0; g < ng; ++g) {
            if (group_end_[g] <= group_beg_[g]) continue;
            ccfg_[g].ms = time_color(g, ccfg_[g].L, ccfg_[g].B, ccfg_[g].variant, 4);
        }
        tuned_ms_ = tbest;
        tuned_ = true;
    }

    // After construction or a re-tune: per-color configurations in place, and the
    // configuration of the largest color reported as the engine's.
    void finalize_cfg() {
        if (!tuned_) uniform_cfg(lanes_ ? lanes_ : 4, block_ ? block_ : 128, variant_);
        size_t big = 0;
        for (size_t g = 0; g < group_beg_.size(); ++g)
            if (group_end_[g] - group_beg_[g] > group_end_[big] - group_beg_[big]) big = g;
        if (!ccfg_.empty()) {
            lanes_ = ccfg_[big].L;
            block_ = ccfg_[big].B;
            variant_ = ccfg_[big].variant;
        }
    }

    // ---- persistent scene-major sweep (k_sweep_scenes) ------------------------------
    void setup_scenes() {
        std::vector<int64_t> work(size_t(nmesh_), 0);
        for (int m = 0; m < nmesh_; ++m)
            for (int32_t ci = scene_ofs_[m]; ci < scene_ofs_[m + 1]; ++ci)
                work[size_t(m)] += inc_ofs_[scene_colors_[ci].z] - inc_ofs_[scene_colors_[ci].x];
        std::vector<int32_t> order;
        for (int m = 0; m < nmesh_; ++m)
            if (scene_ofs_[m + 1] > scene_ofs_[m]) order.push_back(m);
        // largest scene first: the work counter hands them out in this order
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[size_t(a)] > work[size_t(b)]; });
        nscenes_ = int32_t(order.size());
        d_scene_colors_.upload(scene_colors_, &bytes_, st_);
        d_scene_ofs_.upload(scene_ofs_, &bytes_, st_);
        d_scene_order_.upload(order, &bytes_, st_);
        d_scene_work_.alloc(1, &bytes_);
        GAIA_CUDA(cudaMemsetAsync(d_scene_work_.p, 0, sizeof(int32_t), st_));
        int dev = 0;
        GAIA_CUDA(cudaGetDevice(&dev));
        GAIA_CUDA(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    template <int L, int MAXB, bool LONG>
    void launch_scenes_lb(int B) {
        auto kern = dev::k_sweep_scenes<L, LONG, ST, R, MAXB>;
        const size_t smem = sweep_stage_bytes(L, B);
        allow_smem(kern, smem);
        const int per_sm = blocks_per_sm(kern, B, smem);
        const int grid = std::max(1, std::min(nscenes_, std::max(per_sm, 1) * num_sms_));
        kern<<<grid, B, smem, st_>>>(ptrs(), c_, d_scene_colors_.p, d_scene_ofs_.p, d_scene_order_.p, nscenes_,
                                     sc_.p.iterations, sc_.p.frictionStartIter, d_scene_work_.p, sweep_stage(L));
        GAIA_CUDA(cudaGetLastError());
    }

    template <int L>
    void launch_scenes_l(int B) {
        if (B <= 256) any_long_ ? launch_scenes_lb<L, 256, true>(B) : launch_scenes_lb<L, 256, false>(B);
        else any_long_ ? launch_scenes_lb<L, 1024, true>(B) : launch_scenes_lb<L, 1024, false>(B);
    }

    // One substep's iterations: reset the work counter, one persistent launch.
    void enqueue_scenes_sweep(int L, int B) {
        if (nscenes_ == 0 || sc_.p.iterations == 0) return;
        GAIA_CUDA(cudaMemsetAsync(d_scene_work_.p, 0, sizeof(int32_t), st_));
        switch (fit_sweep_lanes(L, B)) {
            case 2: launch_scenes_l<2>(B); break;
            case 4: launch_scenes_l<4>(B); break;
            case 8: launch_scenes_l<8>(B); break;
            case 16: launch_scenes_l<16>(B); break;
            default: launch_scenes_l<32>(B); break;
        }
    }

    // Lanes per vertex and block size of the persistent sweep: every pair timed on a full
    // sweep of the current state (restored afterwards); ms per iteration of the fastest.
    void autotune_scenes() {
        if (nactive_ == 0 || nscenes_ == 0 || sc_.p.iterations == 0) return;
        TuneState tune(*this, false);
        const int Ls[] = {4, 8, 16, 32};
        const int Bs[] = {256, 512, 1024};
        float best = 1e30f;
        for (int L : Ls) {
            if (lanes_ && L != lanes_) continue;
            for (int B : Bs) {
                if (block_ && B != block_) continue;
                if (!lanes_ && fit_sweep_lanes(L, B) != L) continue;  // another candidate runs so
                float ms = 0.f;
                for (int r = 0; r < 2; ++r) {  // the first one warms up
                    GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, tune.state(), nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
                    GAIA_CUDA(cudaEventRecord(ev_a_, st_));
                    enqueue_scenes_sweep(L, B);
                    GAIA_CUDA(cudaEventRecord(ev_b_, st_));
                    GAIA_CUDA(cudaEventSynchronize(ev_b_));
                    ms = 0.f;
                    GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
                }
                if (ms < kFaster * best) {
                    best = ms;
                    scene_L_ = L;
                    scene_B_ = B;
                }
            }
        }
        tuned_ms_ = double(best) / sc_.p.iterations;
        tuned_ = true;
    }

    // ---- cluster sweep (vbd_cluster.cuh) ---------------------------------------------
    // Per scene: its active and fixed slot ranges, and how many states and records one
    // block of a C-block cluster holds; the cluster sizes whose largest block fits.
    void setup_cluster() {
        std::vector<int4> slots(size_t(nmesh_), make_int4(0, 0, 0, 0));
        int64_t f0 = nactive_;
        for (int m = 0; m < nmesh_; ++m) {
            int32_t a0 = 0, a1 = 0;
            if (scene_ofs_[m + 1] > scene_ofs_[m]) {
                a0 = scene_colors_[scene_ofs_[m]].x;
                a1 = scene_colors_[scene_ofs_[m + 1] - 1].z;
            }
            int64_t nf = 0;
            for (int v = 0; v < sc_.meshes[m].nv; ++v) nf += sc_.meshes[m].fixed[v] ? 1 : 0;
            slots[size_t(m)] = make_int4(a0, a1, int32_t(f0), int32_t(f0 + nf));
            f0 += nf;
        }
        int dev = 0;
        GAIA_CUDA(cudaGetDevice(&dev));
        int smem_optin = 0;
        GAIA_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        const size_t budget = size_t(std::max(0, smem_optin - 4096));  // static shared memory and slack
        cluster_fits_.clear();
        for (int C : {2, 4, 8, 16}) {
            int64_t pos_cap = 0, nbr_cap = 0, inc_cap = 0;
            bool ok = true;
            const std::vector<int4> rg = cluster_ranges(C);
            for (int m = 0; m < nmesh_ && ok; ++m) {
                const int4 sl = slots[size_t(m)];
                pos_cap = std::max<int64_t>(pos_cap, int64_t(sl.y - sl.x) + (sl.w - sl.z));
                if (scene_ofs_[m + 1] - scene_ofs_[m] > dev::kClusterMaxColors) ok = false;
                for (int r = 0; r < C; ++r) {
                    int64_t nbr = 0, inc = 0;
                    for (int32_t ci = scene_ofs_[m]; ci < scene_ofs_[m + 1]; ++ci) {
                        for (int kind = 0; kind < 2; ++kind) {
                            const int4 q = rg[2 * (size_t(ci) * C + r) + kind];
                            nbr += int64_t(dev::kSlice) * (q.y - q.x);
                            inc += int64_t(dev::kSlice) * (q.w - q.z);
                        }
                    }
                    nbr_cap = std::max(nbr_cap, nbr);
                    inc_cap = std::max(inc_cap, inc);
                }
            }
            nbr_cap = (nbr_cap + 1) & ~int64_t(1);
            inc_cap = (inc_cap + 1) & ~int64_t(1);
            // states, rest positions and records; the staging areas come on top (per lanes and block)
            const size_t min_stage = sweep_stage_bytes(32, kMinBlock);
            const size_t lean = sizeof(S4) * size_t(pos_cap);
            const size_t bytes = lean + sizeof(float4) * size_t(pos_cap) + sizeof(dev::NbrRec<R>) * size_t(nbr_cap) +
                                 sizeof(dev::IncRec<R>) * size_t(inc_cap);
            // The limit of the mode, the same whether it is asked for or timed by the autotuner (whose
            // pick can then be asked for): the states and 48 bytes (FP64: 96) per owned incidence in
            // each block. The records take less, at most about a third of it on a lattice, but every
            // scene within the limit is accepted: the lean form holds the states only.
            if (lean + (sizeof(R) == 8 ? 96 : 48) * size_t(cluster_incidences(C)) > budget) ok = false;
            if (ok && bytes + min_stage <= budget)
                cluster_fits_.push_back({C, int32_t(pos_cap), int32_t(nbr_cap), int32_t(inc_cap), bytes, false});
            else if (ok && lean + min_stage <= budget)
                cluster_fits_.push_back({C, int32_t(pos_cap), 0, 0, lean, true});
        }
        cluster_budget_ = budget;
        if (cluster_fits_.empty())
            throw std::runtime_error("sweepMode \"cluster\" is not supported: a scene does not fit in the shared "
                                     "memory of a 16-block cluster");
        if (sc_.p.clusterSize && !cluster_fit(sc_.p.clusterSize))
            throw std::runtime_error("sweepMode \"cluster\" is not supported with clusterSize " +
                                     std::to_string(sc_.p.clusterSize) + ": a scene does not fit in the shared "
                                     "memory of a cluster of that many blocks");
        d_scene_slots_.upload(slots, &bytes_, st_);
        std::vector<std::vector<int4>> ranges;
        for (auto& f : cluster_fits_) ranges.push_back(cluster_ranges(f.C));
        for (size_t i = 0; i < ranges.size(); ++i) {
            auto& buf = cluster_range_bufs_[cluster_fits_[i].C];
            buf.reset(new DevBuf<int4>());
            buf->upload(ranges[i], &bytes_, st_);
        }
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    // Incidences of the fullest block of a cluster of C blocks when each color's vertices are
    // dealt out evenly, in the order of the color.
    int64_t cluster_incidences(int C) const {
        int64_t most = 0;
        for (int m = 0; m < nmesh_; ++m) {
            std::vector<int64_t> per_rank(size_t(C), 0);
            for (int32_t ci = scene_ofs_[m]; ci < scene_ofs_[m + 1]; ++ci) {
                const int4 rg = scene_colors_[ci];
                const int per = (rg.z - rg.x + C - 1) / C;
                for (int r = 0; r < C; ++r) {
                    const int beg = std::min(rg.z, rg.x + r * per), end = std::min(rg.z, beg + per);
                    per_rank[size_t(r)] += deal_ofs_[size_t(end)] - deal_ofs_[size_t(beg)];
                }
            }
            for (int64_t x : per_rank) most = std::max(most, x);
        }
        return most;
    }

    // Record rows of every color's chunks (short and long lists) of every rank in a cluster of C
    // blocks (2 C per color): the chunks are whole slices, so a chunk's rows end where the next
    // slice's begin.
    std::vector<int4> cluster_ranges(int C) const {
        std::vector<int4> out;
        auto at = [&](int v) {
            if (v >= nactive_) return make_int2(nbr_end_, inc_end_);
            return make_int2(vrec_[size_t(v)].x, vrec_[size_t(v)].y);
        };
        for (const int4 c : scene_colors_)
            for (int r = 0; r < C; ++r)
                for (int kind = 0; kind < 2; ++kind) {
                    const int lo = kind ? c.y : c.x, hi = kind ? c.z : c.y;
                    const int per = dev::cluster_chunk(hi - lo, C);
                    const int beg = std::min(hi, lo + r * per), end = std::min(hi, beg + per);
                    const int2 a = at(beg), b = at(end);
                    out.push_back(beg < end ? make_int4(a.x, b.x, a.y, b.y) : make_int4(0, 0, 0, 0));
                }
        return out;
    }

    const ClusterFit* cluster_fit(int C) const {
        for (auto& f : cluster_fits_)
            if (f.C == C) return &f;
        return nullptr;
    }

    template <int L, bool LEAN = false>
    void launch_cluster_l(const ClusterFit& f, int B) {
        if (any_long_) launch_cluster_k<L, true, LEAN>(f, B);
        else launch_cluster_k<L, false, LEAN>(f, B);
    }
    template <int L, bool LONG, bool LEAN>
    void launch_cluster_k(const ClusterFit& f, int B) {
        auto kern = dev::k_sweep_cluster<L, LONG, LEAN, ST, R>;
        const size_t smem = f.bytes + sweep_stage_bytes(L, B);
        GAIA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cluster_budget_)));
        if (f.C > 8) GAIA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(f.C);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.blockDim = dim3(unsigned(B));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st_;
        cfg.gridDim = dim3(unsigned(f.C));
        int nclusters = 0;
        GAIA_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg));
        if (nclusters < 1) throw std::runtime_error("no cluster of this size fits on the device");
        cfg.gridDim = dim3(unsigned(f.C * std::min(nscenes_, nclusters)));
        dev::ClusterScenes S;
        S.colors = d_scene_colors_.p;
        S.scene_ofs = d_scene_ofs_.p;
        S.scene_order = d_scene_order_.p;
        S.scene_slots = d_scene_slots_.p;
        S.nscenes = nscenes_;
        S.iterations = sc_.p.iterations;
        S.friction_start = sc_.p.frictionStartIter;
        S.pos_cap = f.pos_cap;
        S.nbr_cap = f.nbr_cap;
        S.inc_cap = f.inc_cap;
        S.stage = sweep_stage(L);
        S.ranges = cluster_range_bufs_.at(f.C)->p;
        GAIA_CUDA(cudaLaunchKernelEx(&cfg, kern, ptrs(), c_, S, d_scene_work_.p));
    }

    // The shape that a cluster sweep of L lanes per vertex and B threads runs with: more lanes, then
    // fewer threads, where the staging areas do not fit beside the scene.
    void fit_cluster(const ClusterFit& f, int& L, int& B) const {
        auto fits = [&](int l) { return f.bytes + sweep_stage_bytes(l, B) <= cluster_budget_; };
        if (f.lean || L == 2) L = 32;  // (the kernel has no form of two lanes)
        while (L < 32 && !fits(L)) L *= 2;
        while (B > kMinBlock && !fits(L)) B = smaller_block(B);
    }

    void enqueue_cluster_sweep(int C, int L, int B) {
        if (nscenes_ == 0 || sc_.p.iterations == 0) return;
        const ClusterFit* f = cluster_fit(C);
        if (!f) throw std::runtime_error("clusterSize: scenes do not fit a cluster of " + std::to_string(C) + " blocks");
        GAIA_CUDA(cudaMemsetAsync(d_scene_work_.p, 0, sizeof(int32_t), st_));
        fit_cluster(*f, L, B);
        if (f->lean) {
            launch_cluster_l<32, true>(*f, B);
            return;
        }
        switch (L) {
            case 4: launch_cluster_l<4>(*f, B); break;
            case 8: launch_cluster_l<8>(*f, B); break;
            case 16: launch_cluster_l<16>(*f, B); break;
            default: launch_cluster_l<32>(*f, B); break;
        }
    }

    // Cluster size, lanes per vertex and block size of the cluster sweep, each combination
    // timed on a full sweep of the current state (restored afterwards).
    void autotune_cluster() {
        if (nactive_ == 0 || nscenes_ == 0 || sc_.p.iterations == 0) return;
        TuneState tune(*this, false);
        float best = 1e30f;
        for (const ClusterFit& f : cluster_fits_) {
            if (sc_.p.clusterSize && f.C != sc_.p.clusterSize) continue;
            for (int L : {4, 8, 16, 32}) {
                if (lanes_ && L != lanes_) continue;
                for (int B : {128, 256}) {
                    if (block_ && B != block_) continue;
                    int l = L, b = B;
                    fit_cluster(f, l, b);
                    if ((!lanes_ && l != L) || (!block_ && b != B && b == 128)) continue;  // another candidate runs so
                    float ms = 0.f;
                    for (int r = 0; r < 2; ++r) {  // the first one warms up
                        GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, tune.state(), nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
                        GAIA_CUDA(cudaEventRecord(ev_a_, st_));
                        enqueue_cluster_sweep(f.C, L, B);
                        GAIA_CUDA(cudaEventRecord(ev_b_, st_));
                        GAIA_CUDA(cudaEventSynchronize(ev_b_));
                        ms = 0.f;
                        GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
                    }
                    if (ms < kFaster * best) {
                        best = ms;
                        scene_C_ = f.C;
                        scene_L_ = L;
                        scene_B_ = B;
                    }
                }
            }
        }
        if (!(best < 1e30f)) throw std::runtime_error("cluster sweep: no configuration was timed");
        tuned_ms_ = double(best) / sc_.p.iterations;
        tuned_ = true;
    }

    void finalize_cluster() {
        if (!tuned_) {
            scene_C_ = sc_.p.clusterSize ? sc_.p.clusterSize : cluster_fits_.back().C;
            scene_L_ = lanes_ ? lanes_ : 8;
            scene_B_ = block_ ? block_ : 128;
        }
        if (!cluster_fit(scene_C_))
            throw std::runtime_error("clusterSize: scenes do not fit a cluster of " + std::to_string(scene_C_) + " blocks");
        fit_cluster(*cluster_fit(scene_C_), scene_L_, scene_B_);
        lanes_ = scene_L_;
        block_ = scene_B_;
        variant_ = 3;
        ccfg_.assign(sc_.groups.size(), ColorCfg{scene_L_, scene_B_, 3, float(tuned_ms_)});
    }

    // ---- grid sweep (vbd_grid.cuh) -----------------------------------------------------
    void setup_grid() {
        std::vector<int4> colors;
        for (size_t g = 0; g < group_beg_.size(); ++g)
            if (group_end_[g] > group_beg_[g]) colors.push_back(make_int4(group_beg_[g], group_mid_[g], group_end_[g], 0));
        grid_ncolors_ = int32_t(colors.size());
        grid_max_color_ = 0;
        grid_max_long_ = 0;
        for (const int4& c : colors) {
            grid_max_color_ = std::max(grid_max_color_, c.y - c.x);
            grid_max_long_ = std::max(grid_max_long_, c.z - c.y);
        }
        d_grid_colors_.upload(colors, &bytes_, st_);
        d_grid_bar_.alloc(2, &bytes_);
        int dev = 0, coop = 0;
        GAIA_CUDA(cudaGetDevice(&dev));
        GAIA_CUDA(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev));
        GAIA_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop) throw std::runtime_error("sweepMode \"grid\" is not supported: no cooperative launch on this device");
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    // Blocks of the grid sweep: enough for the largest color at one vertex per group, at most
    // as many as are resident at once (the cooperative launch requires it).
    template <int L, bool LONG>
    int grid_blocks(int B, size_t smem) {
        const int per_sm = blocks_per_sm(dev::k_sweep_grid<L, LONG, ST, R>, B, smem);
        if (per_sm < 1) throw std::runtime_error("grid sweep: no block of this size fits on an SM");
        const int need = std::max(1, int(div_up(std::max(int64_t(grid_max_color_) * L, int64_t(grid_max_long_) * 32), B)));
        return std::min(need, per_sm * num_sms_);
    }

    template <int L>
    void launch_grid_l(int B) {
        if (any_long_) launch_grid_k<L, true>(B);
        else launch_grid_k<L, false>(B);
    }
    template <int L, bool LONG>
    void launch_grid_k(int B) {
        dev::GridSweep G;
        G.colors = d_grid_colors_.p;
        G.ncolors = grid_ncolors_;
        G.iterations = sc_.p.iterations;
        G.friction_start = sc_.p.frictionStartIter;
        G.bar = d_grid_bar_.p;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const size_t smem = sweep_stage_bytes(L, B);
        allow_smem(dev::k_sweep_grid<L, LONG, ST, R>, smem);
        cfg.gridDim = dim3(unsigned(grid_blocks<L, LONG>(B, smem)));
        cfg.blockDim = dim3(unsigned(B));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st_;
        GAIA_CUDA(cudaLaunchKernelEx(&cfg, dev::k_sweep_grid<L, LONG, ST, R>, ptrs(), c_, G, sweep_stage(L)));
    }

    // One substep's iterations: the barrier's counter and flag zeroed, one cooperative launch.
    void enqueue_grid_sweep(int L, int B) {
        if (grid_ncolors_ == 0 || sc_.p.iterations == 0) return;
        GAIA_CUDA(cudaMemsetAsync(d_grid_bar_.p, 0, 2 * sizeof(uint32_t), st_));
        switch (fit_sweep_lanes(L, B)) {
            case 2: launch_grid_l<2>(B); break;
            case 4: launch_grid_l<4>(B); break;
            case 8: launch_grid_l<8>(B); break;
            case 16: launch_grid_l<16>(B); break;
            default: launch_grid_l<32>(B); break;
        }
    }

    // Lanes per vertex and block size of the grid sweep, each pair timed on a full sweep of
    // the current state (restored afterwards).
    void autotune_grid() {
        if (nactive_ == 0 || grid_ncolors_ == 0 || sc_.p.iterations == 0) return;
        TuneState tune(*this, false);
        float best = 1e30f;
        for (int L : {4, 8, 16, 32}) {
            if (lanes_ && L != lanes_) continue;
            for (int B : {128, 256}) {
                if (block_ && B != block_) continue;
                if (!lanes_ && fit_sweep_lanes(L, B) != L) continue;  // another candidate runs so
                float ms = 0.f;
                for (int r = 0; r < 2; ++r) {  // the first one warms up
                    GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, tune.state(), nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
                    GAIA_CUDA(cudaEventRecord(ev_a_, st_));
                    enqueue_grid_sweep(L, B);
                    GAIA_CUDA(cudaEventRecord(ev_b_, st_));
                    GAIA_CUDA(cudaEventSynchronize(ev_b_));
                    ms = 0.f;
                    GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
                }
                if (ms < kFaster * best) {
                    best = ms;
                    scene_L_ = L;
                    scene_B_ = B;
                }
            }
        }
        if (!(best < 1e30f)) throw std::runtime_error("grid sweep: no configuration was timed");
        tuned_ms_ = double(best) / sc_.p.iterations;
        tuned_ = true;
    }

    void finalize_grid() {
        if (!tuned_) {
            scene_L_ = lanes_ ? lanes_ : 16;
            scene_B_ = block_ ? block_ : 256;
        }
        scene_L_ = fit_sweep_lanes(scene_L_, scene_B_);
        lanes_ = scene_L_;
        block_ = scene_B_;
        variant_ = kVariantGrid;
        ccfg_.assign(sc_.groups.size(), ColorCfg{scene_L_, scene_B_, kVariantGrid, float(tuned_ms_)});
    }

    void finalize_scenes() {
        if (!tuned_) {
            scene_L_ = lanes_ ? lanes_ : 8;
            scene_B_ = block_ ? block_ : 512;
        }
        scene_L_ = fit_sweep_lanes(scene_L_, scene_B_);
        lanes_ = scene_L_;
        block_ = scene_B_;
        variant_ = 2;
        ccfg_.assign(sc_.groups.size(), ColorCfg{scene_L_, scene_B_, 2, float(tuned_ms_)});
    }

    double get_time() override {
        double t = 0.0;
        GAIA_CUDA(cudaMemcpyAsync(&t, d_time_.p, sizeof(double), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        return t;
    }
    void set_time(double t) override {
        GAIA_CUDA(cudaMemcpyAsync(d_time_.p, &t, sizeof(double), cudaMemcpyHostToDevice, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    void reset() override {
        GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, h_pos_.data(), nslots_ * sizeof(S4), cudaMemcpyHostToDevice, st_));
        GAIA_CUDA(cudaMemcpyAsync(d_vel_.p, h_vel_.data(), nslots_ * sizeof(V4), cudaMemcpyHostToDevice, st_));
        GAIA_CUDA(cudaMemcpyAsync(d_y_.p, h_pos_.data(), nslots_ * sizeof(S4), cudaMemcpyHostToDevice, st_));
        GAIA_CUDA(cudaMemcpyAsync(d_xprev_.p, h_pos_.data(), nslots_ * sizeof(S4), cudaMemcpyHostToDevice, st_));
        GAIA_CUDA(cudaMemsetAsync(d_time_.p, 0, sizeof(double), st_));
        // the status counters (non-finite solves, device timeouts) start again from zero
        GAIA_CUDA(cudaMemsetAsync(d_counters_.p + dev::CNT_NONFINITE, 0, 3 * sizeof(unsigned long long), st_));
        cd_.reset(st_);
        GAIA_CUDA(cudaStreamSynchronize(st_));
        reset_frames();
        stepped_ = false;
    }

    void autotune() override {
        lanes_ = sc_.p.lanesPerVertex;
        block_ = sc_.p.blockSize;
        tuned_ = false;
        if (mode_ == kSweepScenes) {
            autotune_scenes();
            finalize_scenes();
        } else if (mode_ == kSweepCluster) {
            autotune_cluster();
            finalize_cluster();
        } else if (mode_ == kSweepGrid) {
            autotune_grid();
            finalize_grid();
        } else {
            autotune_impl();
            finalize_cfg();
        }
        capture();
    }

    double tuned_ms() const override { return tuned_ms_; }

    // Device time of the captured sweep graph (all iterations of one substep) on the state of
    // the autotuners, per iteration; the state is restored afterwards.
    double measure_sweep_ms() override {
        TuneState tune(*this, false);
        GAIA_CUDA(cudaGraphLaunch(g_sweep_, st_));  // warm-up
        const int reps = 3;
        float total = 0.f;
        for (int r = 0; r < reps; ++r) {
            GAIA_CUDA(cudaMemcpyAsync(d_pos_.p, tune.state(), nslots_ * sizeof(S4), cudaMemcpyDeviceToDevice, st_));
            GAIA_CUDA(cudaEventRecord(ev_a_, st_));
            GAIA_CUDA(cudaGraphLaunch(g_sweep_, st_));
            GAIA_CUDA(cudaEventRecord(ev_b_, st_));
            GAIA_CUDA(cudaEventSynchronize(ev_b_));
            float ms = 0.f;
            GAIA_CUDA(cudaEventElapsedTime(&ms, ev_a_, ev_b_));
            total += ms;
        }
        return double(total) / reps / std::max(sc_.p.iterations, 1);
    }

    // ---- state access -------------------------------------------------------------
    // Status of the device work so far: a bounded wait that ran out, then non-finite solves.
    // Each is reported once: the call that throws moves the device counts into the handle's
    // totals (stats) and clears them, so the calls after it see the state as it was left.
    void check_nonfinite() {
        unsigned long long h[dev::CNT_N];
        GAIA_CUDA(cudaMemcpyAsync(h, d_counters_.p, sizeof(h), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        if (!h[dev::CNT_TIMEOUT] && !h[dev::CNT_NONFINITE]) return;
        reported_timeouts_ += int64_t(h[dev::CNT_TIMEOUT]);
        reported_nonfinite_ += int64_t(h[dev::CNT_NONFINITE]);
        GAIA_CUDA(cudaMemsetAsync(d_counters_.p + dev::CNT_NONFINITE, 0, 3 * sizeof(unsigned long long), st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        if (h[dev::CNT_TIMEOUT])
            throw DeviceTimeout(std::to_string(h[dev::CNT_TIMEOUT]) +
                                " solve block(s) gave up on a bounded device wait and skipped their vertices" +
                                (h[dev::CNT_DRAIN] ? " (" + std::to_string(h[dev::CNT_DRAIN]) +
                                                         " still had copies in flight)"
                                                   : std::string()));
        if (h[dev::CNT_NONFINITE])
            throw std::domain_error(std::to_string(h[dev::CNT_NONFINITE]) +
                                    " vertex solve(s) met a non-finite force or step (not written)");
    }

    void sync() override {
        GAIA_CUDA(cudaStreamSynchronize(st_));
        check_nonfinite();
    }

    void mesh_range(int mesh, int64_t& off, int64_t& n) {
        if (mesh < 0 || mesh >= nmesh_) throw std::invalid_argument("mesh index out of range");
        off = mesh_off_[mesh];
        n = mesh_off_[mesh + 1] - off;
    }

    void get_positions(int mesh, double* out) override {
        check_nonfinite();
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (n == 0) return;
        dev::k_gather_positions<ST><<<div_up(n, 256), 256, 0, st_>>>(d_pos_.p, d_rest_.p, nullptr, d_stage_f64_.p,
                                                                     d_slot_of_.p + off, int32_t(n), frame_ptr(),
                                                                     d_slot_mesh_.p);
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaMemcpyAsync(out, d_stage_f64_.p, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }
    void get_velocities(int mesh, double* out) override {
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (n == 0) return;
        dev::k_gather_velocities<V4><<<div_up(n, 256), 256, 0, st_>>>(d_vel_.p, nullptr, d_stage_f64_.p,
                                                                      d_slot_of_.p + off, int32_t(n));
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaMemcpyAsync(out, d_stage_f64_.p, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }
    void set_positions(int mesh, const double* in) override {
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (n == 0) return;
        GAIA_CUDA(cudaMemcpyAsync(d_stage_f64_.p, in, 3 * n * sizeof(double), cudaMemcpyHostToDevice, st_));
        dev::k_scatter_positions_f64<ST><<<div_up(n, 256), 256, 0, st_>>>(d_pos_.p, d_rest_.p, d_stage_f64_.p,
                                                                          d_slot_of_.p + off, int32_t(n), frame_ptr(),
                                                                          d_slot_mesh_.p);
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }
    void set_prev_positions(int mesh, const double* in) override {
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (n == 0) return;
        GAIA_CUDA(cudaMemcpyAsync(d_stage_f64_.p, in, 3 * n * sizeof(double), cudaMemcpyHostToDevice, st_));
        dev::k_scatter_positions_f64<ST><<<div_up(n, 256), 256, 0, st_>>>(d_xprev_.p, d_rest_.p, d_stage_f64_.p,
                                                                          d_slot_of_.p + off, int32_t(n), frame_ptr(),
                                                                          d_slot_mesh_.p);
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    // A substep-start detection pass on the current positions (trajectories from the
    // start-of-substep positions); returns the number of vertices with a contact.
    int collide() override {
        if (!cd_.enabled()) return 0;
        stepped_ = true;
        enqueue_detection(false, true);
        std::vector<int32_t> rows;
        cd_.contacts(rows, st_);
        return int(rows.size() / 3);
    }

    // Rows of 8: mesh, vertex, face mesh, face vertices (3, mesh-local), surface face
    // (mesh-local), kind (1 = CCD, 2 = DCD), in (mesh, surface vertex) order.
    void contacts(std::vector<int32_t>& out) override {
        out.clear();
        if (!cd_.enabled()) return;
        std::vector<int32_t> rows;
        cd_.contacts(rows, st_);
        std::vector<int32_t> face_ofs(nmesh_ + 1, 0);
        for (int m = 0; m < nmesh_; ++m) face_ofs[m + 1] = face_ofs[m] + int32_t(sc_.meshes[m].sfaces.size() / 3);
        for (size_t r = 0; r + 2 < rows.size(); r += 3) {
            const int32_t gi = orig_of_[rows[r]];
            const int m = int(std::upper_bound(mesh_off_.begin(), mesh_off_.end(), int64_t(gi)) - mesh_off_.begin()) - 1;
            const int32_t g = rows[r + 1];
            const int fm = int(std::upper_bound(face_ofs.begin(), face_ofs.end(), g) - face_ofs.begin()) - 1;
            const int32_t f = g - face_ofs[fm];
            const int32_t* fv = &sc_.meshes[fm].sfaces[3 * size_t(f)];
            const int32_t row[8] = {m, gi - int32_t(mesh_off_[m]), fm, fv[0], fv[1], fv[2], f, rows[r + 2]};
            out.insert(out.end(), row, row + 8);
        }
    }

    void set_velocities(int mesh, const double* in) override {
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (n == 0) return;
        GAIA_CUDA(cudaMemcpyAsync(d_stage_f64_.p, in, 3 * n * sizeof(double), cudaMemcpyHostToDevice, st_));
        dev::k_scatter_velocities_f64<ST><<<div_up(n, 256), 256, 0, st_>>>(d_vel_.p, d_stage_f64_.p,
                                                                           d_slot_of_.p + off, int32_t(n));
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    void set_state_f32(const float* x, const float* v) override {
        float* dx = d_stage_f32_.p;
        float* dv = d_stage_f32_.p + 3 * size_t(nslots_);
        if (x) GAIA_CUDA(cudaMemcpyAsync(dx, x, 3 * nslots_ * sizeof(float), cudaMemcpyHostToDevice, st_));
        if (v) GAIA_CUDA(cudaMemcpyAsync(dv, v, 3 * nslots_ * sizeof(float), cudaMemcpyHostToDevice, st_));
        dev::k_scatter_state<ST><<<div_up(nslots_, 256), 256, 0, st_>>>(d_pos_.p, d_rest_.p, d_vel_.p, x ? dx : nullptr,
                                                                       v ? dv : nullptr, d_slot_of_.p,
                                                                       int32_t(nslots_), frame_ptr(), d_slot_mesh_.p);
        GAIA_CUDA(cudaGetLastError());
    }

    void get_positions_f32(float* x) override {
        dev::k_gather_positions<ST><<<div_up(nslots_, 256), 256, 0, st_>>>(d_pos_.p, d_rest_.p, d_stage_f32_.p,
                                                                          nullptr, d_slot_of_.p, int32_t(nslots_),
                                                                          frame_ptr(), d_slot_mesh_.p);
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaMemcpyAsync(x, d_stage_f32_.p, 3 * nslots_ * sizeof(float), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        check_nonfinite();
    }
    void get_velocities_f32(float* v) override {
        dev::k_gather_velocities<V4><<<div_up(nslots_, 256), 256, 0, st_>>>(d_vel_.p, d_stage_f32_.p, nullptr,
                                                                            d_slot_of_.p, int32_t(nslots_));
        GAIA_CUDA(cudaGetLastError());
        GAIA_CUDA(cudaMemcpyAsync(v, d_stage_f32_.p, 3 * nslots_ * sizeof(float), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    // ---- FP64 convergence reduction (vbd_convergence.cuh) -----------------------------
    // Per-tet FP64 data (global tet order: meshes in order, tets in order), each active
    // slot's incidences as (tet, order) in the solve's CSR, partial-sum buffers and the
    // record log; built on first use, or at construction when the step logs records.
    void setup_conv() {
        if (conv_ready_) return;
        std::vector<int4> ts;
        std::vector<double> dm, vol;
        std::vector<int32_t> tm, tet_off(nmesh_ + 1, 0);
        for (int m = 0; m < nmesh_; ++m) {
            const TetMesh& M = sc_.meshes[m];
            tet_off[m + 1] = tet_off[m] + M.ntet;
            for (int t = 0; t < M.ntet; ++t) {
                const int32_t* tv = &M.tets[4 * size_t(t)];
                ts.push_back(make_int4(slot_of_[mesh_off_[m] + tv[0]], slot_of_[mesh_off_[m] + tv[1]],
                                       slot_of_[mesh_off_[m] + tv[2]], slot_of_[mesh_off_[m] + tv[3]]));
                dm.insert(dm.end(), M.dminv.begin() + 9 * size_t(t), M.dminv.begin() + 9 * size_t(t) + 9);
                vol.push_back(M.vol[t]);
                tm.push_back(m);
            }
        }
        // incidences in slot order, as the solve's records are stored
        std::vector<int32_t> inc_tet;
        std::vector<int8_t> inc_ord;
        inc_tet.reserve(size_t(ninc_));
        inc_ord.reserve(size_t(ninc_));
        for (int32_t sl = 0; sl < nactive_; ++sl) {
            const int m = slot_mesh_[sl];
            const TetMesh& M = sc_.meshes[m];
            const int v = orig_of_[sl] - int32_t(mesh_off_[m]);
            const int32_t base = tet_off[m];
            for (int k = M.nbr_ofs[v]; k < M.nbr_ofs[v + 1]; ++k) {
                inc_tet.push_back(base + M.nbr_tet[k]);
                inc_ord.push_back(static_cast<int8_t>(M.nbr_order[k]));
            }
        }
        std::vector<double4> mat(nmesh_);
        for (int m = 0; m < nmesh_; ++m) {
            const ObjectParams& o = sc_.objs[m];
            mat[m] = make_double4(o.miu, o.lmbd, o.dampingHydrostatic, o.dampingDeviatoric);
        }
        std::vector<double> mass(size_t(nslots_), 0.0);
        for (int m = 0; m < nmesh_; ++m)
            for (int v = 0; v < sc_.meshes[m].nv; ++v) mass[size_t(slot_of_[mesh_off_[m] + v])] = sc_.meshes[m].mass[v];
        d_tet_slots_.upload(ts, &bytes_, st_);
        d_tet_dminv_.upload(dm, &bytes_, st_);
        d_tet_vol_.upload(vol, &bytes_, st_);
        d_tet_mesh_.upload(tm, &bytes_, st_);
        d_conv_inc_tet_.upload(inc_tet, &bytes_, st_);
        d_conv_inc_ord_.upload(inc_ord, &bytes_, st_);
        d_conv_mat_.upload(mat, &bytes_, st_);
        d_conv_mass_.upload(mass, &bytes_, st_);
        conv_nb_t_ = std::max(1, div_up(int64_t(ts.size()), dev::kConvThreads));
        conv_nb_v_ = std::max(1, div_up(nslots_, dev::kConvThreads));
        d_conv_part_.alloc(size_t(conv_nb_t_) + 2 * size_t(conv_nb_v_), &bytes_);
        d_conv_out_.alloc(4, &bytes_);
        conv_per_substep_ = 1 + (sc_.p.iterations + sc_.p.evaluationSteps - 1) / sc_.p.evaluationSteps;
        if (sc_.p.iterations == 0) conv_per_substep_ = 1;
        conv_cap_ = sc_.p.evaluateConvergence ? conv_per_substep_ * sc_.p.numSubsteps : 0;
        d_conv_log_.alloc(4 * size_t(std::max(conv_cap_, 1)), &bytes_);
        d_conv_count_.alloc(1, &bytes_);
        GAIA_CUDA(cudaMemsetAsync(d_conv_count_.p, 0, sizeof(int32_t), st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        conv_ready_ = true;
    }

    dev::ConvData conv_data() const {
        dev::ConvData D;
        D.tet_slots = d_tet_slots_.p;
        D.tet_dminv = d_tet_dminv_.p;
        D.tet_vol = d_tet_vol_.p;
        D.tet_mesh = d_tet_mesh_.p;
        D.mesh_mat = d_conv_mat_.p;
        D.slot_mesh = d_slot_mesh_.p;
        D.slot_mass = d_conv_mass_.p;
        D.inc_ofs = d_inc_ofs_.p;
        D.inc_tet = d_conv_inc_tet_.p;
        D.inc_ord = d_conv_inc_ord_.p;
        D.ntet = int32_t(d_tet_slots_.n);
        D.nactive = nactive_;
        D.nslots = int32_t(nslots_);
        D.dt2inv = sc_.p.dtSqrReciprocal;
        D.inv_dt = 1.0 / sc_.p.dt;
        return D;
    }

    // Three kernels: elastic partials, inertia / force-norm partials, the fixed-order finish
    // into the log (to_log) or into the single-record output.
    void enqueue_conv(bool to_log) {
        const dev::ConvData D = conv_data();
        double* pe = d_conv_part_.p;
        double* pi = pe + conv_nb_t_;
        double* pf = pi + conv_nb_v_;
        if (D.ntet) dev::k_conv_tets<ST><<<conv_nb_t_, dev::kConvThreads, 0, st_>>>(d_pos_.p, d_rest_.p, D, pe);
        else GAIA_CUDA(cudaMemsetAsync(pe, 0, sizeof(double), st_));
        dev::k_conv_verts<ST><<<conv_nb_v_, dev::kConvThreads, 0, st_>>>(d_pos_.p, d_y_.p, d_xprev_.p, d_rest_.p, D, pi,
                                                                         pf);
        dev::k_conv_finish<<<1, dev::kConvThreads, 0, st_>>>(pe, D.ntet ? conv_nb_t_ : 1, pi, pf, conv_nb_v_,
                                                             1.0 / double(std::max<int64_t>(nslots_, 1)),
                                                             to_log ? d_conv_log_.p : d_conv_out_.p,
                                                             to_log ? d_conv_count_.p : nullptr,
                                                             to_log ? conv_cap_ : 1);
        GAIA_CUDA(cudaGetLastError());
    }

    // evaluateConvergenceGPU on the current state: energy, inertia, elastic, average force norm.
    void convergence(double* out4) override {
        setup_conv();
        enqueue_conv(false);
        GAIA_CUDA(cudaMemcpyAsync(out4, d_conv_out_.p, 4 * sizeof(double), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
    }

    double energy() override {
        double out[4];
        convergence(out);
        return out[0];
    }

    // Records of the last step: (substep, iteration, energy, inertia, elastic, average force norm).
    void convergence_log(std::vector<double>& rows) override {
        rows.clear();
        if (!sc_.p.evaluateConvergence) return;
        int32_t n = 0;
        GAIA_CUDA(cudaMemcpyAsync(&n, d_conv_count_.p, sizeof(int32_t), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        n = std::min(n, conv_cap_);
        std::vector<double> log(4 * size_t(std::max(n, 1)));
        if (n) GAIA_CUDA(cudaMemcpyAsync(log.data(), d_conv_log_.p, 4 * size_t(n) * sizeof(double),
                                         cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        for (int k = 0; k < n; ++k) {
            const int sub = k / conv_per_substep_, e = k % conv_per_substep_;
            rows.push_back(double(sub));
            rows.push_back(e == 0 ? -1.0 : double((e - 1) * sc_.p.evaluationSteps));
            rows.insert(rows.end(), log.begin() + 4 * size_t(k), log.begin() + 4 * size_t(k) + 4);
        }
    }

    void vertex_force_hessian(int mesh, int v, int friction, double* f3, double* h9) override {
        int64_t off, n;
        mesh_range(mesh, off, n);
        if (v < 0 || v >= n) throw std::invalid_argument("vertex index out of range");
        int32_t s = slot_of_[off + v];
        if (s >= nactive_) throw std::invalid_argument("vertex is fixed (not solved)");
        if (cd_.enabled()) enqueue_contact_snapshot(0);
        const int flags = friction ? dev::kSolveFriction : 0;
        const int2 own = make_int2(s, s + 1);
        if (long_slot(s)) launch_solve_wide<true>(block_, s, s + 1, own, flags, d_probe_.p, false);
        else launch_solve_reg<true, false>(lanes_, block_, s, s + 1, own, flags, d_probe_.p, false, false);
        double h[12];
        GAIA_CUDA(cudaMemcpyAsync(h, d_probe_.p, sizeof(h), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        for (int i = 0; i < 3; ++i) f3[i] = h[i];
        for (int i = 0; i < 9; ++i) h9[i] = h[3 + i];
    }

    void stats(gaia_vbd_stats* s) override {
        unsigned long long h[dev::CNT_N];
        GAIA_CUDA(cudaMemcpyAsync(h, d_counters_.p, sizeof(h), cudaMemcpyDeviceToHost, st_));
        GAIA_CUDA(cudaStreamSynchronize(st_));
        s->precision = ST::kCode;
        s->lanes_per_vertex = lanes_;
        s->block_size = block_;
        s->num_groups = int32_t(sc_.groups.size());
        s->sweep_mode = mode_;
        s->cluster_size = mode_ == kSweepCluster ? scene_C_ : 0;
        s->num_vertices = nslots_;
        s->num_active_vertices = nactive_;
        s->num_incidences = ninc_;
        s->kernel_launches_per_step = launches_per_step_;
        s->fp64_fallback_solves = int64_t(h[dev::CNT_FP64_SOLVES]);
        s->failed_solves = int64_t(h[dev::CNT_FAILED_SOLVES]);
        s->device_bytes = int64_t(bytes_);
        s->autotune_ms_per_iteration = tuned_ms_;
        s->solve_variant = variant_;
        s->mesh_frames = frames_ ? 1 : 0;
        unsigned long long cc[cloth::CC_N];
        cd_.counters(cc, st_);
        s->contact_detections = int64_t(cc[cloth::CC_DETECTIONS]);
        s->contact_stack_overflow = int64_t(cc[cloth::CC_STACK_OVERFLOW]);
        s->contact_traverse_bounds = int64_t(cc[cloth::CC_TRUNCATIONS]);
        s->device_timeouts = reported_timeouts_ + int64_t(h[dev::CNT_TIMEOUT]);
        s->nonfinite_solves = reported_nonfinite_ + int64_t(h[dev::CNT_NONFINITE]);
    }

private:
    const Scene& sc_;
    cudaStream_t st_ = nullptr;
    cudaEvent_t ev_a_ = nullptr, ev_b_ = nullptr, ev_c_ = nullptr;
    cudaGraphExec_t g_init_ = nullptr, g_init_rb_ = nullptr, g_sweep_ = nullptr, g_vel_ = nullptr;
    cudaGraphExec_t g_step_ = nullptr, g_step_rb_ = nullptr;  // init + sweep + velocity of one substep
    tetcd::Detector cd_;
    DevBuf<float4> d_xf_;
    DevBuf<double2> d_mesh_fric_;
    DevBuf<S4> d_snap_;
    int nmesh_ = 0;
    int64_t nslots_ = 0;
    int32_t nactive_ = 0, ninc_ = 0;
    int lanes_ = 0, block_ = 0;
    std::vector<ColorCfg> ccfg_;
    bool tuned_ = false;
    bool stepped_ = false;  // a step or a detection ran since the start or the last reset
    bool use_pdl_ = true;
    int small_color_ = 16384;
    int variant_ = 0;          // 0 = register-pipelined k_solve, 1 = TMA-staged k_solve_tma, 2 = k_sweep_scenes,
                               // 3 = k_sweep_cluster, 4 = k_solve with DEEP, 5 = k_sweep_grid, 6 = k_solve with L2
                               // prefetch of the next wave's records, 7 = k_solve_pipe
    int mode_ = 0;             // kSweepMerged, kSweepScenes, kSweepCluster or kSweepGrid
    // scene-major mode: per mesh its color slot ranges, in sweep order
    std::vector<int64_t> deal_ofs_;   // incidences before each vertex, in the order of the colors
    std::vector<int4> scene_colors_;  // first slot, first of the long lists, end
    std::vector<int32_t> scene_ofs_;
    int32_t nscenes_ = 0;
    int scene_L_ = 8, scene_B_ = 512, scene_C_ = 8, num_sms_ = 1;
    DevBuf<int4> d_scene_colors_;
    DevBuf<int32_t> d_scene_ofs_, d_scene_order_, d_scene_work_;
    std::vector<ClusterFit> cluster_fits_;
    size_t cluster_budget_ = 0;  // dynamic shared memory of a cluster's block
    std::map<int, std::unique_ptr<DevBuf<int4>>> cluster_range_bufs_;
    DevBuf<int4> d_scene_slots_;
    // grid mode: the merged colors' slot ranges, the barrier's counter and abort flag
    DevBuf<int4> d_grid_colors_;
    // mesh frames: per mesh the reference slot, the FP64 offset, this substep's shift, the planes
    bool frames_ = false;
    DevBuf<int32_t> d_frame_ref_;
    DevBuf<double4> d_frame_F_;
    DevBuf<float4> d_frame_shift_;
    DevBuf<float4> d_rest_fh_, d_rest_fl_;
    DevBuf<uint32_t> d_grid_bar_;
    int32_t grid_ncolors_ = 0, grid_max_color_ = 0, grid_max_long_ = 0;
    int variant_fixed_ = -1;   // from PhysicsParams solveVariant (-1 = autotune)
    std::map<std::pair<int, int>, int2> maxrec_cache_;
    std::map<std::tuple<const void*, int, size_t>, int> occ_cache_;  // (kernel, block, shared bytes) -> blocks per SM
    int sms_ = 0;
    static constexpr size_t kTmaSmemMax = 200 * 1024;
    static constexpr int kContactBlocks = 64;
    double tuned_ms_ = 0.0;
    int64_t launches_per_substep_ = 0, launches_per_step_ = 0;
    int64_t reported_timeouts_ = 0, reported_nonfinite_ = 0;  // status counts already reported
    size_t bytes_ = 0;
    dev::Consts<R> c_{};
    std::vector<int64_t> mesh_off_;
    std::vector<int32_t> slot_of_, orig_of_, slot_mesh_, inc_ofs_, group_beg_, group_mid_, group_end_;
    std::vector<std::vector<uint8_t>> long_;  // per mesh (empty: none) its vertices with long lists
    bool any_long_ = false;
    // one-ring and incidence records
    std::vector<dev::NbrRec<R>> h_nbr_;
    std::vector<dev::IncRec<R>> h_inc_;
    std::vector<int4> vrec_, segs_;
    std::vector<int2> vmore_;
    bool multi_seg_ = false;  // some vertex has more than kSegNbrs neighbours
    int max_nbr_all_ = 2, max_nbr_short_ = 2, max_inc_all_ = 1, nbr_end_ = 0, inc_end_ = 0;
    std::map<std::pair<int, int>, int2> lists_cache_;
    std::vector<S4> h_pos_;
    std::vector<V4> h_vel_;
    std::vector<float4> h_rest_;
    std::vector<dev::MeshMat<R>> h_mats_;
    std::vector<dev::DeformerDev> h_defs_;
    std::vector<int32_t> h_def_slot_, h_def_idx_;
    std::vector<double> h_def_a_, h_def_b_;
    DevBuf<S4> d_pos_, d_y_, d_xprev_, d_acc_pp_, d_acc_prev_;
    DevBuf<V4> d_vel_, d_vprev_;
    DevBuf<int32_t> d_inc_ofs_, d_slot_mesh_, d_slot_of_, d_def_slot_, d_def_idx_, d_tet_mesh_;
    DevBuf<int4> d_tet_slots_;
    DevBuf<int4> d_vrec_, d_segs_;
    DevBuf<int2> d_vmore_;
    DevBuf<dev::NbrRec<R>> d_nbr_;
    DevBuf<dev::IncRec<R>> d_inc_;
    DevBuf<dev::MeshMat<R>> d_mats_;
    DevBuf<unsigned long long> d_counters_;
    DevBuf<double> d_time_, d_def_a_, d_def_b_, d_stage_f64_, d_probe_, d_tet_dminv_, d_tet_vol_;
    // convergence reduction
    bool conv_ready_ = false;
    int conv_nb_t_ = 1, conv_nb_v_ = 1, conv_per_substep_ = 1, conv_cap_ = 0;
    DevBuf<int32_t> d_conv_inc_tet_, d_conv_count_;
    DevBuf<int8_t> d_conv_inc_ord_;
    DevBuf<double4> d_conv_mat_;
    DevBuf<double> d_conv_part_, d_conv_out_, d_conv_log_, d_conv_mass_;
    DevBuf<dev::DeformerDev> d_defs_;
    DevBuf<float4> d_rest_;
    DevBuf<float> d_stage_f32_;
};

// The engine of each precision mode, built in its own translation unit.
EngineBase* make_engine_f32(const Scene& s, int mode);
EngineBase* make_engine_df(const Scene& s, int mode);
EngineBase* make_engine_dfh(const Scene& s, int mode);
EngineBase* make_engine_f64(const Scene& s, int mode);

}  // namespace gaia

