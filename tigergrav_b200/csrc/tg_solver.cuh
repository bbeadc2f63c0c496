/*
 * tg_solver.cuh -- host-side solver state and the internal entry points the
 * C ABI (tg_capi.cu) drives.  Device data layout (all in particle/node order
 * after the Morton sort; "sorted order"):
 *
 *   particles  pos[n]   int4   (x, y, z fixed point, w = caller index)
 *              vel[n]   float4 (vx, vy, vz, 0)
 *              acc[n]   float4 (phi, gx, gy, gz)      FP32 path
 *              accd[n]  double4-like 4 doubles        FP64 path
 *   nodes      level order, increasing box id within a level
 *              nd_pb/pe  int32 particle range
 *              nd_child0 int32 (-1 leaf), nd_parent int32, nd_key u64 (Morton prefix << (63-level))
 *              nd_ms[n]  tg_msrc: 17 multipole floats + com int32[3] (80 B, the reference's multi_src)
 *              nd_r, nd_rmax float, nd_cnt int32, nd_level uint8
 *              nd_aabb  6 int32 (particle AABB, fixed point), nd_prange 6 double
 *              nd_L     35 doubles (local expansion after L2L)
 *   lists      per kind k: nd_loff[k][node] (int64), nd_llen[k][node] (int32) into pool[k]
 */
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/tigergrav_b200.h"
#include "tg_common.cuh"

#define TG_CUDA(call)                                                                          \
    do {                                                                                       \
        cudaError_t _e = (call);                                                               \
        if (_e != cudaSuccess) {                                                               \
            tg::set_last_cuda_error(_e, #call, __FILE__, __LINE__);                            \
            return TG_ERR_CUDA;                                                                \
        }                                                                                      \
    } while (0)

#define TG_TRY(call)                                                                           \
    do {                                                                                       \
        int _s = (call);                                                                       \
        if (_s != TG_OK) return _s;                                                            \
    } while (0)

namespace tg {

void set_last_cuda_error(cudaError_t e, const char *what, const char *file, int line);

struct __align__(16) MSrc {
    float m[MP];
    int32_t x[3];
};
static_assert(sizeof(MSrc) == 80, "multi_src layout");

/* a node as a check item, one 32-byte sector: COM x, y, z and r (float bits);
 * child0, or NODE_EMPTY for a node without particles */
struct __align__(32) WalkRec {
    int4 x, kind;
};

template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0; /* capacity in elements */
};

constexpr int NLIST = 8;

/* Bytes of each of the two scratch areas of the leaf Ewald sums, the chunks of one
 * batch of leaves and the source leaves' sums (tg_ewald_leaf.cuh): EW_SCRATCH, or
 * EW_SCRATCH_N per particle where that is more.  The source leaves' sums take 9 KB
 * per leaf in FP32, 256 B per particle at 36 particles a leaf; 256^3 at theta 0.19
 * (2.1 GB of them) runs in one batch like smaller boxes, where 1 GiB gave two batches
 * and two ranges of vectors and 4 ms of 878 more. */
constexpr size_t EW_SCRATCH = 1ull << 30, EW_SCRATCH_N = 256;

struct Solver {
    tg_params prm{};
    int dev = 0;
    int64_t n = 0;
    bool have_tree = false, have_multipoles = false, have_lists = false, have_forces = false;

    /* particles */
    DevBuf<int4> pos, pos_alt;
    DevBuf<float4> vel, vel_alt;
    DevBuf<float4> acc;
    DevBuf<double> accd; /* FP64 path: 4 per particle */
    DevBuf<unsigned long long> keys, keys_alt;
    DevBuf<int32_t> idx, idx_alt;
    DevBuf<unsigned char> cub_tmp;

    /* nodes */
    int64_t nnodes = 0;
    std::vector<int64_t> level_off;    /* host: first node of each level, size depth+2 */
    std::vector<int64_t> level_leaves; /* host: leaves (childless nodes) of each level, size depth+1 */
    int depth = 0;
    DevBuf<int32_t> nd_pb, nd_pe, nd_child0, nd_parent;
    DevBuf<long long> tb_out; /* the tree build's level table and status */
    DevBuf<int32_t> tb_flag, tb_scan; /* a wide level's nodes to split, and their exclusive scan */
    DevBuf<unsigned long long> nd_key;
    DevBuf<unsigned char> nd_level;
    DevBuf<MSrc> nd_ms;
    DevBuf<float> nd_r, nd_rmax;
    DevBuf<int32_t> nd_aabb;   /* 6 per node: min xyz, max xyz (fixed point) */
    DevBuf<double> nd_prange;  /* 6 per node: min xyz, max xyz */
    DevBuf<double> nd_L;       /* 35 per node */
    DevBuf<double> nd_Lloc;    /* 35 per node: CC/CP contributions */

    /* walk */
    DevBuf<int64_t> loff[NLIST];
    DevBuf<int32_t> llen[NLIST];
    DevBuf<int32_t> pool[NLIST];
    DevBuf<unsigned long long> pool_top; /* NLIST + 2 counters */
    DevBuf<int64_t> nxt_off[2];          /* per node: offset of next list (direct, ewald) */
    DevBuf<int32_t> nxt_len[2];
    DevBuf<int32_t> nxt_pool[2];         /* two halves each: even and odd levels */
    DevBuf<unsigned long long> nx_top;   /* per level: next-list tops (direct, ewald), drain counter, spare */
    DevBuf<int32_t *> wk_pools, wk_llen; /* device copies of the list pointer tables */
    DevBuf<int64_t *> wk_loff;
    DevBuf<int64_t> wk_caps;
    DevBuf<WalkRec> wk_rec;              /* per node: what the opening tests read */
    DevBuf<int4> pp_rec;                 /* 2 per node: source leaves as PP direct selects them */
    DevBuf<double> pp_part;              /* list shares' sums, 4 per share and particle */
    DevBuf<int32_t> scratch;             /* leaf drain per-warp scratch */
    int64_t scratch_per_warp = 0;
    int drain_warps = 0;
    int64_t list_cap[NLIST] = {0, 0, 0, 0, 0, 0, 0, 0}; /* pool capacities that served the last walk */
    int64_t nx_cap[2] = {0, 0};
    int64_t cap_start = 0; /* tg_set_walk_capacity: first capacity of every pool (0: sized from the tree) */

    /* status / stats */
    DevBuf<uint32_t> dev_err;
    DevBuf<unsigned long long> dev_cnt; /* 16 counters */
    uint32_t *h_err = nullptr;          /* pinned */
    unsigned long long *h_cnt = nullptr;
    void *h_stage = nullptr;            /* pinned staging for host transfers */
    /* pinned, 4 KB: [0, 2048) uploads of small tables, [2048, 4096) small
     * readbacks (pageable copies would go through the driver's staging,
     * which host threads driving other solvers contend for) */
    unsigned char *h_small = nullptr;
    size_t h_stage_bytes = 0;

    /* Ewald tables */
    /* leapfrog checkpoints (caller order) and adjoint state */
    DevBuf<int32_t> ck_x;
    DevBuf<float> ck_v;
    int ck_steps = -1;
    double ck_dt = 0.0;
    DevBuf<double> adj_x, adj_v, tid_u, tid_o, tid_U, tid_V, tid_tile;
    DevBuf<int32_t> ew_cnt, ew_off; /* leaf Ewald chunks per leaf, and their exclusive scan */
    DevBuf<double> ew_part;          /* 64 x 4 partial sums per chunk */
    DevBuf<float4> ew_real, ew_four;
    DevBuf<float> ew_Hf;
    DevBuf<double> ew_Hd;
    DevBuf<float4> ew_Pf;
    DevBuf<double2> ew_Pd;
    DevBuf<int4> ew_sep_h;       /* PP Ewald split: reciprocal vectors and weights */
    DevBuf<double> ew_sep_w;
    DevBuf<int4> ew_sep_run; /* FP32: runs of the vectors */
    int ew_sep_nrun = 0;
    double ew_sep_k = 0.0, ew_sep_r0 = 0.0, ew_sep_r2 = 0.0;
    SepNear ew_near{}; /* FP32 path */
    DevBuf<int32_t> ew_slot, ew_src; /* per node: its row of ew_sf, or -1; the nodes of the rows, then their count */
    DevBuf<unsigned char> ew_sf;    /* per PP_E source leaf and h: (cos, sin) sums over its particles (double2) */
    DevBuf<unsigned char> ew_tpart; /* per PP_E chunk and h: source sums (double2) */
    size_t ew_scratch_set = 0; /* tg_set_ewald_scratch; 0: by EW_SCRATCH */
    size_t ew_scratch() const {
        return ew_scratch_set ? ew_scratch_set : std::max(EW_SCRATCH, EW_SCRATCH_N * (size_t)n);
    }
    int32_t ew_max_npp = 0, ew_max_nsrc = 0; /* most PP_E chunks and source leaves of any evaluation */
    bool ew_use_tab = false;       /* a periodic solver of the FP32 path */
    const float *ew_tab = nullptr; /* the device's table of local expansions (FP32 path), shared by its solvers */
    bool have_tables = false;

    /* rung (individual) time steps: the rung lives in vel[i].w */
    DevBuf<int32_t> rung_flag, rung_scan, rung_nact; /* active flag per particle, its scan, active per node */
    DevBuf<int8_t> rung_out;                         /* caller-order rungs for tg_get_rungs */
    const int32_t *walk_nact = nullptr;              /* set during a rung step's walk only */

    /* friends-of-friends (sorted order unless noted) */
    DevBuf<int32_t> fof_P, fof_leaves, fof_key, fof_mem, fof_runs;
    DevBuf<int64_t> fof_gmin, fof_group; /* fof_group: caller order */
    DevBuf<uint8_t> fof_has;
    DevBuf<int2> fof_pairs;
    DevBuf<float> fof_radii;
    DevBuf<double> fof_stats;
    int64_t fof_ngroups = 0, fof_npairs = 0;
    double fof_link = 0.0; /* linking length of the groups held, 0: none for this tree */
    int32_t fof_tries = 65536; /* hook attempts per union before the union-find gives up */

    /* events for phase timing */
    cudaEvent_t ev[8];
    bool have_events = false;
    bool pp_timed = false; /* ev[6] marks the start of the FP32 PP kernel in the last solve */
    bool kd_timed = false; /* ev[7] marks a fused kick-drift that the last solve's build followed */
    bool kd_pending = false;
    tg_stats st{};
    int num_sms = 148;
    int64_t launches = 0; /* kernels of this library launched on this handle */
};

/* count a kernel launch of this library and check it */
inline int launched(Solver &S) {
    S.launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_cuda_error(e, "kernel launch", __FILE__, __LINE__);
        return TG_ERR_CUDA;
    }
    return TG_OK;
}

/* device bytes held by every DevBuf of the process (all handles) */
inline std::atomic<long long> g_dev_bytes{0};

template <class T>
int ensure(DevBuf<T> &b, size_t count) {
    if (b.n >= count && b.p) return TG_OK;
    if (b.p) {
        cudaFree(b.p);
        g_dev_bytes -= (long long)(b.n * sizeof(T));
    }
    b.p = nullptr;
    b.n = 0;
    size_t c = count < 16 ? 16 : count;
    c = c + c / 4;
    if (cudaMalloc(&b.p, c * sizeof(T)) != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        return TG_ERR_NOMEM;
    }
    b.n = c;
    g_dev_bytes += (long long)(c * sizeof(T));
    return TG_OK;
}
template <class T>
void release(DevBuf<T> &b) {
    if (b.p) {
        cudaFree(b.p);
        g_dev_bytes -= (long long)(b.n * sizeof(T));
    }
    b.p = nullptr;
    b.n = 0;
}

int init_constants();
int ewald_tables(Solver &S, cudaStream_t st);
/* the device's shared Ewald expansion table: made by the first solver that needs it, freed with the last */
int ewald_table_acquire(int dev, const float4 *real, const float4 *four, const float **tab, cudaStream_t st);
void ewald_table_release(int dev);
size_t ewald_table_bytes();
int tree_build(Solver &S, cudaStream_t st);
int tree_multipoles(Solver &S, cudaStream_t st);
int tree_walk(Solver &S, cudaStream_t st);
int gravity_forces(Solver &S, cudaStream_t st);
int kick(Solver &S, double dt, cudaStream_t st);
int drift(Solver &S, double dt, cudaStream_t st);
int kick_drift(Solver &S, double dt_close, double dt_open, double dt_drift, cudaStream_t st);
int energy(Solver &S, double out[5], cudaStream_t st);
int truth(Solver &S, const int64_t *samples, int64_t ns, double alpha, double *phi, double *g, cudaStream_t st);
int read_err(Solver &S, cudaStream_t st, uint32_t *err);
/* bytes (<= 2048) from device memory to dst through the pinned h_small; waits for st */
int read_small(Solver &S, cudaStream_t st, void *dst, const void *src, size_t bytes);
int fp32_peak(int device, double *tflops, cudaStream_t st);

} // namespace tg
