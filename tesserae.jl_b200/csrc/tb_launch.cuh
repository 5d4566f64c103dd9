// tb_launch.cuh -- host-side launchers shared between the kernel files and the
// C-ABI layer of libtesserae_b200.so.
#pragma once

#include "tb_common.cuh"

namespace tb {

// Device buffers of one binning pass (GPUBlockStrategy arrays plus scratch).
struct BinBuffers {
    int* blockids;        // [n] caller
    int* counts;          // [nb] caller
    int* offsets;         // [nb+1] caller
    int* blocklist;       // [nb] caller
    int* perm;            // [n] caller, 1-based particle ids
    int* cursors;         // [nb] scratch
    int* perm_tmp;        // [n] scratch, 0-based ids in warp-run order
    unsigned long long* partials;  // [ntiles] scratch
    unsigned long long* sort_scratch;  // [2n] scratch for large blocks
    int* totals;          // [2] device: nactive, nassigned
    unsigned long long* bnd_count;  // [1] blocks P2G leaves to its second launch; zeroed by every binning
    bool fresh = false;   // the partition is that of the positions P2G reads
};

// Node blocks that a step's transfer touches, found by the scan of its binning:
// flags of this and the previous transfer, the list of blocks with either set.
struct TouchArgs {
    unsigned char* cur = nullptr;         // [nb]; null: not wanted
    const unsigned char* prev = nullptr;  // [nb]
    int* list = nullptr;                  // [nb]
    int* count = nullptr;                 // [1] zero on entry
    int* next_count = nullptr;            // [1] zeroed (the next step's count)
    int3 nb = {1, 1, 1};                  // blocks per axis
};

// Scratch of a sparse grid's numbering pass (one int per block each, the scan
// partials, two totals).
struct SparseScratch {
    int* act;       // [nb] block activity
    int* offsets;   // [nb+1]
    int* cursors;   // [nb] (written by the shared scan, unused)
    unsigned long long* partials;  // [ntiles]
    int* totals;    // [2]
};

constexpr int SCAN_TILE = 1024;  // blocks per scan tile (256 threads x 4)

inline int scan_tiles(int nb) { return (nb + SCAN_TILE - 1) / SCAN_TILE; }

// Optional per-kernel timing: CUDA events recorded on the launching stream
// around every launch while profiling is enabled (tb_profile_enable).
struct Profiler {
    virtual void begin(const char* name, cudaStream_t s) = 0;
    virtual void end(cudaStream_t s) = 0;
    virtual ~Profiler() = default;
};

struct LaunchCfg {
    cudaStream_t stream;
    int num_sms;
    long long* launches;  // incremented per kernel launch
    int* err;             // device status word
    Profiler* prof;       // null unless profiling
    bool early = false;   // launch_chained may set blocks up early
};

// Scenes up to this many particles set their blocks up early: a launch is then a
// good part of its kernel. Whole steps early / in order, us: 2D 361 k particles 79.5 / 91.6;
// 3D FP32 with FP64 positions 262 k 76 / 88, 1.0 M 190 / 202, 2.7 M 473 / 479, 8.0 M 1195 / 1199,
// 16.8 M 2338 / 2324; FP64 512 k 175 / 179, 2.7 M 788 / 794, 5.8 M 1518 / 1516; WLS + APIC 2.6 M 743 / 759,
// 18 M 5069 / 5065. Two kernels follow in order where they lose by it (p2g_plane_kernel;
// bin_fixup_kernel in crowded scenes): their large blocks arrive on SMs that still run the
// launch before.
constexpr long long EARLY_N = 1 << 23;

// Launches of a step follow each other on one stream; each waits for the one before
// on the device (chain_wait, its first statement) instead of at launch, so that its
// blocks are set up while the last blocks of the one before still run
// (programmatic dependent launch; cfg.early). A kernel launched this way must call chain_wait.
template <class... Params, class... Args>
cudaError_t launch_chained(void (*kern)(Params...), unsigned grid, unsigned threads, size_t smem, const LaunchCfg& cfg,
                           Args&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = cfg.stream;
    c.attrs = &attr;
    c.numAttrs = cfg.early ? 1 : 0;
    return cudaLaunchKernelEx(&c, kern, static_cast<Params>(args)...);
}

// Lets the next launch of the chain set up its blocks, then waits until the launch
// before has completed and its writes are visible.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// RAII scope naming the kernel launches it encloses.
struct KernelScope {
    const LaunchCfg& cfg;
    KernelScope(const LaunchCfg& c, const char* name) : cfg(c) {
        if (cfg.prof) cfg.prof->begin(name, cfg.stream);
    }
    ~KernelScope() {
        if (cfg.prof) cfg.prof->end(cfg.stream);
    }
};

template <int D, class T>
cudaError_t launch_bin(const DMesh<D, T>& M, const T* const* x, long long n, const BinBuffers& b,
                       const LaunchCfg& cfg, const TouchArgs& touch = TouchArgs{}, bool zero_counts = false);

// Count kernel alone (positions -> blockids, counts); the rest of the pass in
// launch_bin_rest. Split so a fused step can count inside G2P.
template <int D, class T>
cudaError_t launch_bin_count(const DMesh<D, T>& M, const T* const* x, long long n, const BinBuffers& b,
                             const LaunchCfg& cfg);
// `zero_counts`: b.counts are zero again afterwards (for a G2P that counts ahead).
cudaError_t launch_bin_rest(int nblocks, long long n, const BinBuffers& b, const LaunchCfg& cfg,
                            const TouchArgs& touch = TouchArgs{}, bool zero_counts = false);

// update_sparsity! from a binning pass: the node blocks within one block of a
// block that holds particles (b.blocklist / b.totals), numbered in ascending
// order into bnum (0 inactive, k >= 1), their 1-based ids into blist, the count
// into nact[0] (src/Grids/sparsity.jl:19-60, 192-232).
cudaError_t launch_sparsity(int dim, const int* nbv, int nblocks, const BinBuffers& b, const SparseScratch& sc,
                            int* bnum, int* blist, int* nact, const LaunchCfg& cfg);

// P2G scatter into a grid whose m, mv, f are already zero where it will add.
template <int D, class T, int BW>
cudaError_t launch_p2g(const DMesh<D, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                       const BinBuffers& b, const LaunchCfg& cfg);

template <int D, class T>
cudaError_t launch_grid_update(const DMesh<D, T>& M, const GView<T>& G, const Scalars<T>& s, const LaunchCfg& cfg);

template <int D, class T>
cudaError_t launch_grid_zero(const DMesh<D, T>& M, const GView<T>& G, const LaunchCfg& cfg);

// With `count_next`, G2P also writes every moved particle's block id for the
// next step into b.blockids and adds it to b.counts (zeroed by this step's
// binning): the count pass of the next step's binning, so that step runs
// launch_bin_rest only.
template <int D, class T, int BW>
cudaError_t launch_g2p(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                       const BinBuffers& b, const LaunchCfg& cfg, bool count_next = false);

// Grid maintenance over the listed node blocks (TouchArgs): see tb_transfer.cu.
template <int D, class T, int BW>
cudaError_t launch_sparse_zero(const DMesh<D, T>& M, const GView<T>& G, const int* list, const int* count,
                               const LaunchCfg& cfg);
template <int D, class T, int BW>
cudaError_t launch_sparse_grid_update(const DMesh<D, T>& M, const GView<T>& G, const Scalars<T>& s,
                                      const unsigned char* cur, const int* list, const int* count,
                                      const LaunchCfg& cfg, bool zero_after = false);

// max over the particles of sqrt((lambda + 2 mu) / (m / V)) + |v| into *out
// (the bits of a double).
template <int D, class T>
cudaError_t launch_wave_speed(const PView<T>& P, const Scalars<T>& s, unsigned long long* out, const LaunchCfg& cfg);

template <int D, class T>
cudaError_t launch_g2p_direct(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                              const LaunchCfg& cfg);

// Reverse mode: the caller's FP64 sensitivity arrays (tb_adjoint) and the
// context's FP64 grid sensitivities (component-major, nnodes each).
struct AdjView {
    double* x[3];
    double* v[3];
    double* F[9];
    double* mu;
    double* lam;
    double* B[9];  // APIC only
};
struct GradGrid {
    double* vb[3];   // d loss / d v_i (scattered by G2P backwards)
    double* vnb[3];  // d loss / d vn_i
    double* mb;      // d loss / d m_i
    double* pb[3];   // d loss / d mv_i
    double* fb[3];   // d loss / d f_i
    double* coef;    // per permutation slot: G2P backwards' scatter coefficients (2 D + D^2 arrays of n)
};

// The partition of the step being reversed (device arrays).
struct AdjPartition {
    const int* totals;     // [2] nactive, nassigned
    const int* blocklist;
    const int* offsets;
    const int* perm;
    const int* blockids;
};

// G2P, grid update and P2G backwards for one step whose forward grid is in G
// and whose partition is `part` (tb_adjoint.cu). Zeroes GB's v / vn
// sensitivities first.
template <int D, class T, int BW>
cudaError_t launch_adjoint(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                           const AdjView& A, const GradGrid& GB, const AdjPartition& part, const LaunchCfg& cfg);
// The same for WLS / KernelCorrection bases and the APIC transfer (particle-parallel,
// weight derivatives in Dual1).
template <int D, class T>
cudaError_t launch_adjoint_general(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                                   const AdjView& A, const GradGrid& GB, const AdjPartition& part, const LaunchCfg& cfg);

template <int D, class T>
cudaError_t launch_update_weights(const DMesh<D, T>& M, const PView<T>& P, const Scalars<T>& s, T* w, T* grad_w,
                                  long long* window, const LaunchCfg& cfg);

// reorder_particles! (tb_reorder.cu). One particle field: a device array of n
// elements of `elem` (4 or 8) bytes.
struct ReorderField {
    void* ptr;
    int elem;
};
struct ReorderArgs {
    long long n;
    int nblocks;
    int* blockids;         // [n] permuted with the particles
    int* perm;             // [n] 1-based block-sorted permutation; identity after a reorder
    const int* offsets;    // [nblocks + 1]
    double threshold;      // reorder when the score is below it (always at >= 1, never at <= 0)
    unsigned long long* acc;  // [2] scratch: same-block neighbours, non-empty blocks
    int* decision;         // [2] reorder now; reorder wanted but particles lie outside the mesh
    double* score;         // [1] contiguity score
    void* scratch;         // [n] x 8 bytes
    bool report_outside;   // raise ERR_REORDER_OUTSIDE in the status word when a reorder is refused
};
// Score and decision on the device (no host synchronisation).
cudaError_t launch_reorder_score(const ReorderArgs& a, const LaunchCfg& cfg);
// Permute `fields`, the block ids and the permutation when decision[0] is set.
cudaError_t launch_reorder_apply(const ReorderArgs& a, const ReorderField* fields, int nfields, const LaunchCfg& cfg);

}  // namespace tb
