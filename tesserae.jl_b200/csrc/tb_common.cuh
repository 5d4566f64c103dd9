// tb_common.cuh -- device-side data views and basis math shared by the kernels
// of libtesserae_b200.so (sm_100a).
//
// Mesh, window and weight rules follow the reference:
//   findblock / windows    Tesserae.jl src/Mesh/cartesian.jl:146-285
//   quadratic B-spline     src/Basis/bspline.jl:28-184 (fast full-support path and
//                          the nodewise path for truncated windows)
//   uGIMP                  src/Basis/gimp.jl:16-40
//   WLS (MLS-MPM)          src/Basis/wls.jl:22-84
// The basis values are evaluated inside the transfers ("deferred" weights,
// src/Transfer/runtime.jl:55-130), so no weight array crosses HBM.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tesserae_b200.h"

namespace tb {

// Error bits a kernel raises in the context's device status word.
enum : int {
    ERR_TILE_RANGE = 1,   // a support window left its block tile
    ERR_GIMP_LENGTH = 2,  // uGIMP requires 0 <= l <= h (gimp.jl:22)
    ERR_WLS_SINGULAR = 4,  // WLS moment matrix not invertible
    ERR_REORDER_OUTSIDE = 8,  // a reorder was due but particles lie outside the mesh
    ERR_INACTIVE_NODE = 16,   // a scatter reached a node of an inactive block of a sparse grid
    ERR_SPGRID_CAPACITY = 32  // a sparse grid's active blocks exceed its field arrays
};

// CTAs that share one block of the block list: the average particle count of
// the non-empty blocks (totals = {nactive, nassigned}) over `per_cta`, the
// particles one CTA takes per pass, between 1 and 8. A crowded scene (4^3
// particles per cell: 4096 per 4^3-cell block) has fewer blocks than the GPU
// has CTA slots; splitting each block's passes over several CTAs (CTA `sub` of
// `split` takes passes sub, sub + split, ...) restores the parallelism. The
// transfers add each pass's tile to the grid with global atomics anyway, so
// the split costs no extra work.
__device__ __forceinline__ int block_split(const int* totals, int per_cta) {
    const long long nact = totals[0], nass = totals[1];
    if (nact <= 0) return 1;
    const long long s = (nass / nact + per_cta / 2) / per_cta;
    return int(s < 1 ? 1 : (s > 8 ? 8 : s));
}

// CTAs that share one block in a kernel that takes passes of up to `nb` particles
// and may sum several passes before it adds them to the grid, for `nblk` blocks
// on a grid of `ctas`: enough for about twelve pieces per CTA while every piece
// still has a full pass (2.1 M-particle FP64 sphere of 64 per cell: P2G 0.455 ms at four,
// 0.378 at twelve), and for one piece per CTA where the blocks are fewer than
// the CTAs (passes of `per` < nb particles then, at least 128). Short passes cost:
// a 64^3 B-spline block of 262 k particles (512 blocks on 444 CTAs) took 5% longer
// per step with two half passes per block than with one.
__device__ __forceinline__ int block_pieces(const int* totals, int nblk, int nb, int ctas, int& per) {
    per = nb;
    const int nact = totals[0];
    if (nact <= 0 || nblk <= 0) return 1;
    const int avg = int((long long)totals[1] / nact), passes = (avg + nb - 1) / nb;
    const int full = min(passes, (12 * ctas + nblk - 1) / nblk), fill = min(ctas / nblk, (avg + 127) / 128);
    const int pieces = max(1, min(8, max(full, fill)));
    if (pieces > passes) per = min(nb, max(128, ((avg + pieces - 1) / pieces + 7) & ~7));
    return pieces;
}

// The passes of one block's particle range [s0, s1) for kernels that hold `per`
// particles (a multiple of 8) at a time: pass i of count() = ceil(n / per)
// takes the 8-particle chunks i, i + count(), i + 2 count(), ..., so every pass
// samples the whole block. A block denser than one pass whose particles lie in
// lattice order (4^3 per cell: 16 lattice rows of x per block row) would
// otherwise give each pass a few (y, z) rows of the block, all of its records
// to a few pencils, and a sweep as long as the longest of them. A 32-particle
// warp load touches 4 chunks of 8, the same sectors as a contiguous one for
// 4-byte fields. With one pass this is the range itself, in order.
struct BlockPasses {
    int s0, s1, npass;
    __device__ __forceinline__ BlockPasses(int a, int b, int per) : s0(a), s1(b), npass((b - a + per - 1) / per) {}
    __device__ __forceinline__ int count() const { return npass; }
    // position in the block list of item t (0 <= t < per) of pass i (>= s1: past the range)
    __device__ __forceinline__ int pos(int i, int t) const { return s0 + ((i + npass * (t >> 3)) << 3) + (t & 7); }
    // pos(i, t + nt) - pos(i, t) for nt a multiple of 8
    __device__ __forceinline__ int step(int nt) const { return npass * nt; }
};

// Forward-mode dual number: a value and its derivative with respect to one
// coordinate of the particle. Every basis of this path is built axis by axis, so
// one derivative (of each axis's jets with respect to that axis's coordinate) gives
// dN/dx_p and d(grad N)/dx_p of the reverse step for every basis (WLS,
// KernelCorrection, cut windows) without hand-derived second derivatives. Floors and
// comparisons act on the value, |x| follows the value's sign. In a namespace of
// its own, so that floor, fabs and signbit of plain numbers inside tb still
// resolve to the CUDA functions (the Dual1 overloads are found by argument-
// dependent lookup).
namespace ad {
struct Dual1 {
    double v, d;
    __host__ __device__ Dual1() : v(0.0), d(0.0) {}
    __host__ __device__ Dual1(double a) : v(a), d(0.0) {}
    __host__ __device__ explicit operator double() const { return v; }
    __host__ __device__ explicit operator float() const { return float(v); }
    __host__ __device__ explicit operator int() const { return int(v); }
    __host__ __device__ Dual1 operator-() const {
        Dual1 r;
        r.v = -v;
        r.d = -d;
        return r;
    }
    __host__ __device__ Dual1& operator+=(const Dual1& o) {
        v += o.v;
        d += o.d;
        return *this;
    }
    __host__ __device__ Dual1& operator-=(const Dual1& o) {
        v -= o.v;
        d -= o.d;
        return *this;
    }
    __host__ __device__ Dual1& operator*=(const Dual1& o) {
        d = d * o.v + v * o.d;
        v *= o.v;
        return *this;
    }
    __host__ __device__ Dual1& operator/=(const Dual1& o) {
        const double iv = 1.0 / o.v;
        d = (d - v * iv * o.d) * iv;
        v *= iv;
        return *this;
    }
};
__host__ __device__ inline Dual1 operator+(Dual1 a, const Dual1& b) { return a += b; }
__host__ __device__ inline Dual1 operator-(Dual1 a, const Dual1& b) { return a -= b; }
__host__ __device__ inline Dual1 operator*(Dual1 a, const Dual1& b) { return a *= b; }
__host__ __device__ inline Dual1 operator/(Dual1 a, const Dual1& b) { return a /= b; }
__host__ __device__ inline bool operator<(const Dual1& a, const Dual1& b) { return a.v < b.v; }
__host__ __device__ inline bool operator>(const Dual1& a, const Dual1& b) { return a.v > b.v; }
__host__ __device__ inline bool operator<=(const Dual1& a, const Dual1& b) { return a.v <= b.v; }
__host__ __device__ inline bool operator>=(const Dual1& a, const Dual1& b) { return a.v >= b.v; }
__host__ __device__ inline bool operator==(const Dual1& a, const Dual1& b) { return a.v == b.v; }
__host__ __device__ inline bool operator!=(const Dual1& a, const Dual1& b) { return a.v != b.v; }
__device__ inline Dual1 floor(const Dual1& a) { return Dual1(::floor(a.v)); }
__device__ inline Dual1 fabs(const Dual1& a) { return ::signbit(a.v) ? -a : a; }
__device__ inline bool signbit(const Dual1& a) { return ::signbit(a.v); }
}  // namespace ad
using ad::Dual1;

template <int D, class T>
struct DMesh {
    int n[3];      // nodes per axis
    int nb[3];     // blocks per axis
    int L;         // block_log2
    int nblocks;
    long long nnodes;
    T xmin[3];
    T h, h_inv;
    double xmin64[3], h64, h_inv64;
};

template <int D, class T>
inline DMesh<D, T> make_dmesh(const tb_mesh& m) {
    DMesh<D, T> M{};
    M.L = m.block_log2;
    M.nblocks = 1;
    M.nnodes = 1;
    for (int d = 0; d < 3; ++d) {
        M.n[d] = d < D ? int(m.n_nodes[d]) : 1;
        M.nb[d] = d < D ? ((M.n[d] - 1) >> M.L) + 1 : 1;
        M.xmin[d] = T(m.xmin[d]);
        M.xmin64[d] = m.xmin[d];
        M.nblocks *= M.nb[d];
        M.nnodes *= M.n[d];
    }
    M.h = T(m.h);          // the Float32 form casts h and h_inv separately (src/adapt.jl:53-57)
    M.h_inv = T(m.h_inv);
    M.h64 = m.h;
    M.h_inv64 = m.h_inv;
    return M;
}

// Particle SoA views. T is the state scalar; F is always double. In the
// FP64-position form (FP32 state with FP64 positions) x is NULL and x64 holds
// the positions; otherwise x64 is NULL.
template <class T>
struct PView {
    long long n;
    T* x[3];
    double* x64[3];
    T* v[3];
    T* V;
    const T* m;
    const T* l;
    T* gv[9];
    T* sig[6];
    double* F[9];
    T* B[9];
    const T* V0;
    const T* mu;
    const T* lam;
    T* eps_p;      // von Mises: equivalent plastic strain
    T* Cp_inv[6];  // von Mises: inverse plastic right Cauchy-Green tensor (symmetric)
    // Where G2P stores the new positions when they must not replace x yet
    // (G2P2G: its P2G half weighs at the old ones); NULL = in place.
    T* x_out[3];
    double* x64_out[3];
};

template <class T>
struct GView {
    T* m;
    T* mv[3];
    T* f[3];
    T* v[3];
    T* vn[3];
    // block-sparse grid (bnum set): node block numbering (0 inactive, k >= 1
    // storage block k), the node block of each storage block (1-based ids),
    // the active block count (device), the nodes the fields hold and log2 of
    // the block edge
    const int* bnum;
    const int* blist;
    const int* nact;
    long long cap;
    int L;
};

// Storage slot of node (x, y, z) (z = 0 in 2D): the column-major linear index
// on a dense grid; on a block-sparse grid (src/Grids/spindices.jl storageindex)
// (k - 1) blocklength + the node's column-major index inside its block, k the
// block's storage number. -1: the block is inactive; -2: past the fields'
// capacity.
template <int D, class T, class MT>
__device__ __forceinline__ long long grid_slot(const GView<T>& G, const MT& M, int x, int y, int z) {
    if (!G.bnum) return (long long)x + (long long)M.n[0] * ((long long)y + (D == 3 ? (long long)M.n[1] * z : 0ll));
    const int L = G.L, W = 1 << L, mk = W - 1;
    const int B = (x >> L) + M.nb[0] * ((y >> L) + (D == 3 ? M.nb[1] * (z >> L) : 0));
    const int k = G.bnum[B];
    if (k <= 0) return -1;
    const int q = (x & mk) + W * ((y & mk) + (D == 3 ? W * (z & mk) : 0));
    const long long sl = (long long)(k - 1) * (D == 3 ? W * W * W : W * W) + q;
    return sl < G.cap ? sl : -2;
}

// Adds one node's P2G sums (m, mv[D], f[D], gravity already in f) to the grid,
// one atomic per non-zero value. A non-zero sum for a node that a sparse grid
// does not store sets ERR_INACTIVE_NODE (update_sparsity! was not run for these
// positions: src/Transfer/runtime.jl:152-161) or ERR_SPGRID_CAPACITY.
template <int D, class T, class MT, class V>
__device__ __forceinline__ void grid_add(const GView<T>& G, const MT& M, int* err, int x, int y, int z,
                                         const V* val) {
    bool any = val[0] != V(0);
#pragma unroll
    for (int c = 1; c < 1 + 2 * D; ++c) any = any || val[c] != V(0);
    if (!any) return;
    const long long sl = grid_slot<D>(G, M, x, y, z);
    if (sl < 0) {
        atomicOr(err, sl == -1 ? ERR_INACTIVE_NODE : ERR_SPGRID_CAPACITY);
        return;
    }
    if (val[0] != V(0)) atomicAdd(G.m + sl, T(val[0]));
#pragma unroll
    for (int d = 0; d < D; ++d) {
        if (val[1 + d] != V(0)) atomicAdd(G.mv[d] + sl, T(val[1 + d]));
        if (val[1 + D + d] != V(0)) atomicAdd(G.f[d] + sl, T(val[1 + D + d]));
    }
}

// A particle's uGIMP length over the spacing: in the state type, its inverse,
// and in FP64 (for the windows of the FP64-position form).
template <class T>
struct GimpLen {
    T ln, il;
    double ln64;
};

// Step scalars, converted once to the state type.
template <class T>
struct Scalars {
    T dt, mass, V0, g[3], gimp_l, alpha;
    double dt64, V0_64, mu, lam, hardening, yield_stress;
    GimpLen<T> gimp;  // of gimp_l, for all particles when none has its own
    int basis, transfer, material, wall_mask, wall_layers;
};

template <class T>
inline Scalars<T> make_scalars(const tb_step_params& p, const tb_mesh& m) {
    Scalars<T> s{};
    s.gimp.ln = T(p.gimp_l) / T(m.h);
    s.gimp.il = T(1) / s.gimp.ln;
    s.gimp.ln64 = double(T(p.gimp_l)) / m.h;
    s.dt = T(p.dt);
    s.mass = T(p.mass);
    s.V0 = T(p.V0);
    for (int d = 0; d < 3; ++d) s.g[d] = T(p.gravity[d]);
    s.gimp_l = T(p.gimp_l);
    s.alpha = T(p.flip_alpha);
    s.dt64 = p.dt;
    s.V0_64 = p.V0;
    s.mu = p.mu;
    s.lam = p.lambda;
    s.basis = p.basis;
    s.transfer = p.transfer;
    s.material = p.material;
    s.wall_mask = p.wall_mask;
    s.wall_layers = p.wall_layers;
    s.hardening = p.hardening;
    s.yield_stress = p.yield_stress;
    return s;
}

// Basis kinds whose support window is uGIMP's, and the KernelCorrection kinds.
__host__ __device__ inline bool basis_is_gimp(int basis) {
    return basis == TB_UGIMP || basis == TB_WLS_UGIMP || basis == TB_KC_UGIMP;
}
__host__ __device__ inline bool basis_is_kc(int basis) {
    return basis == TB_KC_BSPLINE_QUADRATIC || basis == TB_KC_UGIMP;
}

template <int D>
__host__ __device__ constexpr int nsym() { return D == 3 ? 6 : 3; }

// Index of (r, c) in Tensorial's symmetric independent-component order.
template <int D>
__host__ __device__ constexpr int symidx(int r, int c) {
    return (r >= c) ? (c * D - c * (c - 1) / 2 + (r - c)) : (r * D - r * (r - 1) / 2 + (c - r));
}

// Node coordinate X_d(i) = xmin + i h, rounded once in FP64 and cast to T
// (the reference stores the axes as Vector{T}(range(xmin; step=h, length=n))).
template <int D, class T>
__device__ __forceinline__ T node_coord(const DMesh<D, T>& M, int d, int i) {
    return T(__dadd_rn(M.xmin64[d], __dmul_rn(double(i), M.h64)));
}

// 1-based linear block id (0 = outside), cartesian.jl:271-285 + sub2ind.
template <int D, class T>
__device__ __forceinline__ int findblock(const DMesh<D, T>& M, const T* x) {
    int lin = 0;
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
        T c = floor((x[d] - M.xmin[d]) * M.h_inv);
        if (!(c >= T(0) && c <= T(M.n[d] - 2))) return 0;
        lin = lin * M.nb[d] + (int(c) >> M.L);
    }
    return lin + 1;
}

// findblock of an FP64 position with the mesh's FP64 xmin and h_inv (the
// Float64 rule of cartesian.jl:271-285, as findblock<D, double>).
template <int D, class T>
__device__ __forceinline__ int findblock_x64(const DMesh<D, T>& M, const double* x) {
    int lin = 0;
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
        const double c = floor((x[d] - M.xmin64[d]) * M.h_inv64);
        if (!(c >= 0.0 && c <= double(M.n[d] - 2))) return 0;
        lin = lin * M.nb[d] + (int(c) >> M.L);
    }
    return lin + 1;
}

// Per-axis basis data of one particle: window start/count and the 1-D jets.
template <class T>
struct Axis {
    int lo, cnt;
    T val[3], der[3];
};

// 1-D jets, forward-mode derivative through abs() as in the reference's AD.
template <class T>
__device__ __forceinline__ void jet_bspline_quadratic(T xi, T& val, T& der) {
    T s = signbit(xi) ? T(-1) : T(1);
    T a = fabs(xi);
    if (a < T(0.5)) {
        val = (T(3) - T(4) * (a * a)) / T(4);
        der = -(T(2) * a) * s;
    } else if (a < T(1.5)) {
        T t = T(3) - T(2) * a;
        val = (t * t) / T(8);
        der = -(t / T(2)) * s;
    } else {
        val = T(0);
        der = T(0);
    }
}

// a / l given il = 1 / l: the product, corrected once by its residual a - q l
// (the final quotient step of P. Markstein, IBM J. Res. Dev. 34, 1990), so that a
// length shared by all particles does not put the rounding of its inverse into
// every weight.
__device__ __forceinline__ float quotient(float a, float l, float il) {
    const float q = a * il;
    return fmaf(fmaf(-q, l, a), il, q);
}
__device__ __forceinline__ double quotient(double a, double l, double il) {
    const double q = a * il;
    return fma(fma(-q, l, a), il, q);
}
__device__ __forceinline__ Dual1 quotient(const Dual1& a, const Dual1& l, const Dual1&) { return a / l; }

// uGIMP jets (gimp.jl:16-40); il = 1 / l, computed once per particle or per scene.
// (The nine jets of a 3D particle held 27 divisions by l, about half of the
// instructions of the WLS(uGIMP) kernels' basis.)
template <class T>
__device__ __forceinline__ void jet_ugimp(T xi, T l, T il, T& val, T& der) {
    T s = signbit(xi) ? T(-1) : T(1);
    T a = fabs(xi);
    const T hl = l * T(0.5);
    if (a < hl) {
        val = T(1) - quotient(a * a + hl * hl, l, il);
        der = -quotient(T(2) * a, l, il) * s;
    } else if (a < T(1) - hl) {
        val = T(1) - a;
        der = -s;
    } else if (a < T(1) + hl) {
        T t = T(1) + hl - a;
        const T q = quotient(t, l, il);
        val = T(0.5) * (t * q);
        der = -q * s;
    } else {
        val = T(0);
        der = T(0);
    }
}

// Fast full-support axis values (bspline.jl:90-100): t = fract(xi - 1/2),
// N = (1/2 - t + t^2/2, 1/2 + t - t^2, t^2/2), N' = (t - 1, 1 - 2t, t).
template <class T>
__device__ __forceinline__ void bspline_quadratic_poly(T t, T* v0, T* v1) {
    const T half = T(0.5);
    v0[0] = half + t * (T(-1) + t * half);
    v0[1] = half + t * (T(1) + t * T(-1));
    v0[2] = t * (t * half);
    v1[0] = T(-1) + t;
    v1[1] = T(1) + t * T(-2);
    v1[2] = t;
}

template <class T>
__device__ __forceinline__ void bspline_quadratic_axis(T xi, T* v0, T* v1) {
    T u = xi - T(0.5);
    T t = u - floor(u);
    bspline_quadratic_poly(t, v0, v1);
}

// Window and 1-D jets of one particle for B-spline / uGIMP kernels (the
// kernel part of WLS too). Returns false when the particle is outside the mesh
// (empty window, cartesian.jl:190-199). `full` reports a 3^D window.
// Support window of one particle: xi = (x - xmin) h_inv per axis, the clamped
// window start and node count per axis (supportnodes, bspline.jl:28-40 and
// cartesian.jl:190-199). Returns false when the particle is outside the mesh.
template <int D, class T>
__device__ __forceinline__ bool axis_window(const DMesh<D, T>& M, int basis, const T* x, T lnorm, T* xi, int* lo,
                                            int* cnt, bool* cut = nullptr) {
    bool inside = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        xi[d] = (x[d] - M.xmin[d]) * M.h_inv;
        T c = floor(xi[d]);
        inside = inside && (c >= T(0) && c <= T(M.n[d] - 2));
    }
    if (!inside) return false;
    const bool gimp = basis_is_gimp(basis);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        int s, e;
        if (gimp) {
            T r = T(1) + lnorm / T(2);
            s = int(floor(xi[d] - r)) + 1;
            e = int(floor(xi[d] + r));
        } else {
            s = int(floor(xi[d] - T(0.5)));
            e = s + 2;
        }
        lo[d] = max(s, 0);
        cnt[d] = min(e, M.n[d] - 1) - lo[d] + 1;
        if (cut) cut[d] = s < 0 || e > M.n[d] - 1;  // the mesh cuts the support on this axis
    }
    return true;
}

template <int D, class T>
__device__ __forceinline__ bool axis_weights(const DMesh<D, T>& M, int basis, const T* x, const GimpLen<T>& gl,
                                             Axis<T>* ax, bool& full, bool* cut = nullptr) {
    T xi[3];
    int lo[3], cnt[3];
    if (!axis_window<D, T>(M, basis, x, gl.ln, xi, lo, cnt, cut)) return false;
    const bool gimp = basis_is_gimp(basis);
    full = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        ax[d].lo = lo[d];
        ax[d].cnt = cnt[d];
        full = full && (ax[d].cnt == 3);
    }
    if ((basis == TB_BSPLINE_QUADRATIC || basis == TB_KC_BSPLINE_QUADRATIC) && full) {
#pragma unroll
        for (int d = 0; d < D; ++d) bspline_quadratic_axis(xi[d], ax[d].val, ax[d].der);
        return true;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ax[d].val[k] = T(0);
            ax[d].der[k] = T(0);
            if (k < ax[d].cnt) {
                T xn = (x[d] - node_coord(M, d, ax[d].lo + k)) * M.h_inv;
                if (gimp) jet_ugimp(xn, gl.ln, gl.il, ax[d].val[k], ax[d].der[k]);
                else jet_bspline_quadratic(xn, ax[d].val[k], ax[d].der[k]);
            }
        }
    }
    return true;
}

// KernelCorrection(kernel) with its default MultiLinear polynomial on a
// support the mesh cuts (src/Basis/kernelcorrection.jl:13-64; a whole support
// keeps the plain kernel). Without a node filter the MultiLinear weighted
// least-squares fit of a separable kernel is one 1-D fit with P = (1, X_i - x_p)
// per axis (the moment matrix of the tensor-product polynomial under a product
// weight is the Kronecker product of the axis moment matrices), the
// decomposition the reference evaluates for B-splines (wls.jl:88-103, 177-192).
// Per axis the kernel values w_k become w_k (M^-1 P_k)[0] and their derivative
// w_k (M^-1 P_k)[1]; a whole B-spline axis takes the closed form
// M^-1 = diag(1, 4/h^2) (wls.jl:29-49). `r[d][k]` = X_k - x_p. The derivative is
// stored in units of xi (times h) like the plain jets. False for a singular fit.
template <int D, class T>
__device__ __forceinline__ bool kc_correct(const DMesh<D, T>& M, bool bspline, const T (&r)[3][3], Axis<T>* ax) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        if (bspline && ax[d].cnt == 3) {
            const T c = T(4) / (M.h * M.h);
#pragma unroll
            for (int k = 0; k < 3; ++k) ax[d].der[k] = ax[d].val[k] * (c * r[d][k]) * M.h;
        } else {
            T S0 = T(0), S1 = T(0), S2 = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k >= ax[d].cnt) continue;
                S0 += ax[d].val[k];
                S1 += ax[d].val[k] * r[d][k];
                S2 += ax[d].val[k] * r[d][k] * r[d][k];
            }
            const T det = S0 * S2 - S1 * S1;
            if (det == T(0)) return false;
            const T i00 = S2 / det, i01 = -S1 / det, i11 = S0 / det;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const T w = ax[d].val[k];
                ax[d].val[k] = k < ax[d].cnt ? w * (i00 + i01 * r[d][k]) : T(0);
                ax[d].der[k] = k < ax[d].cnt ? w * (i01 + i11 * r[d][k]) * M.h : T(0);
            }
        }
    }
    return true;
}

// Kernel value and gradient at window slot (i, j, k), product order of
// bspline.jl:133-142 / basis_weight.jl:49-60.
template <int D, class T>
__device__ __forceinline__ void node_weight(const DMesh<D, T>& M, const Axis<T>* ax, int i, int j, int k, T& w,
                                            T* dw) {
    if constexpr (D == 3) {
        T vx = ax[0].val[i], vy = ax[1].val[j], vz = ax[2].val[k];
        w = (vx * vy) * vz;
        dw[0] = ((ax[0].der[i] * vy) * vz) * M.h_inv;
        dw[1] = ((vx * ax[1].der[j]) * vz) * M.h_inv;
        dw[2] = ((vx * vy) * ax[2].der[k]) * M.h_inv;
    } else {
        T vx = ax[0].val[i], vy = ax[1].val[j];
        w = vx * vy;
        dw[0] = (ax[0].der[i] * vy) * M.h_inv;
        dw[1] = (vx * ax[1].der[j]) * M.h_inv;
    }
}

// WLS weights in closed form. The reference inverts the moment matrix
// M = sum_i w_i P_i P_i^T, P = (1, X - x_p) (wls.jl:51-68; diag(1, 4/h^2) for a
// full quadratic B-spline support, wls.jl:29-49). The kernel weight is a product
// of axis factors and P has one axis per component, so with the axis moments
//   S0 = sum w,  u = sum w r / S0,  var = sum w (r - u)^2 / S0   (r = X - x_p)
// M = prod S0 [[1, u^T], [u, diag(var) + u u^T]], whose inverse is known:
//   grad N_i = G_i,  G_{i,d} = W_i (r_d - u_d) / var_d,   N_i = W_i - u . G_i,
// W_i = prod w / S0. Per axis the jets become (w / S0, w / S0 (r - u) / var): the
// weights keep the product form of the plain kernel, and only N needs the
// correction -u . G. On a support that the mesh does not cut, S0 = 1 and u = 0
// (the kernels reproduce linear fields) and N_i is the kernel itself; a
// B-spline's var is h^2/4. `r[d][k]` = X_{lo+k} - x_p; der is stored in units of
// xi (times h) like the plain jets. False where M is singular.
template <int D, class T>
__device__ __forceinline__ bool wls_correct(const DMesh<D, T>& M, bool bspline, const bool* cut, const T (&r)[3][3],
                                            Axis<T>* ax, T* u, T* var) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        u[d] = T(0);
        if (cut[d]) {
            T S0 = T(0), S1 = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                S0 += ax[d].val[k];
                S1 += ax[d].val[k] * r[d][k];
            }
            if (S0 == T(0)) return false;
            u[d] = S1 / S0;
#pragma unroll
            for (int k = 0; k < 3; ++k) ax[d].val[k] = ax[d].val[k] / S0;
        }
        if (bspline && !cut[d]) {
            var[d] = M.h * M.h / T(4);
        } else {
            var[d] = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const T q = r[d][k] - u[d];
                var[d] += ax[d].val[k] * q * q;
            }
        }
        if (var[d] == T(0)) return false;
        const T c = M.h / var[d];
#pragma unroll
        for (int k = 0; k < 3; ++k) ax[d].der[k] = ax[d].val[k] * ((r[d][k] - u[d]) * c);
    }
    return true;
}

// Basis state of one particle, ready for per-node evaluation in a transfer.
// WLS: u and var of wls_correct, `cut` if the mesh cuts the support (u != 0).
template <int D, class T>
struct Basis {
    Axis<T> ax[D];
    T u[D], var[D];
    bool wls, cut;
};

// Prepare the basis of one particle. Returns false for an empty window.
template <int D, class T, bool ALLOW_WLS = true>
__device__ __forceinline__ bool prepare_basis(const DMesh<D, T>& M, int basis, const T* x, const GimpLen<T>& gl,
                                              Basis<D, T>& B, int* err) {
    if (basis_is_gimp(basis) && !(gl.ln >= T(0) && gl.ln <= T(1))) {
        atomicOr(err, ERR_GIMP_LENGTH);
        return false;
    }
    bool full = false, cut[3];
    if (!axis_weights<D, T>(M, basis, x, gl, B.ax, full, cut)) return false;
    B.cut = cut[0] || cut[1] || (D == 3 && cut[2]);
    if (basis_is_kc(basis) && !full) {
        T r[3][3] = {};
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int k = 0; k < 3; ++k) r[d][k] = node_coord(M, d, B.ax[d].lo + k) - x[d];
        if (!kc_correct<D, T>(M, basis == TB_KC_BSPLINE_QUADRATIC, r, B.ax)) {
            atomicOr(err, ERR_WLS_SINGULAR);
            return false;
        }
    }
    B.wls = ALLOW_WLS && (basis == TB_WLS_BSPLINE_QUADRATIC || basis == TB_WLS_UGIMP);
    if constexpr (ALLOW_WLS) if (B.wls) {
        if constexpr (sizeof(T) == 4) {
            // FP32 positions: node coordinates rounded one by one leave sum w and
            // sum w r off by eps |x| / h, 1e-5 on the dam break, which the moments put
            // right on every axis wherever WLS fits them: uGIMP, and B-spline windows
            // that the mesh cuts (a whole B-spline support has the closed form). On the
            // cut axes alone the dam break's 100-step error in v was 3e-5 instead of
            // 1e-6, and N summed to 1 +- 1e-4 beside the walls at |x| / h = 1300. In FP64
            // the same is 1e-13 there and the errors of whole steps against 64 bits do
            // not change, while the moments on every axis cost two FP64 WLS(uGIMP) steps
            // of 2.6 M particles 3.02 against 2.61 ms (G2P's row loop).
            if (basis == TB_WLS_UGIMP || B.cut) B.cut = cut[0] = cut[1] = cut[2] = true;
        }
        T r[3][3] = {};
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int k = 0; k < 3; ++k) r[d][k] = node_coord(M, d, B.ax[d].lo + k) - x[d];
        if (!wls_correct<D, T>(M, basis == TB_WLS_BSPLINE_QUADRATIC, cut, r, B.ax, B.u, B.var)) {
            atomicOr(err, ERR_WLS_SINGULAR);
            return false;
        }
    }
    return true;
}

// FP64-position form: the window and the 1-D jets of a particle whose position
// is FP64. xi = (x - xmin) h_inv and the in-cell offsets are computed in FP64;
// only the offset from the window's first node, a number in [0, 3), is rounded
// to T before the jets are evaluated, so the weights carry T's relative
// precision of that offset rather than of the absolute coordinate. Window rules
// as axis_window.
template <int D, class T>
__device__ __forceinline__ bool axis_window_x64(const DMesh<D, T>& M, int basis, const double* x, double lnorm,
                                                double* xi, int* lo, int* cnt, bool* cut = nullptr) {
    bool inside = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        xi[d] = (x[d] - M.xmin64[d]) * M.h_inv64;
        inside = inside && xi[d] >= 0.0 && xi[d] < double(M.n[d] - 1);  // floor(xi) in [0, n - 2]
    }
    if (!inside) return false;
    const bool gimp = basis_is_gimp(basis);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        int st, e;
        if (gimp) {
            const double r = 1.0 + lnorm / 2.0;
            st = int(floor(xi[d] - r)) + 1;
            e = int(floor(xi[d] + r));
        } else {
            st = int(floor(xi[d] - 0.5));
            e = st + 2;
        }
        lo[d] = max(st, 0);
        cnt[d] = min(e, M.n[d] - 1) - lo[d] + 1;
        if (cut) cut[d] = st < 0 || e > M.n[d] - 1;
    }
    return true;
}

template <int D, class T, bool ALLOW_WLS = false>
__device__ __forceinline__ bool prepare_basis_x64(const DMesh<D, T>& M, int basis, const double* x,
                                                  const GimpLen<T>& gl, Basis<D, T>& B, int* err) {
    const bool gimp = basis_is_gimp(basis);
    if (gimp && !(gl.ln64 >= 0.0 && gl.ln64 <= 1.0)) {
        atomicOr(err, ERR_GIMP_LENGTH);
        return false;
    }
    double xi[3];
    int lo[3], cnt[3];
    bool cut[3];
    if (!axis_window_x64<D, T>(M, basis, x, gl.ln64, xi, lo, cnt, cut)) return false;
    B.cut = cut[0] || cut[1] || (D == 3 && cut[2]);
    B.wls = ALLOW_WLS && (basis == TB_WLS_BSPLINE_QUADRATIC || basis == TB_WLS_UGIMP);
    bool full = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        B.ax[d].lo = lo[d];
        B.ax[d].cnt = cnt[d];
        full = full && cnt[d] == 3;
    }
    if (!gimp && full) {
        // the fast path's t = fract(xi - 1/2) is xi - 1/2 - lo, in [0, 1); kept
        // below 1 after rounding so that the jets stay on the FP64 window
#pragma unroll
        for (int d = 0; d < D; ++d) {
            T t = T(xi[d] - 0.5 - double(lo[d]));
            if (t >= T(1)) t = T(1) - T(1) / T(1 << 24);
            bspline_quadratic_poly(t, B.ax[d].val, B.ax[d].der);
        }
        if (!B.wls) return true;
    }
    // offsets xi - (lo + k) of the particle from its window's nodes in FP64,
    // rounded once to T: the jets' argument and, times -h, X_{lo+k} - x_p
    T r[3][3] = {};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const double t = xi[d] - double(lo[d]);
        const T xn[3] = {T(t), T(t - 1.0), T(t - 2.0)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            r[d][k] = -xn[k] * M.h;
            if (gimp || !full) {
                T v = T(0), g = T(0);
                if (k < cnt[d]) {
                    if (gimp) jet_ugimp(xn[k], gl.ln, gl.il, v, g);
                    else jet_bspline_quadratic(xn[k], v, g);
                }
                B.ax[d].val[k] = v;
                B.ax[d].der[k] = g;
            }
        }
    }
    bool ok = true;
    if (basis_is_kc(basis)) {
        if (!full) ok = kc_correct<D, T>(M, basis == TB_KC_BSPLINE_QUADRATIC, r, B.ax);
    } else if constexpr (ALLOW_WLS) {
        if (B.wls) ok = wls_correct<D, T>(M, basis == TB_WLS_BSPLINE_QUADRATIC, cut, r, B.ax, B.u, B.var);
    }
    if (!ok) atomicOr(err, ERR_WLS_SINGULAR);
    return ok;
}

// The uGIMP length of particle p (its own, or the scene's).
template <int D, class T>
__device__ __forceinline__ GimpLen<T> gimp_len(const DMesh<D, T>& M, const PView<T>& P, const Scalars<T>& s, long long p) {
    if (!P.l) return s.gimp;
    GimpLen<T> g;
    const T l = P.l[p];
    g.ln = l / M.h;
    g.il = T(1) / g.ln;
    g.ln64 = double(l) / M.h64;
    return g;
}

// w and grad w at window slot (i, j, k).
template <int D, class T>
__device__ __forceinline__ void eval_node(const DMesh<D, T>& M, const Basis<D, T>& B, int i, int j, int k, T& w,
                                          T* dw) {
    node_weight<D, T>(M, B.ax, i, j, k, w, dw);
    if (B.wls) {
#pragma unroll
        for (int d = 0; d < D; ++d) w -= B.u[d] * dw[d];
    }
}

// Eigen-decomposition of a symmetric 3x3 matrix by cyclic Jacobi rotations
// (Golub & Van Loan, Matrix Computations, 4th ed., Algorithms 8.5.1-8.5.3):
// A = V diag(e) V^T, eigenvectors in the columns of V; stops when the
// off-diagonal part falls below 1e-15 of the matrix norm (at most 20 sweeps).
__device__ __forceinline__ void sym_eigen3(double (&a)[3][3], double (&e)[3], double (&V)[3][3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) V[r][c] = (r == c) ? 1.0 : 0.0;
    double fro = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) fro += a[r][c] * a[r][c];
    for (int sweep = 0; sweep < 20; ++sweep) {
        const double off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
        if (off <= 1e-30 * fro) break;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            if (a[p][q] == 0.0) continue;
            const double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
            const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double akp = a[k][p], akq = a[k][q];
                a[k][p] = c * akp - sn * akq;
                a[k][q] = sn * akp + c * akq;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double apk = a[p][k], aqk = a[q][k];
                a[p][k] = c * apk - sn * aqk;
                a[q][k] = sn * apk + c * aqk;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double vkp = V[k][p], vkq = V[k][q];
                V[k][p] = c * vkp - sn * vkq;
                V[k][q] = sn * vkp + c * vkq;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) e[k] = a[k][k];
}

// What the von Mises update takes from the trial left Cauchy-Green tensor b: the
// Kirchhoff stress deviator after the return map, the elastic left Cauchy-Green
// tensor after it and the plastic multiplier (symmetric: 11 21 31 22 32 33).
struct VonMisesReturn {
    double tau[6], be[6], dgam;
};

// The return map in principal logarithmic stretches by eigen-decomposition: for
// trial tensors far from spherical. Not inlined; few particles come here.
static __device__ __noinline__ void vonmises_eigen(const double* b, double lJ, double mu, double hardening, double flow,
                                                   VonMisesReturn* o) {
    double a[3][3] = {{b[0], b[1], b[2]}, {b[1], b[3], b[4]}, {b[2], b[4], b[5]}}, ev[3], n[3][3];
    sym_eigen3(a, ev, n);
    double ls[3], tau[3], tt = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        ls[q] = 0.5 * log(ev[q]);
        tau[q] = 2.0 * mu * ls[q] - 2.0 * mu / 3.0 * lJ;
        tt += tau[q] * tau[q];
    }
    const double nrm = sqrt(1.5 * tt), f = nrm - flow;
    o->dgam = 0.0;
    if (f > 0.0) {
        o->dgam = f / (3.0 * mu + hardening);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double deps = o->dgam * (1.5 * tau[q] / nrm);
            ev[q] = exp(2.0 * (ls[q] - deps));
            tau[q] -= 2.0 * mu * deps;
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c <= r; ++c) {
            double t = 0.0, e = 0.0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                t += tau[q] * n[r][q] * n[c][q];
                e += ev[q] * n[r][q] * n[c][q];
            }
            o->tau[symidx<3>(r, c)] = t;
            o->be[symidx<3>(r, c)] = e;
        }
}

// Square of a symmetric 3x3 matrix, and p(A) = r[0] I + r[1] A + r[2] A^2.
__device__ __forceinline__ void sym_square(const double (&a)[6], double (&q)[6]) {
    q[0] = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    q[1] = a[1] * a[0] + a[3] * a[1] + a[4] * a[2];
    q[2] = a[2] * a[0] + a[4] * a[1] + a[5] * a[2];
    q[3] = a[1] * a[1] + a[3] * a[3] + a[4] * a[4];
    q[4] = a[2] * a[1] + a[4] * a[3] + a[5] * a[4];
    q[5] = a[2] * a[2] + a[4] * a[4] + a[5] * a[5];
}

__device__ __forceinline__ double sym_det(const double (&a)[6]) {
    return a[0] * (a[3] * a[5] - a[4] * a[4]) - a[1] * (a[1] * a[5] - a[4] * a[2]) + a[2] * (a[1] * a[4] - a[3] * a[2]);
}

// sum_k coef(k) A^k, k = 0 .. N, of a traceless symmetric 3x3 matrix A with
// j2 = tr(A^2) / 2, j3 = det A, as r[0] I + r[1] A + r[2] A^2: Horner's rule, where
// by Cayley-Hamilton A^3 = j2 A + j3 I, so a step is two multiply-adds.
template <int N, class Coef>
__device__ __forceinline__ void traceless_series(double j2, double j3, Coef coef, double (&r)[3]) {
    r[0] = coef(N);
    r[1] = r[2] = 0.0;
#pragma unroll
    for (int k = N - 1; k >= 0; --k) {
        const double t = r[1];
        r[1] = r[0] + r[2] * j2;
        r[0] = r[2] * j3 + coef(k);
        r[2] = t;
    }
}

// The von Mises update of the Taylor impact (docs/src/gpu.md:352-391), one
// particle, FP64 throughout: F = dF F is given. Hencky elasticity on the trial
// left Cauchy-Green tensor b = F Cp^-1 F^T; yield f = sqrt(3/2 tau'.tau') -
// (tau_y0 + H eps_p) on the Kirchhoff deviator tau = mu log b - 2 mu / 3 log J;
// return map Delta gamma = f / (3 mu + H) along df/dtau in principal logarithmic
// stretches; pressure kappa log J / J with kappa = lambda + 2 mu / 3. Writes
// sigma, Cp^-1 = F^-1 b_e F^-T, eps_p and V = det(dF) V. The G2P kernels that
// call it are instantiated apart from the elastic ones.
//
// All of it are functions of one symmetric matrix. Elastic strains are small in
// shear (the yield stress is a fraction of a percent of mu), so with s = tr b / 3 and
// the traceless E = b / s - I, |E| <= 0.1 (Frobenius; eigenvalues within 0.082),
// log(I + E) and the exponential back are Taylor series of 16 and 11 terms (to 1e-17),
// evaluated in the basis I, E, E^2. Others take the eigen-decomposition. The Jacobi
// rotations of every particle bounded the Taylor impact's G2P (1.48 M particles,
// FP32): 0.379 ms, 0.213 ms with the series.
template <class T>
__device__ __forceinline__ void vonmises_update(const PView<T>& P, const Scalars<T>& s, long long p,
                                             const double (&F)[3][3], double detdF, double lam, double mu) {
    const double kappa = lam + 2.0 * mu / 3.0;
    const double J = F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) -
                     F[0][1] * (F[1][0] * F[2][2] - F[1][2] * F[2][0]) +
                     F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]);
    const double iJ = 1.0 / J;
    const double lJ = log(J);
    const double pr = kappa * lJ * iJ;
    double b[6];
    {
        double Cp[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) Cp[k] = double(P.Cp_inv[k][p]);
        double FC[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                FC[r][c] = F[r][0] * Cp[symidx<3>(0, c)] + F[r][1] * Cp[symidx<3>(1, c)] + F[r][2] * Cp[symidx<3>(2, c)];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = c; r < 3; ++r)
                b[symidx<3>(r, c)] = FC[r][0] * F[c][0] + FC[r][1] * F[c][1] + FC[r][2] * F[c][2];
    }
    const double epn = double(P.eps_p[p]), flow = s.yield_stress + s.hardening * epn;
    double tau[6], be[6], dgam = 0.0;
    const double sb = (b[0] + b[3] + b[5]) * (1.0 / 3.0), isb = 1.0 / sb;
    double E[6], E2[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) E[k] = b[k] * isb - ((k == 0 || k == 3 || k == 5) ? 1.0 : 0.0);
    sym_square(E, E2);
    const double j2 = 0.5 * (E2[0] + E2[3] + E2[5]);
    if (j2 <= 0.005) {
        double c[3];
        traceless_series<15>(j2, sym_det(E), [](int k) { return k == 0 ? 0.0 : (k & 1 ? 1.0 : -1.0) / double(k); }, c);
        const double t0 = mu * (log(sb) + c[0]) - 2.0 * mu / 3.0 * lJ, t1 = mu * c[1], t2 = mu * c[2];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            tau[k] = t1 * E[k] + t2 * E2[k] + ((k == 0 || k == 3 || k == 5) ? t0 : 0.0);
            be[k] = b[k];
        }
        const double tt = tau[0] * tau[0] + tau[3] * tau[3] + tau[5] * tau[5] +
                          2.0 * (tau[1] * tau[1] + tau[2] * tau[2] + tau[4] * tau[4]);
        const double nrm = sqrt(1.5 * tt), f = nrm - flow;
        if (f > 0.0) {
            dgam = f / (3.0 * mu + s.hardening);
            const double q = 1.5 * dgam / nrm;
            // log b_e = log b - 2 q tau = (1/mu - 2 q) tau + 2/3 log J I
            const double w = 1.0 / mu - 2.0 * q, tm = (tau[0] + tau[3] + tau[5]) * (1.0 / 3.0);
            double Dv[6], D2[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) Dv[k] = w * (tau[k] - ((k == 0 || k == 3 || k == 5) ? tm : 0.0));
            sym_square(Dv, D2);
            traceless_series<10>(0.5 * (D2[0] + D2[3] + D2[5]), sym_det(Dv),
                                 [](int k) {
                                     double v = 1.0;
                                     for (int i = 2; i <= k; ++i) v /= double(i);
                                     return v;
                                 },
                                 c);
            const double ex = exp(w * tm + 2.0 / 3.0 * lJ);
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                be[k] = ex * (c[1] * Dv[k] + c[2] * D2[k] + ((k == 0 || k == 3 || k == 5) ? c[0] : 0.0));
                tau[k] *= 1.0 - 2.0 * mu * q;
            }
        }
    } else {
        VonMisesReturn o;
        double bt[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) bt[k] = b[k];
        vonmises_eigen(bt, lJ, mu, s.hardening, flow, &o);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            tau[k] = o.tau[k];
            be[k] = o.be[k];
        }
        dgam = o.dgam;
    }
    double Fi[3][3];
    Fi[0][0] = (F[1][1] * F[2][2] - F[1][2] * F[2][1]) * iJ;
    Fi[0][1] = (F[0][2] * F[2][1] - F[0][1] * F[2][2]) * iJ;
    Fi[0][2] = (F[0][1] * F[1][2] - F[0][2] * F[1][1]) * iJ;
    Fi[1][0] = (F[1][2] * F[2][0] - F[1][0] * F[2][2]) * iJ;
    Fi[1][1] = (F[0][0] * F[2][2] - F[0][2] * F[2][0]) * iJ;
    Fi[1][2] = (F[0][2] * F[1][0] - F[0][0] * F[1][2]) * iJ;
    Fi[2][0] = (F[1][0] * F[2][1] - F[1][1] * F[2][0]) * iJ;
    Fi[2][1] = (F[0][1] * F[2][0] - F[0][0] * F[2][1]) * iJ;
    Fi[2][2] = (F[0][0] * F[1][1] - F[0][1] * F[1][0]) * iJ;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double m[3];  // row r of F^-1 b_e
#pragma unroll
        for (int c = 0; c < 3; ++c)
            m[c] = Fi[r][0] * be[symidx<3>(0, c)] + Fi[r][1] * be[symidx<3>(1, c)] + Fi[r][2] * be[symidx<3>(2, c)];
#pragma unroll
        for (int c = 0; c <= r; ++c) {
            P.sig[symidx<3>(r, c)][p] = T(tau[symidx<3>(r, c)] * iJ + (r == c ? pr : 0.0));
            P.Cp_inv[symidx<3>(r, c)][p] = T(m[0] * Fi[c][0] + m[1] * Fi[c][1] + m[2] * Fi[c][2]);
        }
    }
    P.eps_p[p] = T(epn + dgam);
    P.V[p] = T(detdF * double(P.V[p]));
}

// FP64 particle kinematics and constitutive update (README.md:82-86):
// F = (I + dt grad_v) F, J = det F, sigma by Neo-Hookean or the weakly
// compressible fluid p = -K (J - 1), V = V0 J; or, in 3D, the von Mises model
// of the Taylor impact with V = det(I + dt grad_v) V (vonmises_update). F, J
// and log J stay in FP64.
template <int D, class T>
__device__ __forceinline__ void load_F(const PView<T>& P, long long p, double (&F)[3][3]) {
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) F[r][c] = P.F[r + c * D][p];
}

// F is passed in (the caller chooses when to load it).
template <int D, class T, bool VM = false>
__device__ __forceinline__ void particle_update(const PView<T>& P, const Scalars<T>& s, long long p,
                                                const T (&gv)[3][3], const double (&F)[3][3]) {
    double Fn[3][3];
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) {
            double a = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                double Ark = (r == k ? 1.0 : 0.0) + double(gv[r][k]) * s.dt64;
                a += Ark * F[k][c];
            }
            Fn[r][c] = a;
        }
    double J;
    if constexpr (D == 3)
        J = Fn[0][0] * (Fn[1][1] * Fn[2][2] - Fn[1][2] * Fn[2][1]) -
            Fn[0][1] * (Fn[1][0] * Fn[2][2] - Fn[1][2] * Fn[2][0]) +
            Fn[0][2] * (Fn[1][0] * Fn[2][1] - Fn[1][1] * Fn[2][0]);
    else
        J = Fn[0][0] * Fn[1][1] - Fn[0][1] * Fn[1][0];
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) P.F[r + c * D][p] = Fn[r][c];
    const double mu = P.mu ? double(P.mu[p]) : s.mu;
    const double lam = P.lam ? double(P.lam[p]) : s.lam;
    if constexpr (D == 3 && VM) {
        {
            double dF[3][3];
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = 0; c < 3; ++c) dF[r][c] = (r == c ? 1.0 : 0.0) + double(gv[r][c]) * s.dt64;
            const double detdF = dF[0][0] * (dF[1][1] * dF[2][2] - dF[1][2] * dF[2][1]) -
                                 dF[0][1] * (dF[1][0] * dF[2][2] - dF[1][2] * dF[2][0]) +
                                 dF[0][2] * (dF[1][0] * dF[2][1] - dF[1][1] * dF[2][0]);
            vonmises_update<T>(P, s, p, Fn, detdF, lam, mu);
            return;
        }
    }
    if (s.material == 1) {
        const double pr = lam * (J - 1.0);
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
            for (int c = 0; c <= r; ++c) P.sig[symidx<D>(r, c)][p] = T(r == c ? pr : 0.0);
    } else {
        // sigma = (mu (F F^T - I) + lambda log J I) / J, the division by J taken
        // once as a reciprocal (one rounding more than six divisions)
        const double lj = log(J);
        const double iJ = 1.0 / J;
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
            for (int c = 0; c <= r; ++c) {
                double b = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) b += Fn[r][k] * Fn[c][k];
                double sg = (mu * (b - (r == c ? 1.0 : 0.0)) + (r == c ? lam * lj : 0.0)) * iJ;
                P.sig[symidx<D>(r, c)][p] = T(sg);
            }
    }
    const double V0 = P.V0 ? double(P.V0[p]) : s.V0_64;
    P.V[p] = T(V0 * J);
}

}  // namespace tb
