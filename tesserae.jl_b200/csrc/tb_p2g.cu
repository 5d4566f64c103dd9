// tb_p2g.cu -- block-scheduled P2G scatter of m, mv and f
// (Tesserae.jl src/Transfer/gpu.jl:139-223; equations README.md:72-74,
// test/transfer.jl:96-97 for gravity, docs/src/transfer.md:176-178 for APIC).
//
// One CTA per non-empty grid block or piece of one (grid-stride over the device
// block list). The block's particles reach the (BW+3)^D-node halo tile
// [BW b - 1, BW b + BW + 1] per axis; every support window starts at one of
// (BW+1)^D tile positions ("groups"; particles of a group share their window; a
// row of groups along x is a "pencil"). Every kernel here
//   1. counts a batch of the block's particles into groups (shared counters give
//      each its rank) and writes a record per particle at its group-sorted slot;
//   2. sweeps the records: a lane keeps the sums of a few nodes of one pencil or
//      group in registers and leaves them, with plain stores, in its own slots of
//      a staging array;
//   3. sums, one thread per tile node, the at most 3^(D-1) staged partials that
//      reach the node and adds it to the grid with one global atomic per non-zero
//      value (gravity, sum w m g = g sum w m, from the summed mass).
// The kernels differ in what a lane owns:
//   p2g_plane_kernel      3D FP32, quadratic B-spline, FLIP: one z-slot of a pencil
//                         (3 x 3 nodes of 3 rows), short records
//   p2g_pencil_kernel     3D, everything else: one window row of a pencil (3 nodes)
//   p2g_2d_kernel         2D: one window row of one group
#include <type_traits>

#include "tb_launch.cuh"

namespace tb {

namespace {

template <class T>
struct PairOf;
template <>
struct PairOf<float> {
    using type = float2;
};
template <>
struct PairOf<double> {
    using type = double2;
};
__device__ __forceinline__ float2 pair(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 pair(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double2 pfma(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ double2 pmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ double2 padd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void st2(double* p, double a, double b) {
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

// Window start per axis (and, for axis_window's kernels, whether the particle
// takes part): shared by the kernels whose records hold full jets.
template <int D, class T, bool X64>
__device__ __forceinline__ bool window_start(const DMesh<D, T>& M, const Scalars<T>& s, const double* xd, const T* x,
                                             const GimpLen<T>& gl, int (&lo)[3], int* err) {
    int cnt[3];
    const bool gimp = basis_is_gimp(s.basis);
    if constexpr (X64) {
        if (gimp && !(gl.ln64 >= 0.0 && gl.ln64 <= 1.0)) {
            atomicOr(err, ERR_GIMP_LENGTH);
            return false;
        }
        double xi[3];
        return axis_window_x64<D, T>(M, s.basis, xd, gl.ln64, xi, lo, cnt);
    } else {
        if (gimp && !(gl.ln >= T(0) && gl.ln <= T(1))) {
            atomicOr(err, ERR_GIMP_LENGTH);
            return false;
        }
        T xi[3];
        return axis_window<D, T>(M, s.basis, x, gl.ln, xi, lo, cnt);
    }
}

// Whether a position lies in the mesh (findblock's rule). Every particle of a fresh
// partition does; one that has left the mesh since the binning has no support there.
template <int D, class T, bool X64>
__device__ __forceinline__ bool inside_mesh(const DMesh<D, T>& M, const double* xd, const T* x) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        if constexpr (X64) {
            const double xi = (xd[d] - M.xmin64[d]) * M.h_inv64;
            in = in && xi >= 0.0 && xi < double(M.n[d] - 1);
        } else {
            const T xi = (x[d] - M.xmin[d]) * M.h_inv;
            in = in && xi >= T(0) && xi < T(M.n[d] - 1);
        }
    }
    return in;
}

// Unclipped window start floor(xi - 1/2) of a quadratic B-spline on one axis and
// t = fract(xi - 1/2) (bspline.jl:28-40, 90-100). A B-spline's value at a node does
// not depend on which others exist, so a window that the mesh cuts keeps its
// place in the tile and its sums for nodes outside the mesh are dropped at the end.
template <int D, class T, bool X64>
__device__ __forceinline__ int bspline_start(const DMesh<D, T>& M, int d, double xd, T x, T& t) {
    if constexpr (X64) {
        const double u64 = (xd - M.xmin64[d]) * M.h_inv64 - 0.5;
        const double fl = floor(u64);
        t = T(u64 - fl);
        if (t >= T(1)) t = T(1) - T(1) / T(1 << 24);
        return int(fl);
    } else {
        const T uu = (x - M.xmin[d]) * M.h_inv - T(0.5);
        const T fl = floor(uu);
        t = uu - fl;
        return int(fl);
    }
}

// Shared memory attributes and the grid of a block-scheduled kernel: every CTA
// the GPU holds, at most eight per block (blocks may be split, block_pieces).
template <class K>
cudaError_t prepare_launch(K kern, int threads, size_t smem, const LaunchCfg& cfg, int nblocks, int& grid) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, int(cudaSharedmemCarveoutMaxShared));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    grid = std::min(cfg.num_sms * std::max(per_sm, 1), 8 * nblocks);
    return e;
}

// Coefficients of the quadratic B-spline slot k as a + t (b + t c) and its
// derivative e + t f (bspline_quadratic_poly, slot by slot).
template <class T>
struct SlotPoly {
    T a, b, c, e, f;
};
template <class T>
__device__ __forceinline__ SlotPoly<T> slot_poly(int k) {
    if (k == 0) return {T(0.5), T(-1), T(0.5), T(-1), T(1)};
    if (k == 1) return {T(0.5), T(1), T(-1), T(1), T(-2)};
    return {T(0), T(0), T(0.5), T(0), T(1)};
}

// Staging layout: partial (component c, row jk, pencil pc, tile x) at
// ((c * NJK + jk) * NPENCIL + pc) * TS + x (components in pairs). For one row offset jk the pencils
// (gy, gz) of a tile plane follow each other, so the gather's reads for
// consecutive tile nodes are consecutive words (no bank conflicts within a
// plane).
template <int D, int BW>
struct PencilShape {
    static constexpr int TS = BW + 3;
    static constexpr int TN = (D == 3) ? TS * TS * TS : TS * TS;
    static constexpr int NC = 1 + 2 * D;
    static constexpr int G1 = BW + 1;
    static constexpr int NG = (D == 3) ? G1 * G1 * G1 : G1 * G1;
    static constexpr int NJK = (D == 3) ? 9 : 3;
    static constexpr int NSUB = 32 / NJK;
    static constexpr int NPENCIL = NG / G1;
    static constexpr int NPART = NC * NPENCIL * NJK * TS;
};

// Record kinds and their layout in words of T (pairs, for packed arithmetic;
// S = -V sigma in Tensorial order 11 21 31 22 32 33 = S0..S5):
//   0 (m, m v_x)  2 (m v_y, m v_z)  4 (S0, S1)  6 (S1, S3)  8 (S2, S4)
//   P_BSP   quadratic B-spline, FLIP: 10 (S5, t_z) 12 (t_x, t_y), t = fract(xi - 1/2)
//           per axis (bspline_start); the lanes evaluate the jets
//   others  10 (S5, u_x) and the (w, g = grad) jets of each axis slot:
//           12 + 2k z, 18 + 2j y, 24 + 2i x
//   P_JET   uGIMP, KernelCorrection, FLIP
//   P_WLS   WLS, FLIP: 30 (u_y, u_z)
//   P_APIC, P_WLS_APIC: then (By, Bz) of columns 0..2, (Bx0, Bx1), (Bx2, r0_x),
//           (r0_y, r0_z) with B = m D^-1 B_p, D^-1 = 4/h^2 I, r0 = X_lo - x_p
// With the closed-form WLS weights (wls_correct) every gradient is a product of
// per-axis jets and N_i = W_i - u . G_i, so per window row (y, z fixed)
//   N_x = wx R + gx Q,  R = wyz - uy gyz - uz wgz,  Q = -ux wyz
//   (wyz = wy wz, gyz = gy wz, wgz = wy gz),
//   f   += gx S[:,0] wyz + wx (S[:,1] gyz + S[:,2] wgz),
//   mv  += N_x (m v_p + B[:,0] rx + B[:,1] ry + B[:,2] rz).
enum : int { P_BSP = 0, P_JET = 1, P_WLS = 2, P_WLS_APIC = 3, P_APIC = 4 };

template <int KIND>
struct RecOf {
    static constexpr bool WLS = KIND == P_WLS || KIND == P_WLS_APIC, APIC = KIND == P_WLS_APIC || KIND == P_APIC;
    static constexpr int WZ = 12, WY = 18, WX = 24, UYZ = 30;
    static constexpr int DB = WLS ? 32 : 30;
    // an odd number of pairs, so that neighbouring records fall on different banks
    static constexpr int SIZE = KIND == P_BSP ? 14 : (APIC ? DB + 12 + (KIND == P_WLS_APIC ? 2 : 0) : (WLS ? 34 : 30));
};

// One record's contribution to row (j, k) of its window.
template <class T, int KIND>
__device__ __forceinline__ void accumulate(const T* rec, int j, int k, const SlotPoly<T>& py, const SlotPoly<T>& pz,
                                           T h, T h_inv, typename PairOf<T>::type (&a01)[3],
                                           typename PairOf<T>::type (&a23)[3], typename PairOf<T>::type (&f01)[3],
                                           T (&f2)[3]) {
    using T2 = typename PairOf<T>::type;
    using R = RecOf<KIND>;
    const T2* r = reinterpret_cast<const T2*>(rec);
    T2 u01 = r[0], u23 = r[1];
    const T2 sa = r[2], sb = r[3], sc = r[4], s5u = r[5];
    T wx[3], gx[3], wy, gy, wz, gz;
    if constexpr (KIND == P_BSP) {
        const T2 txy = r[6];
        const T ty = txy.y, tz = s5u.y;
        bspline_quadratic_poly(txy.x, wx, gx);
#pragma unroll
        for (int i = 0; i < 3; ++i) gx[i] *= h_inv;
        wy = py.a + ty * (py.b + ty * py.c);
        gy = (py.e + ty * py.f) * h_inv;
        wz = pz.a + tz * (pz.b + tz * pz.c);
        gz = (pz.e + tz * pz.f) * h_inv;
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const T2 q = r[R::WX / 2 + i];
            wx[i] = q.x;
            gx[i] = q.y;
        }
        const T2 qy = r[R::WY / 2 + j], qz = r[R::WZ / 2 + k];
        wy = qy.x;
        gy = qy.y;
        wz = qz.x;
        gz = qz.y;
    }
    const T wyz = wy * wz, gyz = gy * wz, wgz = wy * gz;
    T rr = wyz, qq = T(0);
    if constexpr (R::WLS) {
        const T2 uyz = r[R::UYZ / 2];
        rr = wyz - uyz.x * gyz - uyz.y * wgz;
        qq = -s5u.y * wyz;
    }
    T rx[3] = {T(0), T(0), T(0)}, bx0 = T(0);
    T2 c0 = pair(T(0), T(0));
    if constexpr (R::APIC) {
        c0 = r[R::DB / 2];
        const T2 bx = r[R::DB / 2 + 3], b2 = r[R::DB / 2 + 4], ryz = r[R::DB / 2 + 5];
        const T ry = ryz.x + T(j) * h, rz = ryz.y + T(k) * h;
        bx0 = bx.x;
        u01.y += bx.y * ry + b2.x * rz;
        u23 = pfma(r[R::DB / 2 + 2], pair(rz, rz), pfma(r[R::DB / 2 + 1], pair(ry, ry), u23));
#pragma unroll
        for (int i = 0; i < 3; ++i) rx[i] = b2.y + T(i) * h;
    }
    if constexpr (KIND == P_BSP || KIND == P_JET) {
        // the row's (m, m v) times wyz once; each x-slot then needs one FMA per pair
        u01 = pmul(u01, pair(wyz, wyz));
        u23 = pmul(u23, pair(wyz, wyz));
    }
    const T2 fa01 = pmul(sa, pair(wyz, wyz));
    const T2 fb01 = pfma(sc, pair(wgz, wgz), pmul(sb, pair(gyz, gyz)));
    const T fa2 = sc.x * wyz, fb2 = s5u.x * wgz + sc.y * gyz;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        T N = wx[i];
        T2 n01 = u01, n23 = u23;
        if constexpr (KIND != P_BSP && KIND != P_JET) {
            N *= rr;
            if constexpr (R::WLS) N += gx[i] * qq;
            if constexpr (R::APIC) {
                n01.y += bx0 * rx[i];
                n23 = pfma(c0, pair(rx[i], rx[i]), n23);
            }
        }
        a01[i] = pfma(pair(N, N), n01, a01[i]);
        a23[i] = pfma(pair(N, N), n23, a23[i]);
        f01[i] = pfma(pair(gx[i], gx[i]), fa01, pfma(pair(wx[i], wx[i]), fb01, f01[i]));
        f2[i] += gx[i] * fa2 + wx[i] * fb2;
    }
}

// The fields of one particle that its record needs, loaded together.
template <class T, bool X64, int KIND>
struct Fields {
    static constexpr int D = 3;
    double xd[3];
    T x[3], v[3], V, m, sg[6], B[9];
    GimpLen<T> gl;
    __device__ __forceinline__ void load(const DMesh<3, T>& M, const PView<T>& P, const Scalars<T>& s, long long p,
                                         bool on) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            if constexpr (X64) xd[d] = on ? P.x64[d][p] : 0.0;
            else x[d] = on ? P.x[d][p] : T(0);
        }
        if constexpr (KIND != P_BSP) gl = on ? gimp_len(M, P, s, p) : s.gimp;
#pragma unroll
        for (int d = 0; d < D; ++d) v[d] = on ? P.v[d][p] : T(0);
        V = on ? P.V[p] : T(0);
        m = (on && P.m) ? P.m[p] : s.mass;
#pragma unroll
        for (int k = 0; k < 6; ++k) sg[k] = on ? P.sig[k][p] : T(0);
        if constexpr (RecOf<KIND>::APIC) {
#pragma unroll
            for (int k = 0; k < 9; ++k) B[k] = on ? P.B[k][p] : T(0);
        }
    }
    // Window start per axis (unclipped for P_BSP, whose t it also leaves in x);
    // false for a particle that takes no part (P_BSP, with STALE: outside the mesh).
    template <bool STALE>
    __device__ __forceinline__ bool window(const DMesh<3, T>& M, const Scalars<T>& s, int (&lo)[3], int* err) {
        if constexpr (KIND == P_BSP) {
            const bool in = !STALE || inside_mesh<D, T, X64>(M, xd, x);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                T t;
                lo[d] = bspline_start<D, T, X64>(M, d, xd[d], x[d], t);
                x[d] = t;
            }
            return in;
        } else {
            return window_start<D, T, X64>(M, s, xd, x, gl, lo, err);
        }
    }
    __device__ __forceinline__ void write(const DMesh<3, T>& M, const Scalars<T>& s, T* r, int* err) {
        using R = RecOf<KIND>;
        const T nV = -V;
        st2(r + 0, m, m * v[0]);
        st2(r + 2, m * v[1], m * v[2]);
        st2(r + 4, nV * sg[0], nV * sg[1]);
        st2(r + 6, nV * sg[1], nV * sg[3]);
        st2(r + 8, nV * sg[2], nV * sg[4]);
        const T s5 = nV * sg[5];
        if constexpr (KIND == P_BSP) {
            st2(r + 10, s5, x[2]);
            st2(r + 12, x[0], x[1]);
        } else {
            Basis<D, T> B_;
            bool in;
            if constexpr (X64) in = prepare_basis_x64<D, T, R::WLS>(M, s.basis, xd, gl, B_, err);
            else in = prepare_basis<D, T, R::WLS>(M, s.basis, x, gl, B_, err);
            if (!in) {  // a singular fit (reported): the particle adds nothing
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    B_.u[d] = T(0);
                    B_.ax[d].lo = 0;
#pragma unroll
                    for (int k = 0; k < 3; ++k) B_.ax[d].val[k] = B_.ax[d].der[k] = T(0);
                }
            }
            st2(r + 10, s5, R::WLS ? B_.u[0] : T(0));
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                st2(r + R::WZ + 2 * k, B_.ax[2].val[k], B_.ax[2].der[k] * M.h_inv);
                st2(r + R::WY + 2 * k, B_.ax[1].val[k], B_.ax[1].der[k] * M.h_inv);
                st2(r + R::WX + 2 * k, B_.ax[0].val[k], B_.ax[0].der[k] * M.h_inv);
            }
            if constexpr (R::WLS) st2(r + R::UYZ, B_.u[1], B_.u[2]);
            if constexpr (R::APIC) {
                T r0[3] = {T(0), T(0), T(0)};
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    if constexpr (X64) r0[d] = T(__dadd_rn(M.xmin64[d], __dmul_rn(double(B_.ax[d].lo), M.h64)) - xd[d]);
                    else r0[d] = node_coord(M, d, B_.ax[d].lo) - x[d];
                }
                const T md = m * (T(4) / (M.h * M.h));
#pragma unroll
                for (int c = 0; c < 3; ++c) st2(r + R::DB + 2 * c, md * B[1 + 3 * c], md * B[2 + 3 * c]);
                st2(r + R::DB + 6, md * B[0], md * B[3]);
                st2(r + R::DB + 8, md * B[6], r0[0]);
                st2(r + R::DB + 10, r0[1], r0[2]);
            }
        }
    }
};

// ---------------------------------------------------------------------------
// Pencil kernel (3D): every kind but the FP32 B-spline. A lane owns one (y, z) row
// of a pencil's window, walks the pencil's groups in x order and keeps the row's
// 3 x-nodes (21 sums) in registers; 9 rows x 3 pencils fill a warp, 9 warps take
// the 25 pencils. After each group the x-node the window leaves for good is final
// for this (pencil, row) and is stored to the lane's own slot of the staging
// array. A block's later batches add to the staged sums, so the gather and the
// global atomics run once per block and piece. The staged partials of a node are
// summed in T for the general kinds (WLS, APIC), in FP64 for the others.
// What bounds it is the chain of a batch (load, rank, record, sweep of the longest
// pencil of a warp) at two CTAs of 9 warps per SM in FP32 and one in FP64, whose
// staging array takes 88 KB: issue slots are about a third used, so the general
// kinds take rows and not planes (9 nodes per lane: half of the lanes' work is
// shared, but each record's chain is twice as long and a third of the warps run).
// Dam break at half resolution (18.2 M particles, WLS(uGIMP) + APIC, FP32 with FP64
// positions): 6.03 ms with a moment inverse at every node of a plane lane, 4.04 ms
// with the closed form on plane lanes, 2.98 ms here. FP64 B-spline, 917 k particles:
// 0.196 ms with full records, 0.177 ms with compact ones.
constexpr int P2G_THREADS = 288;

// STALE (P_BSP): the partition may be older than the positions. A fresh one holds no
// particle outside the mesh, and the check costs a step of 125 k particles 2.5 us of 89.
template <class T, bool X64, int KIND, int NR, int CTAS, bool STALE>
__global__ void __launch_bounds__(P2G_THREADS, CTAS)
    p2g_pencil_kernel(DMesh<3, T> M, PView<T> P, GView<T> G, Scalars<T> s, const int* __restrict__ totals,
                      const int* __restrict__ blocklist, const int* __restrict__ offsets,
                      const int* __restrict__ perm, int* err, const int* __restrict__ list,
                      const unsigned long long* __restrict__ nlist) {
    chain_wait();
    using SH = PencilShape<3, 4>;
    using T2 = typename PairOf<T>::type;
    constexpr int NT = P2G_THREADS, NW = NT / 32, ITEMS = (NR + NT - 1) / NT, RS = RecOf<KIND>::SIZE;
    constexpr int TS = SH::TS, TN = SH::TN, NC = SH::NC, G1 = SH::G1, NG = SH::NG, NPENCIL = SH::NPENCIL;
    constexpr int NJK = SH::NJK, NSUB = 32 / NJK, NTASK = (NPENCIL + NSUB - 1) / NSUB;
    constexpr int CSTR = NPENCIL * NJK * TS;  // stride between staged components
    static_assert(NPENCIL <= 32, "pencil ranking runs in one warp");
    static_assert(NR % 8 == 0 && NT % 8 == 0, "passes in 8-particle chunks");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* rec = reinterpret_cast<T*>(smem_raw);
    // staged partials as (m, m v_x), (m v_y, m v_z), (f_x, f_y) pairs, then f_z.
    // Records of pencil pc start 2 pc words after their slot: pencils of equal size
    // would otherwise put the records a warp reads together in the same banks.
    constexpr int SKW = 2;
    T* part = rec + NR * RS + SKW * NPENCIL;
    T2* part2 = reinterpret_cast<T2*>(part);
    T* partz = part + 6 * CSTR;
    int* gcount = reinterpret_cast<int*>(part + NC * CSTR);
    int* gstart = gcount + NG;
    int* pslot = gstart + NG + 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int jk = lane % NJK, sub = lane / NJK, j = jk % 3, k = jk / 3;
    const SlotPoly<T> py = slot_poly<T>(j), pz = slot_poly<T>(k);
    const T2 z2 = pair(T(0), T(0));

    for (int g = tid; g < NG; g += NT) gcount[g] = 0;
    __syncthreads();

    const int nblk = list ? int(*nlist) : totals[0];
    int per = NR;
    const int split = block_pieces(totals, nblk, NR, gridDim.x, per);
    for (int vi = blockIdx.x; vi < nblk * split; vi += gridDim.x) {
        const int li = split == 1 ? vi : vi / split, piece = vi - li * split;
        const int b = list ? list[li] : blocklist[li] - 1;
        int org[3];
        {
            int r = b;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                org[d] = (r % M.nb[d]) * 4 - 1;
                r /= M.nb[d];
            }
        }
        const int s0 = offsets[b], s1 = offsets[b + 1];
        const BlockPasses bp(s0, s1, per);
        for (int bi = piece; bi < bp.count(); bi += split) {
            const int q0 = bp.pos(bi, tid), qstep = bp.step(NT);
            // ---- 1a. every global load of the batch first (the ids, then all of
            //      the particles' fields: two dependent round trips per batch), then
            //      group and rank; the fields stay in registers for 1b
            int pid[ITEMS], grp[ITEMS], rank[ITEMS];
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const int ti = tid + u * NT, q = q0 + u * qstep;
                pid[u] = (ti < per && q < s1) ? perm[q] - 1 : -1;
            }
            Fields<T, X64, KIND> f[ITEMS];
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) f[u].load(M, P, s, pid[u] >= 0 ? pid[u] : 0, pid[u] >= 0);
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                grp[u] = -1;
                rank[u] = 0;
                int lo[3];
                if (pid[u] < 0) continue;
                const bool in = f[u].template window<STALE>(M, s, lo, err);
                if (KIND != P_BSP && !in) continue;
                int gi = 0;
                bool ok = true;
#pragma unroll
                for (int d = 2; d >= 0; --d) {
                    const int q = lo[d] - org[d];
                    ok = ok && q >= 0 && q < G1;
                    gi = gi * G1 + q;
                }
                if (!ok || !in) {
                    if (in) atomicOr(err, ERR_TILE_RANGE);
                    continue;
                }
                grp[u] = gi;
                rank[u] = atomicAdd(&gcount[gi], 1);
            }
            __syncthreads();
            if (warp == 0) {
                int carry = 0;
#pragma unroll
                for (int g0 = 0; g0 < NG; g0 += 32) {
                    const int g = g0 + lane;
                    const int c = g < NG ? gcount[g] : 0;
                    int incl = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    if (g < NG) gstart[g] = carry + incl - c;
                    carry += __shfl_sync(0xffffffffu, incl, 31);
                }
                if (lane == 0) gstart[NG] = carry;
            } else if (warp == 1) {
                // pencil slots by size, largest first: the pencils a warp sweeps in
                // lockstep then have similar lengths
                const int myp = lane < NPENCIL ? lane : -1;
                int mysize = 0;
                if (myp >= 0) {
                    const int gb = G1 * myp;
#pragma unroll
                    for (int gx = 0; gx < G1; ++gx) mysize += gcount[gb + gx];
                }
                int rk = 0;
                for (int o = 0; o < NPENCIL; ++o) {
                    const int os = __shfl_sync(0xffffffffu, mysize, o);
                    rk += (os > mysize) || (os == mysize && o < lane);
                }
                if (myp >= 0) pslot[rk] = myp;
            }
            __syncthreads();
            // ---- 1b. records at their group-sorted slots
            for (int g = tid; g < NG; g += NT) gcount[g] = 0;  // ready for the next batch
#pragma unroll
            for (int u = 0; u < ITEMS; ++u)
                if (grp[u] >= 0) f[u].write(M, s, rec + (gstart[grp[u]] + rank[u]) * RS + SKW * (grp[u] / G1), err);
            __syncthreads();
            // ---- 2. pencil sweeps; every live (pencil, row) stages all TS x-nodes
            for (int task = warp; task < NTASK; task += NW) {
                const int slot = task * NSUB + sub;
                if (sub >= NSUB || slot >= NPENCIL) continue;
                const int pc = pslot[slot];
                const int gbase = G1 * pc, pbase = (jk * NPENCIL + pc) * TS;
                const T* prec = rec + SKW * pc;
                T2 a01[3] = {z2, z2, z2}, a23[3] = {z2, z2, z2}, f01[3] = {z2, z2, z2};
                T f2[3] = {T(0), T(0), T(0)};
                int qs = gstart[gbase];
#pragma unroll
                for (int gx = 0; gx < G1 + 2; ++gx) {
                    if (gx < G1) {
                        const int qe = gstart[gbase + gx + 1];
#pragma unroll 1
                        for (int q = qs; q < qe; ++q)
                            accumulate<T, KIND>(prec + q * RS, j, k, py, pz, M.h, M.h_inv, a01, a23, f01, f2);
                        qs = qe;
                    }
                    // x-node gx is final for this batch (later groups start further right)
                    const int o = pbase + gx;
                    if (bi != piece) {  // add to the block's earlier batches
                        a01[0] = padd(a01[0], part2[o]);
                        a23[0] = padd(a23[0], part2[CSTR + o]);
                        f01[0] = padd(f01[0], part2[2 * CSTR + o]);
                        f2[0] += partz[o];
                    }
                    part2[o] = a01[0];
                    part2[CSTR + o] = a23[0];
                    part2[2 * CSTR + o] = f01[0];
                    partz[o] = f2[0];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        a01[i] = a01[i + 1];
                        a23[i] = a23[i + 1];
                        f01[i] = f01[i + 1];
                        f2[i] = f2[i + 1];
                    }
                    a01[2] = a23[2] = f01[2] = z2;
                    f2[2] = T(0);
                }
            }
            __syncthreads();
        }
        if (piece >= bp.count()) continue;
        // ---- 3. per tile node: the staged partials, one global atomic per value. The
        //      next piece's barriers come before its first staged store.
        auto gather = [&](auto zero) {
            using A = decltype(zero);
            for (int t = tid; t < TN; t += NT) {
                const int tx = t % TS, ty = (t / TS) % TS, tz = t / (TS * TS);
                const int nx = org[0] + tx, ny = org[1] + ty, nz = org[2] + tz;
                if (nx < 0 || ny < 0 || nz < 0 || nx >= M.n[0] || ny >= M.n[1] || nz >= M.n[2]) continue;
                A val[NC] = {A(0), A(0), A(0), A(0), A(0), A(0), A(0)};
#pragma unroll
                for (int kk = 0; kk < 3; ++kk)
#pragma unroll
                    for (int jj = 0; jj < 3; ++jj) {
                        const int gy = ty - jj, gz = tz - kk;
                        if (gy < 0 || gy >= G1 || gz < 0 || gz >= G1) continue;
                        const int idx = ((jj + 3 * kk) * NPENCIL + gy + G1 * gz) * TS + tx;
                        const T2 p0 = part2[idx], p1 = part2[CSTR + idx], p2 = part2[2 * CSTR + idx];
                        val[0] += A(p0.x);
                        val[1] += A(p0.y);
                        val[2] += A(p1.x);
                        val[3] += A(p1.y);
                        val[4] += A(p2.x);
                        val[5] += A(p2.y);
                        val[6] += A(partz[idx]);
                    }
#pragma unroll
                for (int d = 0; d < 3; ++d) val[4 + d] += A(s.g[d]) * val[0];
                grid_add<3>(G, M, err, nx, ny, nz, val);
            }
        };
        if (KIND != P_BSP && KIND != P_JET) gather(T(0));
        else gather(0.0);
    }
}

template <class T, int KIND, int NR>
size_t pencil_smem_bytes() {
    using SH = PencilShape<3, 4>;
    return sizeof(T) * (size_t(NR) * RecOf<KIND>::SIZE + 2 * SH::NPENCIL + size_t(SH::NC) * SH::NPENCIL * SH::NJK * SH::TS) +
           sizeof(int) * size_t(SH::NG + SH::NG + 1 + 32);
}

// Records per batch: what two CTAs per SM (FP32) or one (FP64) leave beside the
// staging array, a whole 8-per-cell block (512) where the record is short. Fewer
// and longer passes pay: 144 records cost the dam break 4.55 ms against 3.06, 256
// cost the uGIMP sphere (878 k particles, FP32) 0.173 ms against 0.148.
template <class T, int KIND>
constexpr int pencil_nr() {
    if (sizeof(T) == 4) return KIND == P_JET ? 512 : 288;
    return KIND == P_BSP ? 512 : (KIND == P_JET ? 448 : 288);
}

template <class T, bool X64, int KIND>
cudaError_t launch_pencil(const DMesh<3, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                          const BinBuffers& b, const LaunchCfg& cfg, const int* list = nullptr,
                          const unsigned long long* nlist = nullptr) {
    constexpr int NR = pencil_nr<T, KIND>();
    constexpr int CTAS = sizeof(T) == 4 ? 2 : 1;
    auto kern = p2g_pencil_kernel<T, X64, KIND, NR, CTAS, KIND == P_BSP>;
    if (KIND == P_BSP && b.fresh) kern = p2g_pencil_kernel<T, X64, KIND, NR, CTAS, false>;
    const size_t smem = pencil_smem_bytes<T, KIND, NR>();
    int grid = 0;
    cudaError_t e = prepare_launch(kern, P2G_THREADS, smem, cfg, M.nblocks, grid);
    if (e != cudaSuccess) return e;
    launch_chained(kern, grid, P2G_THREADS, smem, cfg, M, P, G, s, b.totals, b.blocklist, b.offsets, b.perm, cfg.err, list,
                                                 nlist);
    ++*cfg.launches;
    return cudaGetLastError();
}

// 3D FP32 compact record, laid out for packed FP32x2 arithmetic (S = -V sigma in
// Tensorial order 11 21 31 22 32 33 = S0..S5):
//   (m, m v_x) (m v_y, m v_z) (S0, S1) (S1, S3) (S2, S4) (S5, t_z) (t_x, t_y)
// so that f_xy = dx (S0, S1) wyz + wx ((S1, S3) dyz + (S2, S4) wdz) is pairwise.
struct PairRec {
    float2 m0, m1, sa, sb, sc, s5z, txy;
};
__device__ __forceinline__ void load_pair_rec(const float* r, PairRec& o) {
    o.m0 = *reinterpret_cast<const float2*>(r + 0);
    o.m1 = *reinterpret_cast<const float2*>(r + 2);
    o.sa = *reinterpret_cast<const float2*>(r + 4);
    o.sb = *reinterpret_cast<const float2*>(r + 6);
    o.sc = *reinterpret_cast<const float2*>(r + 8);
    o.s5z = *reinterpret_cast<const float2*>(r + 10);
    o.txy = *reinterpret_cast<const float2*>(r + 12);
}
// Per x-node of a row lane: (m, m v_x), (m v_y, m v_z), (f_x, f_y) and f_z.
struct PairAcc {
    float2 a01, a23, f01;
    float f2;
};
// ---------------------------------------------------------------------------
// Plane kernel: the 3D FP32 forms of the quadratic B-spline with compact records
// in the packed FP32x2 layout (PairRec). A lane owns one z-slot k of a pencil's
// window, i.e. the 3 x 3 (x, y) nodes of 3 window rows, and walks the pencil's
// groups in x order keeping the 3 x-slots x 3 rows x 7 components (63 FP32
// accumulators) in registers. Per record a lane loads the record once and
// evaluates the x and y jets once for 9 nodes instead of 3, so the per-record
// overhead (loads, jets, row factors) is paid 3 times per particle instead of
// 9; the 25 pencils x 3 z-slots are 75 lanes of the 128-thread CTA.
// FULL (B-spline): blocks at the mesh boundary run the same way (bspline_start), their
// partials summed in FP64. Otherwise (KernelCorrection, whose cut windows have other
// weights) every block whose halo tile leaves the mesh is appended to `bnd` for a
// launch with full records. Whole steps of the B-spline with one launch and with two:
// 34 k particles on a floor 48 / 60 us, 1.0 M in mid-mesh 208 / 211, 1.3 M on a floor
// 241 / 275, 16.8 M in mid-mesh 2355 / 2358, 17.6 M on a floor 2480 / 2559 (FP32 with
// FP64 positions).
constexpr int PLANE_THREADS = 128;
constexpr int PLANE_NR = 512;
constexpr int CRS = 14;  // words of a PairRec record

// One record's contribution to a plane lane's 3 x 3 nodes.
__device__ __forceinline__ void accumulate_plane(const PairRec& o, const SlotPoly<float>& pz, float h_inv,
                                                 PairAcc (&acc)[3][3]) {
    const float tx = o.txy.x, ty = o.txy.y, tz = o.s5z.y;
    const float2 t2 = make_float2(tx, tx);
    // (wx_i, wx_i) and (dx_i, dx_i): the B-spline factors of the three x slots
    const float2 wx0 = __ffma2_rn(t2, __ffma2_rn(t2, make_float2(0.5f, 0.5f), make_float2(-1.f, -1.f)),
                                  make_float2(0.5f, 0.5f));
    const float2 wx1 = __ffma2_rn(t2, __ffma2_rn(t2, make_float2(-1.f, -1.f), make_float2(1.f, 1.f)),
                                  make_float2(0.5f, 0.5f));
    const float2 wx2 = __fmul2_rn(t2, __fmul2_rn(t2, make_float2(0.5f, 0.5f)));
    const float2 hh = make_float2(h_inv, h_inv);
    const float2 dx0 = __fmul2_rn(__fadd2_rn(t2, make_float2(-1.f, -1.f)), hh);
    const float2 dx1 = __fmul2_rn(__ffma2_rn(t2, make_float2(-2.f, -2.f), make_float2(1.f, 1.f)), hh);
    const float2 dx2 = __fmul2_rn(t2, hh);
    const float2 wxs[3] = {wx0, wx1, wx2}, dxs[3] = {dx0, dx1, dx2};
    // y jets of the three window rows, z jet of this lane's slot
    const float wy[3] = {0.5f + ty * (-1.0f + ty * 0.5f), 0.5f + ty * (1.0f + ty * -1.0f), ty * (ty * 0.5f)};
    const float dy[3] = {(-1.0f + ty) * h_inv, (1.0f + ty * -2.0f) * h_inv, ty * h_inv};
    const float wz = pz.a + tz * (pz.b + tz * pz.c);
    const float dz = (pz.e + tz * pz.f) * h_inv;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float wyz = wy[j] * wz, dyz = dy[j] * wz, wdz = wy[j] * dz;
        const float2 WYZ = make_float2(wyz, wyz);
        const float2 fa01 = __fmul2_rn(o.sa, WYZ);
        // the row's (m, m v) times wyz once; each x-slot then needs one FMA per pair
        const float2 m0j = __fmul2_rn(o.m0, WYZ), m1j = __fmul2_rn(o.m1, WYZ);
        const float2 fb01 = __ffma2_rn(o.sc, make_float2(wdz, wdz), __fmul2_rn(o.sb, make_float2(dyz, dyz)));
        const float fa2 = o.sc.x * wyz;
        const float fb2 = __fmaf_rn(o.s5z.x, wdz, o.sc.y * dyz);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            acc[i][j].a01 = __ffma2_rn(wxs[i], m0j, acc[i][j].a01);
            acc[i][j].a23 = __ffma2_rn(wxs[i], m1j, acc[i][j].a23);
            acc[i][j].f01 = __ffma2_rn(dxs[i], fa01, __ffma2_rn(wxs[i], fb01, acc[i][j].f01));
            acc[i][j].f2 = __fmaf_rn(dxs[i].x, fa2, __fmaf_rn(wxs[i].x, fb2, acc[i][j].f2));
        }
    }
}

template <bool X64, bool FULL>
__global__ void __launch_bounds__(PLANE_THREADS, 3)
    p2g_plane_kernel(DMesh<3, float> M, PView<float> P, GView<float> G, Scalars<float> s,
                     const int* __restrict__ totals, const int* __restrict__ blocklist,
                     const int* __restrict__ offsets, const int* __restrict__ perm, int* err,
                     int* __restrict__ bnd, unsigned long long* __restrict__ bnd_count) {
    chain_wait();
    using SH = PencilShape<3, 4>;
    constexpr int NT = PLANE_THREADS, NR = PLANE_NR, ITEMS = NR / NT;
    constexpr int TS = SH::TS, TN = SH::TN, NC = SH::NC, G1 = SH::G1, NG = SH::NG;
    constexpr int NJK = SH::NJK, NPENCIL = SH::NPENCIL;
    constexpr int CSTR = NPENCIL * NJK * TS;  // stride between components in the staging array
    constexpr int SKW = 2;                    // record skew per pencil (words)
    static_assert(NR % NT == 0 && NT % 8 == 0, "whole items per thread, passes in 8-particle chunks");
    static_assert(3 * NPENCIL <= NT, "one plane lane per (pencil, z slot)");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* rec = reinterpret_cast<float*>(smem_raw);
    // staged partials as (m, m v_x), (m v_y, m v_z), (f_x, f_y) pairs, then f_z:
    // [pair][jk][pencil][x] float2 and [jk][pencil][x] float (8-byte aligned)
    float* part = rec + NR * CRS + SKW * NPENCIL;
    float2* part2 = reinterpret_cast<float2*>(part);
    float* partz = part + 6 * CSTR;
    int* gcount = reinterpret_cast<int*>(part + NC * CSTR);
    int* gstart = gcount + NG;
    int* pslot = gstart + NG + 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nactive = totals[0];

    for (int g = tid; g < NG; g += NT) gcount[g] = 0;
    __syncthreads();

    // a piece per pass on crowded scenes, shorter passes where the blocks are few
    int per = NR;
    const int crowd = block_split(totals, NR);
    const int split = crowd > 1 ? crowd : block_pieces(totals, nactive, NR, gridDim.x, per);
    for (int vi = blockIdx.x; vi < nactive * split; vi += gridDim.x) {
        const int bi = split == 1 ? vi : vi / split, piece = vi - bi * split;
        const int b = blocklist[bi] - 1;
        int org[3];
        bool interior = true;
        {
            int r = b;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                org[d] = (r % M.nb[d]) * 4 - 1;
                r /= M.nb[d];
                interior = interior && org[d] >= 0 && org[d] + TS - 1 <= M.n[d] - 1;
            }
        }
        if constexpr (!FULL) {
            if (!interior) {  // the full-record launch's block (uniform over the CTA)
                if (tid == 0 && piece == 0) bnd[atomicAdd(bnd_count, 1ull)] = b;
                continue;
            }
        }
        const int s0 = offsets[b], s1 = offsets[b + 1];
        const BlockPasses bp(s0, s1, per);
        for (int bi = piece; bi < bp.count(); bi += split) {
            const int q0 = bp.pos(bi, tid), qstep = bp.step(NT);
            // ---- 1a. every global load of the batch first, then group and rank;
            //      the record's 14 values stay in registers until the slot is known
            int pid[ITEMS], grp[ITEMS], rank[ITEMS];
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const int ti = tid + u * NT, q = q0 + u * qstep;
                pid[u] = (ti < per && q < s1) ? perm[q] - 1 : -1;
            }
            float pv[ITEMS][3], pV[ITEMS], pm[ITEMS], psg[ITEMS][6], pt[ITEMS][3];
            double pxd[ITEMS][3];
            float pxf[ITEMS][3];
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const long long p = pid[u] >= 0 ? pid[u] : 0;
                const bool on = pid[u] >= 0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if constexpr (X64) pxd[u][d] = on ? P.x64[d][p] : 0.0;
                    else pxf[u][d] = on ? P.x[d][p] : 0.0f;
                    pv[u][d] = on ? P.v[d][p] : 0.0f;
                }
                pV[u] = on ? P.V[p] : 0.0f;
                pm[u] = (on && P.m) ? P.m[p] : s.mass;
#pragma unroll
                for (int k = 0; k < 6; ++k) psg[u][k] = on ? P.sig[k][p] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                grp[u] = -1;
                rank[u] = 0;
                if (pid[u] < 0) continue;
                // a particle outside the mesh has no window in an interior block's tile
                if constexpr (FULL)
                    if (!interior && !inside_mesh<3, float, X64>(M, pxd[u], pxf[u])) continue;
                int gi = 0;
                bool ok = true;
#pragma unroll
                for (int d = 2; d >= 0; --d) {
                    float t;
                    const int lo = bspline_start<3, float, X64>(M, d, pxd[u][d], pxf[u][d], t);
                    pt[u][d] = t;
                    const int q = lo - org[d];
                    ok = ok && q >= 0 && q < G1;
                    gi = gi * G1 + q;
                }
                if (!ok) {
                    atomicOr(err, ERR_TILE_RANGE);
                    continue;
                }
                grp[u] = gi;
                rank[u] = atomicAdd(&gcount[gi], 1);
            }
            __syncthreads();
            if (warp == 0) {
                int carry = 0;
                for (int g0 = 0; g0 < NG; g0 += 32) {
                    const int g = g0 + lane;
                    const int c = g < NG ? gcount[g] : 0;
                    int incl = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    if (g < NG) gstart[g] = carry + incl - c;
                    carry += __shfl_sync(0xffffffffu, incl, 31);
                }
                if (lane == 0) gstart[NG] = carry;
            } else if (warp == 1) {
                // pencil slots by size, largest first: the pencils of one warp
                // then have similar lengths
                const int myp = lane < NPENCIL ? lane : -1;
                int mysize = 0;
                if (myp >= 0) {
                    const int gb = G1 * myp;
#pragma unroll
                    for (int gx = 0; gx < G1; ++gx) mysize += gcount[gb + gx];
                }
                int rk = 0;
                for (int o = 0; o < NPENCIL; ++o) {
                    const int os = __shfl_sync(0xffffffffu, mysize, o);
                    rk += (os > mysize) || (os == mysize && o < lane);
                }
                if (myp >= 0) pslot[rk] = myp;
            }
            __syncthreads();
            // ---- 1b. records at their group-sorted slots (PairRec layout)
            for (int g = tid; g < NG; g += NT) gcount[g] = 0;  // ready for the next batch
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                if (grp[u] < 0) continue;
                float* r = rec + (gstart[grp[u]] + rank[u]) * CRS + SKW * (grp[u] / G1);
                const float mp = pm[u], nV = -pV[u];
                st2(r + 0, mp, mp * pv[u][0]);
                st2(r + 2, mp * pv[u][1], mp * pv[u][2]);
                st2(r + 4, nV * psg[u][0], nV * psg[u][1]);
                st2(r + 6, nV * psg[u][1], nV * psg[u][3]);
                st2(r + 8, nV * psg[u][2], nV * psg[u][4]);
                st2(r + 10, nV * psg[u][5], pt[u][2]);
                st2(r + 12, pt[u][0], pt[u][1]);
            }
            __syncthreads();
            // ---- 2. plane sweeps: lane (pencil slot, z slot k)
            if (tid < 3 * NPENCIL) {
                const int slot = tid / 3, k = tid - 3 * slot;
                const int pc = pslot[slot];
                const int gbase = G1 * pc;
                const float* prec = rec + SKW * pc;
                const SlotPoly<float> pz = slot_poly<float>(k);
                PairAcc acc[3][3];
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        acc[i][j].a01 = acc[i][j].a23 = acc[i][j].f01 = make_float2(0.f, 0.f);
                        acc[i][j].f2 = 0.f;
                    }
                int qs = gstart[gbase];
#pragma unroll
                for (int gx = 0; gx < G1 + 2; ++gx) {
                    if (gx < G1) {
                        const int qe = gstart[gbase + gx + 1];
#pragma unroll 1
                        for (int q = qs; q < qe; ++q) {
                            PairRec r0;
                            load_pair_rec(prec + q * CRS, r0);
                            accumulate_plane(r0, pz, M.h_inv, acc);
                        }
                        qs = qe;
                    }
                    // x-node gx of rows (j, k) is final: stage it, shift the rows
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const int o = ((j + 3 * k) * NPENCIL + pc) * TS + gx;
                        part2[o] = acc[0][j].a01;
                        part2[CSTR + o] = acc[0][j].a23;
                        part2[2 * CSTR + o] = acc[0][j].f01;
                        partz[o] = acc[0][j].f2;
                        acc[0][j] = acc[1][j];
                        acc[1][j] = acc[2][j];
                        acc[2][j].a01 = acc[2][j].a23 = acc[2][j].f01 = make_float2(0.f, 0.f);
                        acc[2][j].f2 = 0.f;
                    }
                }
            }
            __syncthreads();
            // ---- 3. per tile node: the staged partials, in FP32 (blocks at the mesh
            //      boundary: FP64), one global atomic per non-zero value (gravity from
            //      the summed mass)
            auto gather = [&](auto zero, auto clipped) {
                using A = decltype(zero);
                for (int t = tid; t < TN; t += NT) {
                    const int tx = t % TS, ty = (t / TS) % TS, tz = t / (TS * TS);
                    const int nx = org[0] + tx, ny = org[1] + ty, nz = org[2] + tz;
                    if constexpr (decltype(clipped)::value)
                        if (nx < 0 || ny < 0 || nz < 0 || nx >= M.n[0] || ny >= M.n[1] || nz >= M.n[2]) continue;
                    A val[NC] = {A(0), A(0), A(0), A(0), A(0), A(0), A(0)};
#pragma unroll
                    for (int kk = 0; kk < 3; ++kk)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) {
                            const int gy = ty - jj, gz = tz - kk;
                            if (gy < 0 || gy >= G1 || gz < 0 || gz >= G1) continue;
                            const int idx = ((jj + 3 * kk) * NPENCIL + gy + G1 * gz) * TS + tx;
                            const float2 p0 = part2[idx], p1 = part2[CSTR + idx], p2 = part2[2 * CSTR + idx];
                            val[0] += A(p0.x);
                            val[1] += A(p0.y);
                            val[2] += A(p1.x);
                            val[3] += A(p1.y);
                            val[4] += A(p2.x);
                            val[5] += A(p2.y);
                            val[6] += A(partz[idx]);
                        }
#pragma unroll
                    for (int d = 0; d < 3; ++d) val[4 + d] += A(s.g[d]) * val[0];
                    grid_add<3>(G, M, err, nx, ny, nz, val);
                }
            };
            if constexpr (FULL) {
                if (interior) gather(0.0f, std::false_type{});
                else gather(0.0, std::true_type{});
            } else {
                gather(0.0f, std::false_type{});
            }
        }
    }
}

size_t plane_smem_bytes() {
    using SH = PencilShape<3, 4>;
    return sizeof(float) * (size_t(PLANE_NR) * CRS + 2 * SH::NPENCIL + SH::NPART) +
           sizeof(int) * size_t(SH::NG + SH::NG + 1 + 32);
}

template <bool X64, bool FULL>
cudaError_t launch_plane(const DMesh<3, float>& M, const PView<float>& P, const GView<float>& G,
                         const Scalars<float>& s, const BinBuffers& b, const LaunchCfg& cfg, int* bnd,
                         unsigned long long* bnd_count) {
    auto kern = p2g_plane_kernel<X64, FULL>;
    const size_t smem = plane_smem_bytes();
    int grid = 0;
    cudaError_t e = prepare_launch(kern, PLANE_THREADS, smem, cfg, M.nblocks, grid);
    if (e != cudaSuccess) return e;
    // In order: set up early, its blocks (76 KB of shared memory, three per SM) arrive where
    // the fix-up still runs, and whole steps of 0.5 M particles and more take 2 to 10%
    // longer (1.0 M: 209 us early, 202 with every launch in order, 191 with this one).
    LaunchCfg in_order = cfg;
    in_order.early = false;
    launch_chained(kern, grid, PLANE_THREADS, smem, in_order, M, P, G, s, b.totals, b.blocklist, b.offsets, b.perm, cfg.err,
                                                   bnd, bnd_count);
    ++*cfg.launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// 2D kernel: every basis and transfer. A block of 8 x 8 cells has 81 groups in
// 9 pencils, too few pencils for a CTA: a lane owns one window row (3 x-nodes) of
// one group. The groups are taken class by class, gx = 0, 1, 2 (mod 3): no two
// groups of a class and a pencil share an x-node, so a lane adds its sums to its
// own staging slots with plain loads and stores; within a class the groups are
// ranked by size, so the lanes of a warp end together. A block is split into
// pieces of 128 particles or more until the GPU is full (block_pieces).
// 2D scenes are small: what bounds this kernel is the chain of a piece (load, rank,
// record, three classes, gather). 25 steps of a 111 k particle WLS + APIC scene in FP32: 0.185
// ms per step with one lane per pencil row, a moment inverse at every node and FP64
// shared atomics; 0.027 ms here.
//
// Record (words of T, in pairs): 0 (m, m v_x)  2 (m v_y, S11)  4 (S00, S01)
//   Q_BSP   quadratic B-spline, FLIP: 6 (t_x, t_y)
//   others  6 + 2j (wy, gy), 12 + 2i (wx, gx): jets (value, gradient)
//   Q_WLS   18 (u_x, u_y)
//   Q_APIC  (plain kernel) 18, Q_WLS_APIC 20: (B00, B10) (B01, B11) (r0_x, r0_y), B = m D^-1 B_p
// S = -V sigma; the weights and sums are those of the pencil kernel, without z.
enum : int { Q_BSP = 0, Q_JET = 1, Q_WLS = 2, Q_WLS_APIC = 3, Q_APIC = 4 };

template <int KIND>
struct Rec2 {
    static constexpr bool WLS = KIND == Q_WLS || KIND == Q_WLS_APIC, APIC = KIND == Q_WLS_APIC || KIND == Q_APIC;
    static constexpr int TXY = 6, WY = 6, WX = 12, U = 18, DB = WLS ? 20 : 18;
    // an odd number of pairs, so that neighbouring records fall on different banks
    static constexpr int SIZE = KIND == Q_BSP ? 10 : (KIND == Q_JET ? 18 : (KIND == Q_WLS ? 22 : 26));
};

// Type of the staged sums: WLS and APIC add a crowded block's passes (hundreds in one
// piece) in FP64 and round once per piece; the plain kinds' partials are T's. FP32
// staging left 6e-6 of a sum of 2^20 particles, FP64 less than 1e-6; 25 steps of a
// 111 k particle WLS + APIC scene take 1488 us instead of 1474.
template <class T, int KIND>
using Staged2 = typename std::conditional<Rec2<KIND>::WLS || Rec2<KIND>::APIC, double, T>::type;

constexpr int P2D_THREADS = 128, P2D_NB = 256, P2D_NR = 128;

template <class T, int BW, bool X64, int KIND>
__global__ void __launch_bounds__(P2D_THREADS, 4)
    p2g_2d_kernel(DMesh<2, T> M, PView<T> P, GView<T> G, Scalars<T> s, const int* __restrict__ totals,
                  const int* __restrict__ blocklist, const int* __restrict__ offsets, const int* __restrict__ perm,
                  int* err) {
    chain_wait();
    using SH = PencilShape<2, BW>;
    using R = Rec2<KIND>;
    using T2 = typename PairOf<T>::type;
    using A = Staged2<T, KIND>;
    using A2 = typename PairOf<A>::type;
    constexpr int NT = P2D_THREADS, NB = P2D_NB, NR = P2D_NR, ITEMS = NB / NT, RS = R::SIZE;
    constexpr int TS = SH::TS, TN = SH::TN, G1 = SH::G1, NG = SH::NG, CSTR = 3 * G1 * TS;
    constexpr int N0 = G1 * ((G1 + 2) / 3), N1 = N0 + G1 * ((G1 + 1) / 3);  // first group of classes 1 and 2
    static_assert(NB % NT == 0 && NT % 8 == 0, "whole items per thread, passes in 8-particle chunks");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* rec = reinterpret_cast<T*>(smem_raw);
    // staged (m, m v_x), (f_x, f_y) pairs and m v_y per (row offset j, pencil, x)
    static_assert(NR * RS * sizeof(T) % 16 == 0, "staged pairs aligned");
    A2* part2 = reinterpret_cast<A2*>(rec + NR * RS);
    A* party = reinterpret_cast<A*>(part2 + 2 * CSTR);
    int* gcount = reinterpret_cast<int*>(party + CSTR + 1);
    int* gstart = gcount + NG;
    int* order = gstart + NG + 1;  // the groups of each class by size
    int* slots = order + NG;       // particle of each slot
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = totals[0];
    const T2 z2 = pair(T(0), T(0));
    int per = NB;
    const int split = block_pieces(totals, nblk, NB, gridDim.x, per);
    auto class_begin = [&](int c) { return c == 0 ? 0 : (c == 1 ? N0 : (c == 2 ? N1 : NG)); };

    for (int g = tid; g < NG; g += NT) gcount[g] = 0;
    for (int vi = blockIdx.x; vi < nblk * split; vi += gridDim.x) {
        const int bi = split == 1 ? vi : vi / split, piece = vi - bi * split;
        const int b = blocklist[bi] - 1;
        const int org[2] = {(b % M.nb[0]) * BW - 1, (b / M.nb[0]) * BW - 1};
        const int s0 = offsets[b], s1 = offsets[b + 1];
        const BlockPasses bp(s0, s1, per);
        if (piece >= bp.count()) continue;
        __syncthreads();  // the last piece's gather is done
        for (int t = tid; t < 2 * CSTR; t += NT) part2[t] = pair(A(0), A(0));
        for (int t = tid; t < CSTR; t += NT) party[t] = A(0);
        for (int pi = piece; pi < bp.count(); pi += split) {
            // ---- 1. group and rank of every particle of the pass
            int pid[ITEMS], grp[ITEMS], rank[ITEMS];
            double xd[ITEMS][2] = {};
            T x[ITEMS][2] = {};
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const int ti = tid + u * NT, q = bp.pos(pi, ti);
                pid[u] = (ti < per && q < s1) ? perm[q] - 1 : -1;
                grp[u] = -1;
                rank[u] = 0;
            }
#pragma unroll
            for (int u = 0; u < ITEMS; ++u)
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    if constexpr (X64) xd[u][d] = pid[u] >= 0 ? P.x64[d][pid[u]] : 0.0;
                    else x[u][d] = pid[u] >= 0 ? P.x[d][pid[u]] : T(0);
                }
            __syncthreads();  // gcount is zero
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                if (pid[u] < 0) continue;
                int lo[3];
                if constexpr (KIND == Q_BSP) {
                    if (!inside_mesh<2, T, X64>(M, xd[u], x[u])) continue;
                    T t;
#pragma unroll
                    for (int d = 0; d < 2; ++d) lo[d] = bspline_start<2, T, X64>(M, d, xd[u][d], x[u][d], t);
                } else if (!window_start<2, T, X64>(M, s, xd[u], x[u], gimp_len(M, P, s, pid[u]), lo, err)) {
                    continue;
                }
                const int qx = lo[0] - org[0], qy = lo[1] - org[1];
                if (qx < 0 || qx >= G1 || qy < 0 || qy >= G1) {
                    atomicOr(err, ERR_TILE_RANGE);
                    continue;
                }
                grp[u] = class_begin(qx % 3) + (qx / 3) * G1 + qy;
                rank[u] = atomicAdd(&gcount[grp[u]], 1);
            }
            __syncthreads();
            if (warp == 0) {
                int carry = 0;
#pragma unroll
                for (int g0 = 0; g0 < NG; g0 += 32) {
                    const int g = g0 + lane;
                    const int c = g < NG ? gcount[g] : 0;
                    int incl = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    if (g < NG) gstart[g] = carry + incl - c;
                    carry += __shfl_sync(0xffffffffu, incl, 31);
                }
                if (lane == 0) gstart[NG] = carry;
            } else {
                for (int g = tid - 32; g < NG; g += NT - 32) {
                    const int c = g >= N1 ? 2 : (g >= N0 ? 1 : 0);
                    const int g0 = class_begin(c), g1 = class_begin(c + 1), mine = gcount[g];
                    int rk = g0;
                    for (int o = g0; o < g1; ++o) {
                        const int os = gcount[o];
                        rk += (os > mine) || (os == mine && o < g);
                    }
                    order[rk] = g;
                }
            }
            __syncthreads();
            for (int g = tid; g < NG; g += NT) gcount[g] = 0;  // ready for the next pass
#pragma unroll
            for (int u = 0; u < ITEMS; ++u)
                if (grp[u] >= 0) slots[gstart[grp[u]] + rank[u]] = pid[u];
            __syncthreads();
            // ---- 2. class by class: records, sweep, staging
#pragma unroll 1
            for (int c = 0; c < 3; ++c) {
                const int g0 = class_begin(c), g1 = class_begin(c + 1), c1 = gstart[g1];
#pragma unroll 1
                for (int r0 = gstart[g0]; r0 < c1; r0 += NR) {
                    const int r1 = min(r0 + NR, c1);
#pragma unroll 1
                    for (int t = r0 + tid; t < r1; t += NT) {
                        const long long p = slots[t];
                        T* r = rec + (t - r0) * RS;
                        double yd[2] = {};
                        T y[2] = {};
#pragma unroll
                        for (int d = 0; d < 2; ++d) {
                            if constexpr (X64) yd[d] = P.x64[d][p];
                            else y[d] = P.x[d][p];
                        }
                        const T mp = P.m ? P.m[p] : s.mass, nV = -P.V[p];
                        const T v0 = P.v[0][p], v1 = P.v[1][p], S0 = P.sig[0][p], S1 = P.sig[1][p], S2 = P.sig[2][p];
                        T Bp[4] = {};
                        if constexpr (R::APIC) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) Bp[k] = P.B[k][p];
                        }
                        st2(r + 0, mp, mp * v0);
                        st2(r + 2, mp * v1, nV * S2);
                        st2(r + 4, nV * S0, nV * S1);
                        if constexpr (KIND == Q_BSP) {
                            T t0, t1;
                            bspline_start<2, T, X64>(M, 0, yd[0], y[0], t0);
                            bspline_start<2, T, X64>(M, 1, yd[1], y[1], t1);
                            st2(r + R::TXY, t0, t1);
                        } else {
                            Basis<2, T> B = {};
                            bool in;
                            const GimpLen<T> gl = gimp_len(M, P, s, p);
                            if constexpr (X64) in = prepare_basis_x64<2, T, R::WLS>(M, s.basis, yd, gl, B, err);
                            else in = prepare_basis<2, T, R::WLS>(M, s.basis, y, gl, B, err);
                            const T on = in ? T(1) : T(0);  // a singular fit (reported) adds nothing
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                st2(r + R::WY + 2 * k, in ? B.ax[1].val[k] : on, in ? B.ax[1].der[k] * M.h_inv : on);
                                st2(r + R::WX + 2 * k, in ? B.ax[0].val[k] : on, in ? B.ax[0].der[k] * M.h_inv : on);
                            }
                            if constexpr (R::WLS) st2(r + R::U, in ? B.u[0] : on, in ? B.u[1] : on);
                            if constexpr (R::APIC) {
                                const T md = mp * (T(4) / (M.h * M.h));
                                T q[2];
#pragma unroll
                                for (int d = 0; d < 2; ++d) {
                                    if constexpr (X64)
                                        q[d] = T(__dadd_rn(M.xmin64[d], __dmul_rn(double(B.ax[d].lo), M.h64)) - yd[d]);
                                    else
                                        q[d] = node_coord(M, d, B.ax[d].lo) - y[d];
                                }
                                st2(r + R::DB, md * Bp[0], md * Bp[1]);
                                st2(r + R::DB + 2, md * Bp[2], md * Bp[3]);
                                st2(r + R::DB + 4, in ? q[0] : on, in ? q[1] : on);
                            }
                        }
                    }
                    __syncthreads();
#pragma unroll 1
                    for (int t = tid; t < 3 * (g1 - g0); t += NT) {
                        const int g = order[g0 + t / 3], j = t % 3;
                        const int q0 = max(gstart[g], r0), q1 = min(gstart[g + 1], r1);
                        if (q0 >= q1) continue;
                        const SlotPoly<T> py = slot_poly<T>(j);
                        T2 am[3] = {z2, z2, z2}, af[3] = {z2, z2, z2};
                        T ay[3] = {T(0), T(0), T(0)};
#pragma unroll 1
                        for (int q = q0; q < q1; ++q) {
                            const T2* r = reinterpret_cast<const T2*>(rec + (q - r0) * RS);
                            T2 mx = r[0];
                            const T2 ys = r[1], sa = r[2];
                            T my = ys.x, wx[3], gx[3], wy, gy;
                            if constexpr (KIND == Q_BSP) {
                                const T2 txy = r[R::TXY / 2];
                                T dx[3];
                                bspline_quadratic_poly(txy.x, wx, dx);
#pragma unroll
                                for (int i = 0; i < 3; ++i) gx[i] = dx[i] * M.h_inv;
                                wy = py.a + txy.y * (py.b + txy.y * py.c);
                                gy = (py.e + txy.y * py.f) * M.h_inv;
                            } else {
#pragma unroll
                                for (int i = 0; i < 3; ++i) {
                                    const T2 q2 = r[R::WX / 2 + i];
                                    wx[i] = q2.x;
                                    gx[i] = q2.y;
                                }
                                const T2 q2 = r[R::WY / 2 + j];
                                wy = q2.x;
                                gy = q2.y;
                            }
                            T rr = wy, qq = T(0), bxx = T(0), byx = T(0), r0x = T(0);
                            if constexpr (R::WLS) {
                                const T2 u = r[R::U / 2];
                                rr = wy - u.y * gy;
                                qq = -u.x * wy;
                            }
                            if constexpr (R::APIC) {
                                const T2 b0 = r[R::DB / 2], b1 = r[R::DB / 2 + 1], r0v = r[R::DB / 2 + 2];
                                const T ry = r0v.y + T(j) * M.h;
                                mx.y += b1.x * ry;
                                my += b1.y * ry;
                                bxx = b0.x;
                                byx = b0.y;
                                r0x = r0v.x;
                            }
                            // f_x = gx S00 wy + wx S01 gy, f_y = gx S01 wy + wx S11 gy
                            const T2 fa = pmul(sa, pair(wy, wy)), fb = pmul(pair(sa.y, ys.y), pair(gy, gy));
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                T N = wx[i] * rr;
                                if constexpr (R::WLS) N += gx[i] * qq;
                                T2 mi = mx;
                                T yi = my;
                                if constexpr (R::APIC) {
                                    const T rx = r0x + T(i) * M.h;
                                    mi.y += bxx * rx;
                                    yi += byx * rx;
                                }
                                am[i] = pfma(pair(N, N), mi, am[i]);
                                ay[i] += N * yi;
                                af[i] = pfma(pair(gx[i], gx[i]), fa, pfma(pair(wx[i], wx[i]), fb, af[i]));
                            }
                        }
                        const int mem = (g - g0) / G1, gy = (g - g0) - mem * G1;
                        const int o = (j * G1 + gy) * TS + 3 * mem + c;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            part2[o + i] = padd(part2[o + i], pair(A(am[i].x), A(am[i].y)));
                            part2[CSTR + o + i] = padd(part2[CSTR + o + i], pair(A(af[i].x), A(af[i].y)));
                            party[o + i] += A(ay[i]);
                        }
                    }
                    __syncthreads();
                }
            }
        }
        // ---- 3. per tile node inside the mesh: the staged partials, in FP64
        for (int t = tid; t < TN; t += NT) {
            const int tx = t % TS, ty = t / TS, nx = org[0] + tx, ny = org[1] + ty;
            if (nx < 0 || ny < 0 || nx >= M.n[0] || ny >= M.n[1]) continue;
            double val[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int jj = 0; jj < 3; ++jj) {
                const int gy = ty - jj;
                if (gy < 0 || gy >= G1) continue;
                const int idx = (jj * G1 + gy) * TS + tx;
                const A2 p0 = part2[idx], p1 = part2[CSTR + idx];
                val[0] += double(p0.x);
                val[1] += double(p0.y);
                val[2] += double(party[idx]);
                val[3] += double(p1.x);
                val[4] += double(p1.y);
            }
            val[3] += double(s.g[0]) * val[0];
            val[4] += double(s.g[1]) * val[0];
            grid_add<2>(G, M, err, nx, ny, 0, val);
        }
    }
}

template <class T, int BW, bool X64, int KIND>
cudaError_t launch_2d_kind(const DMesh<2, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                           const BinBuffers& b, const LaunchCfg& cfg) {
    using SH = PencilShape<2, BW>;
    auto kern = p2g_2d_kernel<T, BW, X64, KIND>;
    const size_t smem = sizeof(T) * size_t(P2D_NR) * Rec2<KIND>::SIZE +
                        sizeof(Staged2<T, KIND>) * size_t(5 * 3 * SH::G1 * SH::TS + 1) +
                        sizeof(int) * size_t(3 * SH::NG + 1 + P2D_NB);
    int grid = 0;
    cudaError_t e = prepare_launch(kern, P2D_THREADS, smem, cfg, M.nblocks, grid);
    if (e != cudaSuccess) return e;
    launch_chained(kern, grid, P2D_THREADS, smem, cfg, M, P, G, s, b.totals, b.blocklist, b.offsets, b.perm, cfg.err);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <class T, int BW, bool X64>
cudaError_t launch_p2g_2d(const DMesh<2, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                          const BinBuffers& b, const LaunchCfg& cfg) {
    KernelScope ks(cfg, "p2g");
    const bool wls = s.basis == TB_WLS_BSPLINE_QUADRATIC || s.basis == TB_WLS_UGIMP;
    if constexpr (!X64) {  // the FP64-position form runs these in 3D only (checked by the caller)
        if (s.transfer == TB_TRANSFER_APIC)
            return wls ? launch_2d_kind<T, BW, X64, Q_WLS_APIC>(M, P, G, s, b, cfg)
                       : launch_2d_kind<T, BW, X64, Q_APIC>(M, P, G, s, b, cfg);
        if (wls) return launch_2d_kind<T, BW, X64, Q_WLS>(M, P, G, s, b, cfg);
    }
    if (s.basis == TB_BSPLINE_QUADRATIC) return launch_2d_kind<T, BW, X64, Q_BSP>(M, P, G, s, b, cfg);
    return launch_2d_kind<T, BW, X64, Q_JET>(M, P, G, s, b, cfg);
}

// 3D. The quadratic B-spline in the FP32 forms takes the plane kernel (short
// records, 9 nodes per lane). KernelCorrection changes the weights of cut windows
// only: its interior blocks are plain B-spline, the others (their list in binning
// scratch that is free until the next binning: one int per block in the cursors)
// take full records.
template <class T, bool X64>
cudaError_t launch_p2g_3d(const DMesh<3, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                          const BinBuffers& b, const LaunchCfg& cfg) {
    KernelScope ks(cfg, "p2g");
    const bool wls = s.basis == TB_WLS_BSPLINE_QUADRATIC || s.basis == TB_WLS_UGIMP;
    if (s.transfer == TB_TRANSFER_APIC)
        return wls ? launch_pencil<T, X64, P_WLS_APIC>(M, P, G, s, b, cfg)
                   : launch_pencil<T, X64, P_APIC>(M, P, G, s, b, cfg);
    if (wls) return launch_pencil<T, X64, P_WLS>(M, P, G, s, b, cfg);
    if constexpr (sizeof(T) == 4) {
        if (s.basis == TB_BSPLINE_QUADRATIC) return launch_plane<X64, true>(M, P, G, s, b, cfg, nullptr, nullptr);
        if (s.basis == TB_KC_BSPLINE_QUADRATIC) {
            const cudaError_t e = launch_plane<X64, false>(M, P, G, s, b, cfg, b.cursors, b.bnd_count);
            if (e != cudaSuccess) return e;
            return launch_pencil<T, X64, P_JET>(M, P, G, s, b, cfg, b.cursors, b.bnd_count);
        }
    } else if (s.basis == TB_BSPLINE_QUADRATIC) {
        return launch_pencil<T, X64, P_BSP>(M, P, G, s, b, cfg);
    }
    return launch_pencil<T, X64, P_JET>(M, P, G, s, b, cfg);
}

}  // namespace

template <int D, class T, int BW>
cudaError_t launch_p2g(const DMesh<D, T>& M, const PView<T>& P, const GView<T>& G, const Scalars<T>& s,
                       const BinBuffers& b, const LaunchCfg& cfg) {
    if (P.n == 0) return cudaSuccess;
    if (P.x64[0]) {  // FP64-position form: FP32 state only (checked by the caller)
        if constexpr (sizeof(T) == 4) {
            if constexpr (D == 3) return launch_p2g_3d<T, true>(M, P, G, s, b, cfg);
            else return launch_p2g_2d<T, BW, true>(M, P, G, s, b, cfg);
        }
        return cudaErrorInvalidValue;
    }
    if constexpr (D == 3) return launch_p2g_3d<T, false>(M, P, G, s, b, cfg);
    else return launch_p2g_2d<T, BW, false>(M, P, G, s, b, cfg);
}

#define TB_INST_P2G(D, T, BW)                                                                        \
    template cudaError_t launch_p2g<D, T, BW>(const DMesh<D, T>&, const PView<T>&, const GView<T>&, \
                                              const Scalars<T>&, const BinBuffers&, const LaunchCfg&);
TB_INST_P2G(3, double, 4)
TB_INST_P2G(3, float, 4)
TB_INST_P2G(2, double, 8)
TB_INST_P2G(2, float, 8)
TB_INST_P2G(2, double, 4)
TB_INST_P2G(2, float, 4)

}  // namespace tb
