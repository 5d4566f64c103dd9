// tb_transfer.cu -- grid update and G2P kernels of the explicit MPM step.
//
// (P2G is in tb_p2g.cu.)
// grid (src/Transfer/foreach.jl:276-339, docs/src/gpu.md:309-316): vn = mv/m,
//      v = vn + dt f / m guarded by m != 0, then the slip-wall slices.
// G2P  (src/Transfer/gpu.jl:226-232, README.md:79-86): one CTA per non-empty
//      block stages the block's (v, v - vn) tile in shared memory and gathers
//      for each particle of the block (3D FP32: packed FP32x2 FMAs over the
//      component pairs of a node-major tile); particles outside the mesh (empty
//      window) are updated by a particle-parallel pass.
#include "tb_launch.cuh"

namespace tb {

namespace {

template <int D, int BW>
struct Tile {
    static constexpr int TS = BW + 3;
    static constexpr int TN = (D == 3) ? TS * TS * TS : TS * TS;
};

template <int D, class T>
__device__ __forceinline__ void load_x(const PView<T>& P, long long p, T* x) {
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = P.x[d][p];
}

// Stored nodes of a grid: every node of a dense grid; the active blocks' nodes
// (up to the fields' capacity) of a sparse one.
template <int D, class T>
__device__ __forceinline__ long long stored_nodes(const GView<T>& G, long long nnodes) {
    if (!G.bnum) return nnodes;
    const long long n = (long long)G.nact[0] << (G.L * D);
    return n < G.cap ? n : G.cap;
}

// Each array in runs of 32 values that start at a multiple of 32 values in memory: a
// row of a (2^k + 1)^3 mesh starts anywhere, and warps that store across a sector's
// end leave it to two partial writes (257^3 nodes, FP32, 475 MB: 0.162 ms by linear
// index, 0.140 ms here, which is what memsets took).
template <int D, class T>
__global__ void __launch_bounds__(256) grid_zero_kernel(GView<T> G, long long nnodes) {
    chain_wait();
    const long long nn = stored_nodes<D>(G, nnodes);
    for (long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x; I < nn + 31;
         I += (long long)gridDim.x * blockDim.x) {
        auto zero = [&](T* a) {
            const long long J = I - (long long)((reinterpret_cast<unsigned long long>(a) / sizeof(T)) & 31);
            if (J >= 0 && J < nn) a[J] = T(0);
        };
        zero(G.m);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            zero(G.mv[d]);
            zero(G.f[d]);
        }
    }
}

// vn = mv / m, v = vn + dt f / m, slip walls, for one node (m = 0: zero). The loads
// come first, together: a store between them would hold the next ones back.
template <int D, class T>
__device__ __forceinline__ void update_node(const DMesh<D, T>& M, const GView<T>& G, const Scalars<T>& s, const int* idx,
                                            long long I, T m) {
    T vn[D], v[D];
    if (m != T(0)) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            vn[d] = G.mv[d][I];
            v[d] = G.f[d][I];
        }
#pragma unroll
        for (int d = 0; d < D; ++d) {
            vn[d] = vn[d] / m;
            v[d] = vn[d] + (s.dt * v[d]) / m;
        }
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) vn[d] = v[d] = T(0);
    }
    if (s.wall_mask) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const bool lo = (s.wall_mask >> (2 * d)) & 1, hi = (s.wall_mask >> (2 * d + 1)) & 1;
            if ((lo && idx[d] < s.wall_layers) || (hi && idx[d] >= M.n[d] - s.wall_layers)) {
                vn[d] = T(0);
                v[d] = T(0);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        G.vn[d][I] = vn[d];
        G.v[d][I] = v[d];
    }
}

// Every node of a dense grid in memory order, so that the time does not depend on
// which axis is short. A node's place matters to the walls only, and takes 32-bit
// divisions where the mesh allows. Every node with mass, FP32, no walls: 193^3 nodes
// 0.105 ms (0.125 with stores between the loads and 64-bit divisions, 0.191 with a
// warp per row of x), 4096 x 9 nodes 7 us (177 us with a warp per row).
template <int D, class T>
__global__ void __launch_bounds__(256) grid_update_kernel(DMesh<D, T> M, GView<T> G, Scalars<T> s) {
    chain_wait();
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x; I < M.nnodes; I += stride) {
        int idx[3] = {0, 0, 0};
        if (s.wall_mask) {
            if (M.nnodes <= 0xffffffffll) {
                const unsigned i = unsigned(I), r = i / unsigned(M.n[0]);
                idx[0] = int(i - r * unsigned(M.n[0]));
                idx[1] = int(r);
                if constexpr (D == 3) {
                    idx[2] = int(r / unsigned(M.n[1]));
                    idx[1] = int(r) - idx[2] * M.n[1];
                }
            } else {
                long long r = I;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    idx[d] = int(r % M.n[d]);
                    r /= M.n[d];
                }
            }
        }
        update_node<D, T>(M, G, s, idx, I, G.m[I]);
    }
}

// The stored nodes of a block-sparse grid.
template <int D, class T>
__global__ void __launch_bounds__(256) grid_update_sparse_kernel(DMesh<D, T> M, GView<T> G, Scalars<T> s) {
    const long long nn = stored_nodes<D>(G, M.nnodes);
    for (long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x; I < nn;
         I += (long long)gridDim.x * blockDim.x) {
        // slot I of storage block k: node (B's origin) + (column-major local index)
        const int W = 1 << G.L, k = int(I >> (G.L * D)), q = int(I & ((1ll << (G.L * D)) - 1));
        const int B = G.blist[k] - 1;
        const int bidx[3] = {B % M.nb[0], (B / M.nb[0]) % M.nb[1], D == 3 ? B / (M.nb[0] * M.nb[1]) : 0};
        const int qidx[3] = {q % W, (q / W) % W, q / (W * W)};
        int idx[3] = {0, 0, 0};
        bool inside = true;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            idx[d] = bidx[d] * W + qidx[d];
            inside = inside && idx[d] < M.n[d];
        }
        if (!inside) {  // a block's nodes past the mesh edge
#pragma unroll
            for (int d = 0; d < D; ++d) G.vn[d][I] = G.v[d][I] = T(0);
            continue;
        }
        update_node<D, T>(M, G, s, idx, I, G.m[I]);
    }
}

// ---- grid maintenance over the touched node blocks -----------------------
// Node block B owns nodes [BW B, BW B + BW - 1] per axis. A particle block b
// reaches nodes [BW b - 1, BW b + BW + 1], i.e. node blocks b-1 .. b+1 per axis; the
// scan of the binning lists the blocks reached now or in the previous transfer.
// One warp per listed node block. mode 0: zero m, mv, f; mode 1: grid update
// where cur, zero v, vn where the block was touched by the previous transfer only;
// with zero_after, m, mv and f of the cur blocks are zeroed once read (the next
// P2G of the same call then needs no zero pass).
template <int D, class T, int BW, int MODE>
__global__ void __launch_bounds__(256) node_list_kernel(DMesh<D, T> M, GView<T> G, Scalars<T> s,
                                                        const unsigned char* __restrict__ cur,
                                                        const int* __restrict__ list, const int* __restrict__ count,
                                                        int zero_after) {
    chain_wait();
    constexpr int NPB = (D == 3) ? BW * BW * BW : BW * BW;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int nlist = *count;
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nlist; w += warps) {
        const int B = list[w];
        const bool c = MODE == 1 ? cur[B] != 0 : true;
        const int bx = B % M.nb[0], by = (B / M.nb[0]) % M.nb[1], bz = (D == 3) ? B / (M.nb[0] * M.nb[1]) : 0;
        for (int q = lane; q < NPB; q += 32) {
            int idx[3];
            idx[0] = bx * BW + q % BW;
            idx[1] = by * BW + (q / BW) % BW;
            idx[2] = (D == 3) ? bz * BW + q / (BW * BW) : 0;
            bool inside = true;
#pragma unroll
            for (int d = 0; d < D; ++d) inside = inside && idx[d] < M.n[d];
            if (!inside) continue;
            long long I = 0;
#pragma unroll
            for (int d = D - 1; d >= 0; --d) I = I * M.n[d] + idx[d];
            if constexpr (MODE == 0) {
                G.m[I] = T(0);
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    G.mv[d][I] = T(0);
                    G.f[d][I] = T(0);
                }
            } else {
                update_node<D, T>(M, G, s, idx, I, c ? G.m[I] : T(0));
                if (zero_after && c) {
                    G.m[I] = T(0);
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        G.mv[d][I] = T(0);
                        G.f[d][I] = T(0);
                    }
                }
            }
        }
    }
}

// Final per-particle writes of @G2P and the FP64 constitutive update.
template <int D, class T, bool VM = false>
__device__ __forceinline__ void g2p_finish(const PView<T>& P, const Scalars<T>& s, long long p, const T* x,
                                           const T* vp, const T* vpic, const T* dvf, const T (&gv)[3][3],
                                           const T* dxs, const T (&Bn)[3][3], const double (&F)[3][3]) {
    if (s.transfer == TB_TRANSFER_APIC) {
#pragma unroll
        for (int d = 0; d < D; ++d) P.v[d][p] = vpic[d];
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
            for (int c = 0; c < D; ++c) P.B[r + c * D][p] = Bn[r][c];
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const T vflip = vp[d] + dvf[d];
            P.v[d][p] = (s.alpha == T(1)) ? vflip : (T(1) - s.alpha) * vpic[d] + s.alpha * vflip;
        }
    }
#pragma unroll
    for (int r = 0; r < D; ++r)
#pragma unroll
        for (int c = 0; c < D; ++c) P.gv[r + c * D][p] = gv[r][c];
    if (P.x[0]) {  // the FP64-position form writes x itself
#pragma unroll
        for (int d = 0; d < D; ++d) (P.x_out[0] ? P.x_out[d] : P.x[d])[p] = x[d] + dxs[d];
    }
    particle_update<D, T, VM>(P, s, p, gv, F);
}

// GEN: which basis and transfer the kernel gathers for.
//   G_PLAIN    B-spline / uGIMP / KernelCorrection, FLIP/PIC: separable contraction
//   G_WLS      WLS, FLIP/PIC: the same contraction with the WLS jets (wls_correct).
//              N_i = W_i on a window that the mesh does not cut; a cut window
//              takes the per-node loop (N_i = W_i - u . G_i)
//   G_WLS_APIC WLS, APIC: as G_WLS; sum N v (x) r = grad_v diag(var) comes without
//              another sum, since G_{i,d} = W_i r_d / var_d
//   G_APIC     plain kernel, APIC: the contraction with the first moments of r
// Before the closed form every WLS / APIC particle evaluated a (D+1)^2 moment
// inverse at each of its nodes: dam break at half resolution, 18.2 M particles,
// FP32 with FP64 positions, 3.66 ms; 1.75 ms now.
enum : int { G_PLAIN = 0, G_WLS = 1, G_WLS_APIC = 2, G_APIC = 3 };

// CTAs of 128 threads per SM. General kinds in FP32: 6 (80 registers) measured 1.92
// ms on the dam break below, 4 / 5 / 8: 2.01 / 2.28 / 2.10 ms.
constexpr int g2p_ctas(int gen, bool vm, bool fp32) {
    if (vm) return fp32 ? 4 : 2;
    if (gen != G_PLAIN) return fp32 ? 6 : 3;
    return fp32 ? 8 : 4;
}

template <int D, class T, int BW, int GEN, bool X64, bool VM = false>
__global__ void __launch_bounds__(128, g2p_ctas(GEN, VM, sizeof(T) == 4)) g2p_tile_kernel(DMesh<D, T> M, GView<T> G, PView<T> P, Scalars<T> s,
                                                       const int* __restrict__ totals,
                                                       const int* __restrict__ blocklist,
                                                       const int* __restrict__ offsets,
                                                       const int* __restrict__ perm, int* err,
                                                       int* __restrict__ next_bid, int* __restrict__ next_count) {
    chain_wait();
    constexpr int TS = Tile<D, BW>::TS, TN = Tile<D, BW>::TN;
    constexpr bool WLS = GEN == G_WLS || GEN == G_WLS_APIC, APIC = GEN == G_WLS_APIC || GEN == G_APIC;
    // 3D FP32: node-major, (v_x, v_y, v_z, dv_x) as a float4 at [t] and (dv_y, dv_z)
    // as a float2 after the TN float4s, dv = v - vn: two vector loads per node,
    // whose halves feed packed FP32x2 FMAs. Otherwise component-major: v_r at
    // [r TN + t], dv_r at [(D + r) TN + t]; lanes reading different nodes hit
    // different banks. APIC reads no vn: the tile holds v alone.
    constexpr bool VEC = (D == 3 && sizeof(T) == 4);
    __shared__ __align__(16) T tile[APIC ? (VEC ? 4 : D) * TN : 2 * D * TN];
    auto node_vals = [&](int t, T (&vi)[3], T (&dvi)[3]) {
        if constexpr (VEC) {
            const float4 a = reinterpret_cast<const float4*>(tile)[t];
            vi[0] = a.x; vi[1] = a.y; vi[2] = a.z;
            if constexpr (!APIC) {
                const float2 c = reinterpret_cast<const float2*>(tile + 4 * TN)[t];
                dvi[0] = a.w; dvi[1] = c.x; dvi[2] = c.y;
            }
        } else {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                vi[d] = tile[d * TN + t];
                if constexpr (!APIC) dvi[d] = tile[(D + d) * TN + t];
            }
        }
    };
    const int nactive = totals[0];
    const int tid = threadIdx.x, nth = blockDim.x;
    // CTA `piece` of `split` sharing a block takes its particles piece nth + tid,
    // (piece + split) nth + tid, ... (4 particles per thread; fewer, down to one, where
    // the blocks are fewer than the CTAs: a 111 k particle 2D scene of 200 blocks,
    // 0.0209 -> 0.0148 ms per step)
    int per;
    const int split = max(block_split(totals, 4 * nth), block_pieces(totals, nactive, 4 * nth, gridDim.x, per));
    const int stride = split * nth;
    for (int vi = blockIdx.x; vi < nactive * split; vi += gridDim.x) {
        const int bi = split == 1 ? vi : vi / split, piece = vi - bi * split;
        int b = blocklist[bi] - 1;
        int org[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < D; ++d) {
            org[d] = (b % M.nb[d]) * BW - 1;
            b /= M.nb[d];
        }
        b = blocklist[bi] - 1;
        // the block's particle range and this thread's first particle id are
        // loaded before the tile, so their round trips overlap the tile's
        const int s0 = offsets[b] + piece * nth, s1 = offsets[b + 1];
        int pnext = (s0 + tid < s1) ? perm[s0 + tid] : 1;
        for (int t = tid; t < TN; t += nth) {
            int node[3] = {0, 0, 0}, rem = t;
            bool inside = true;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                node[d] = org[d] + rem % TS;
                rem /= TS;
                inside = inside && node[d] >= 0 && node[d] < M.n[d];
            }
            // nodes outside the mesh, and nodes a sparse grid does not store, read as zero
            const long long sl = inside ? grid_slot<D>(G, M, node[0], node[1], node[2]) : -1;
            T vi[3] = {T(0), T(0), T(0)}, dvi[3] = {T(0), T(0), T(0)};
#pragma unroll
            for (int d = 0; d < D; ++d) {
                vi[d] = sl >= 0 ? G.v[d][sl] : T(0);
                if constexpr (!APIC) {
                    const T vni = sl >= 0 ? G.vn[d][sl] : T(0);
                    dvi[d] = vi[d] - vni;
                }
            }
            if constexpr (VEC) {
                reinterpret_cast<float4*>(tile)[t] = make_float4(vi[0], vi[1], vi[2], dvi[0]);
                if constexpr (!APIC) reinterpret_cast<float2*>(tile + 4 * TN)[t] = make_float2(dvi[1], dvi[2]);
            } else {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    tile[d * TN + t] = vi[d];
                    if constexpr (!APIC) tile[(D + d) * TN + t] = dvi[d];
                }
            }
        }
        __syncthreads();
        for (int j = s0 + tid; j < s1; j += stride) {
            const long long p = pnext - 1;
            pnext = (j + stride < s1) ? perm[j + stride] : 1;  // next id in flight during this particle
            T x[3] = {T(0), T(0), T(0)}, vp[3];
            double xd[3] = {0.0, 0.0, 0.0};
            if constexpr (X64) {
#pragma unroll
                for (int d = 0; d < D; ++d) xd[d] = P.x64[d][p];
            } else {
                load_x<D, T>(P, p, x);
            }
#pragma unroll
            for (int d = 0; d < D; ++d) vp[d] = P.v[d][p];
            // F (72 bytes in FP64): the FP32 kernels (64 to 80 registers) load it
            // after the gather, where holding it across the gather cost spills
            // (G2P 1.032 -> 1.019 ms on cube3d); the FP64 kernels load it here so
            // that the load overlaps the gather (loading it late measured 7% slower).
            constexpr bool LATE_F = sizeof(T) == 4;
            double F[3][3];
            if constexpr (!LATE_F) load_F<D, T>(P, p, F);
            const GimpLen<T> l = gimp_len(M, P, s, p);
            T vpic[3] = {T(0), T(0), T(0)}, dvf[3] = {T(0), T(0), T(0)}, dxs[3] = {T(0), T(0), T(0)};
            T gv[3][3] = {}, Bn[3][3] = {};
            Basis<D, T> B;
            bool in;
            if constexpr (X64) in = prepare_basis_x64<D, T, WLS>(M, s.basis, xd, l, B, err);
            else in = prepare_basis<D, T, WLS>(M, s.basis, x, l, B, err);
            if (in) {
                int q0[3] = {0, 0, 0};
                bool ok = true;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    q0[d] = B.ax[d].lo - org[d];
                    ok = ok && q0[d] >= 0 && q0[d] + 2 < TS;
                }
                if (!ok) {
                    atomicOr(err, ERR_TILE_RANGE);
                } else if (WLS && B.cut) {
                    // A WLS window that the mesh cuts, row by row: N_x = wx R + gx Q with
                    // R = wyz - u_y dyz - u_z wdz, Q = -u_x wyz. The row loops are not
                    // unrolled (jets by selection): few particles come here, and 27
                    // unrolled nodes made the kernel wait for instructions (dam break:
                    // 1.83 ms against 1.75).
                    auto sel = [](const T* q, int k) { return k == 0 ? q[0] : (k == 1 ? q[1] : q[2]); };
                    auto rel = [&](int d, int k) {
                        if constexpr (X64)  // X_i - x_p in FP64, rounded once
                            return T(__dadd_rn(M.xmin64[d], __dmul_rn(double(B.ax[d].lo + k), M.h64)) - xd[d]);
                        else
                            return node_coord(M, d, B.ax[d].lo + k) - x[d];
                    };
#pragma unroll 1
                    for (int jk = 0; jk < (D == 3 ? 9 : 3); ++jk) {
                        const int k = jk / 3, jj = jk - 3 * k;
                        const T wy = sel(B.ax[1].val, jj), gy = sel(B.ax[1].der, jj) * M.h_inv;
                        T wz = T(1), gz = T(0);
                        if constexpr (D == 3) {
                            wz = sel(B.ax[D - 1].val, k);
                            gz = sel(B.ax[D - 1].der, k) * M.h_inv;
                        }
                        const T wyz = wy * wz, dyz = gy * wz, wdz = wy * gz;
                        T R = wyz - B.u[1] * dyz;
                        if constexpr (D == 3) R -= B.u[D - 1] * wdz;
                        const T Q = -B.u[0] * wyz;
                        const T ry = APIC ? rel(1, jj) : T(0), rz = (APIC && D == 3) ? rel(D - 1, k) : T(0);
                        const int t0 = (D == 3) ? q0[0] + TS * ((q0[1] + jj) + TS * (q0[D - 1] + k))
                                                : q0[0] + TS * (q0[1] + jj);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const T wx = B.ax[0].val[i], gx = B.ax[0].der[i] * M.h_inv, N = wx * R + gx * Q;
                            T vi[3], dvi[3];
                            node_vals(t0 + i, vi, dvi);
                            const T rx = APIC ? rel(0, i) : T(0);
#pragma unroll
                            for (int r = 0; r < D; ++r) {
                                const T Nv = N * vi[r];
                                vpic[r] += Nv;
                                if constexpr (!APIC) dvf[r] += N * dvi[r];
                                gv[r][0] += (gx * wyz) * vi[r];
                                gv[r][1] += (wx * dyz) * vi[r];
                                if constexpr (D == 3) gv[r][2] += (wx * wdz) * vi[r];
                                if constexpr (APIC) {
                                    Bn[r][0] += Nv * rx;
                                    Bn[r][1] += Nv * ry;
                                    if constexpr (D == 3) Bn[r][2] += Nv * rz;
                                }
                            }
                        }
                    }
                } else if constexpr (APIC && VEC) {
                    float gx[3], rr[3][3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) gx[i] = B.ax[0].der[i] * M.h_inv;
                    if constexpr (GEN == G_APIC) {
#pragma unroll
                        for (int d = 0; d < 3; ++d)
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                if constexpr (X64)
                                    rr[d][k] = float(__dadd_rn(M.xmin64[d], __dmul_rn(double(B.ax[d].lo + k), M.h64)) - xd[d]);
                                else
                                    rr[d][k] = node_coord(M, d, B.ax[d].lo + k) - x[d];
                            }
                    }
                    const float4* tA = reinterpret_cast<const float4*>(tile);
                    const float2 z2 = make_float2(0.f, 0.f);
                    float2 p01 = z2, g0 = z2, g1 = z2, g2 = z2, b0 = z2, b1 = z2, b2 = z2;
                    float pz = 0.f, g0z = 0.f, g1z = 0.f, g2z = 0.f, b0z = 0.f, b1z = 0.f, b2z = 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) {
                            float2 A01 = z2, G01 = z2, R01 = z2;
                            float Az = 0.f, Gz = 0.f, Rz = 0.f;
                            const int t0 = q0[0] + TS * ((q0[1] + jj) + TS * (q0[2] + k));
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                const float4 a = tA[t0 + i];
                                const float wx = B.ax[0].val[i];
                                const float2 v01 = make_float2(a.x, a.y);
                                A01 = __ffma2_rn(make_float2(wx, wx), v01, A01);
                                Az = __fmaf_rn(wx, a.z, Az);
                                G01 = __ffma2_rn(make_float2(gx[i], gx[i]), v01, G01);
                                Gz = __fmaf_rn(gx[i], a.z, Gz);
                                if constexpr (GEN == G_APIC) {
                                    const float wr = wx * rr[0][i];
                                    R01 = __ffma2_rn(make_float2(wr, wr), v01, R01);
                                    Rz = __fmaf_rn(wr, a.z, Rz);
                                }
                            }
                            const float wyz = B.ax[1].val[jj] * B.ax[2].val[k];
                            const float dyz = (B.ax[1].der[jj] * M.h_inv) * B.ax[2].val[k];
                            const float wdz = B.ax[1].val[jj] * (B.ax[2].der[k] * M.h_inv);
                            const float2 W = make_float2(wyz, wyz);
                            p01 = __ffma2_rn(W, A01, p01);
                            pz = __fmaf_rn(wyz, Az, pz);
                            g0 = __ffma2_rn(W, G01, g0);
                            g0z = __fmaf_rn(wyz, Gz, g0z);
                            g1 = __ffma2_rn(make_float2(dyz, dyz), A01, g1);
                            g1z = __fmaf_rn(dyz, Az, g1z);
                            g2 = __ffma2_rn(make_float2(wdz, wdz), A01, g2);
                            g2z = __fmaf_rn(wdz, Az, g2z);
                            if constexpr (GEN == G_APIC) {
                                const float wry = wyz * rr[1][jj], wrz = wyz * rr[2][k];
                                b0 = __ffma2_rn(W, R01, b0);
                                b0z = __fmaf_rn(wyz, Rz, b0z);
                                b1 = __ffma2_rn(make_float2(wry, wry), A01, b1);
                                b1z = __fmaf_rn(wry, Az, b1z);
                                b2 = __ffma2_rn(make_float2(wrz, wrz), A01, b2);
                                b2z = __fmaf_rn(wrz, Az, b2z);
                            }
                        }
                    vpic[0] = p01.x; vpic[1] = p01.y; vpic[2] = pz;
                    gv[0][0] = g0.x; gv[1][0] = g0.y; gv[2][0] = g0z;
                    gv[0][1] = g1.x; gv[1][1] = g1.y; gv[2][1] = g1z;
                    gv[0][2] = g2.x; gv[1][2] = g2.y; gv[2][2] = g2z;
                    if constexpr (GEN == G_APIC) {
                        Bn[0][0] = b0.x; Bn[1][0] = b0.y; Bn[2][0] = b0z;
                        Bn[0][1] = b1.x; Bn[1][1] = b1.y; Bn[2][1] = b1z;
                        Bn[0][2] = b2.x; Bn[1][2] = b2.y; Bn[2][2] = b2z;
                    }
                } else if constexpr (VEC) {
                    // The separable contraction below with the component pairs of the
                    // node-major tile in packed FP32x2 FMAs; every lane of a pair is
                    // the scalar form's FMA with the same operands in the same order.
                    float gx[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) gx[i] = B.ax[0].der[i] * M.h_inv;
                    const float4* tA = reinterpret_cast<const float4*>(tile);
                    const float2* tB = reinterpret_cast<const float2*>(tile + 4 * TN);
                    const float2 z2 = make_float2(0.f, 0.f);
                    // (vpic_x, vpic_y), (vpic_z, dvf_x), (dvf_y, dvf_z), (gv_xc, gv_yc) per column c, gv_zc
                    float2 p01 = z2, p2d0 = z2, d12 = z2, g0 = z2, g1 = z2, g2 = z2;
                    float g0z = 0.f, g1z = 0.f, g2z = 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) {
                            float2 Av01 = z2, Av2d0 = z2, Ad12 = z2, Ag01 = z2;
                            float Ag2 = 0.f;
                            const int t0 = q0[0] + TS * ((q0[1] + jj) + TS * (q0[2] + k));
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                const float4 a = tA[t0 + i];
                                const float2 c = tB[t0 + i];
                                const float2 v01 = make_float2(a.x, a.y);
                                const float2 wxx = make_float2(B.ax[0].val[i], B.ax[0].val[i]);
                                const float2 gxx = make_float2(gx[i], gx[i]);
                                Av01 = __ffma2_rn(wxx, v01, Av01);
                                Av2d0 = __ffma2_rn(wxx, make_float2(a.z, a.w), Av2d0);
                                Ad12 = __ffma2_rn(wxx, c, Ad12);
                                Ag01 = __ffma2_rn(gxx, v01, Ag01);
                                Ag2 = __fmaf_rn(gx[i], a.z, Ag2);
                            }
                            const float wyz = B.ax[1].val[jj] * B.ax[2].val[k];
                            const float dyz = (B.ax[1].der[jj] * M.h_inv) * B.ax[2].val[k];
                            const float wdz = B.ax[1].val[jj] * (B.ax[2].der[k] * M.h_inv);
                            const float2 W = make_float2(wyz, wyz), DY = make_float2(dyz, dyz),
                                         DZ = make_float2(wdz, wdz);
                            p01 = __ffma2_rn(W, Av01, p01);
                            p2d0 = __ffma2_rn(W, Av2d0, p2d0);
                            d12 = __ffma2_rn(W, Ad12, d12);
                            g0 = __ffma2_rn(W, Ag01, g0);
                            g0z = __fmaf_rn(wyz, Ag2, g0z);
                            g1 = __ffma2_rn(DY, Av01, g1);
                            g1z = __fmaf_rn(dyz, Av2d0.x, g1z);
                            g2 = __ffma2_rn(DZ, Av01, g2);
                            g2z = __fmaf_rn(wdz, Av2d0.x, g2z);
                        }
                    vpic[0] = p01.x; vpic[1] = p01.y; vpic[2] = p2d0.x;
                    dvf[0] = p2d0.y; dvf[1] = d12.x; dvf[2] = d12.y;
                    gv[0][0] = g0.x; gv[1][0] = g0.y; gv[2][0] = g0z;
                    gv[0][1] = g1.x; gv[1][1] = g1.y; gv[2][1] = g1z;
                    gv[0][2] = g2.x; gv[1][2] = g2.y; gv[2][2] = g2z;
                } else {
                    // Separable contraction: sum over the x-slot first, then weight
                    // the partial sums with the y (and z) factors.
                    T dxh[3], rr[3][3] = {};
#pragma unroll
                    for (int i = 0; i < 3; ++i) dxh[i] = B.ax[0].der[i] * M.h_inv;
                    if constexpr (GEN == G_APIC) {
#pragma unroll
                        for (int d = 0; d < D; ++d)
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                if constexpr (X64)
                                    rr[d][k] = T(__dadd_rn(M.xmin64[d], __dmul_rn(double(B.ax[d].lo + k), M.h64)) - xd[d]);
                                else
                                    rr[d][k] = node_coord(M, d, B.ax[d].lo + k) - x[d];
                            }
                    }
#pragma unroll
                    for (int k = 0; k < (D == 3 ? 3 : 1); ++k)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj) {
                            T Av[3] = {T(0), T(0), T(0)}, Adv[3] = {T(0), T(0), T(0)}, Ag[3] = {T(0), T(0), T(0)};
                            T Ar[3] = {T(0), T(0), T(0)};
                            const int t0 = (D == 3) ? q0[0] + TS * ((q0[1] + jj) + TS * (q0[D - 1] + k))
                                                    : q0[0] + TS * (q0[1] + jj);
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                const T* nd = tile + (t0 + i);
                                const T wx = B.ax[0].val[i], gx = dxh[i];
#pragma unroll
                                for (int r = 0; r < D; ++r) {
                                    const T vi = nd[r * TN];
                                    Av[r] += wx * vi;
                                    if constexpr (!APIC) Adv[r] += wx * nd[(D + r) * TN];
                                    Ag[r] += gx * vi;
                                    if constexpr (GEN == G_APIC) Ar[r] += (wx * rr[0][i]) * vi;
                                }
                            }
                            T wyz, dyz, wdz;
                            if constexpr (D == 3) {
                                wyz = B.ax[1].val[jj] * B.ax[D - 1].val[k];
                                dyz = (B.ax[1].der[jj] * M.h_inv) * B.ax[D - 1].val[k];
                                wdz = B.ax[1].val[jj] * (B.ax[D - 1].der[k] * M.h_inv);
                            } else {
                                wyz = B.ax[1].val[jj];
                                dyz = B.ax[1].der[jj] * M.h_inv;
                                wdz = T(0);
                            }
#pragma unroll
                            for (int r = 0; r < D; ++r) {
                                vpic[r] += wyz * Av[r];
                                if constexpr (!APIC) dvf[r] += wyz * Adv[r];
                                gv[r][0] += wyz * Ag[r];
                                gv[r][1] += dyz * Av[r];
                                if constexpr (D == 3) gv[r][2] += wdz * Av[r];
                                if constexpr (GEN == G_APIC) {
                                    Bn[r][0] += wyz * Ar[r];
                                    Bn[r][1] += (wyz * rr[1][jj]) * Av[r];
                                    if constexpr (D == 3) Bn[r][2] += (wyz * rr[2][k]) * Av[r];
                                }
                            }
                        }
                }
                if constexpr (GEN == G_WLS_APIC) {
                    if (!B.cut) {
#pragma unroll
                        for (int r = 0; r < D; ++r)
#pragma unroll
                            for (int c = 0; c < D; ++c) Bn[r][c] = gv[r][c] * B.var[c];
                    }
                }
#pragma unroll
                for (int d = 0; d < D; ++d) dxs[d] = vpic[d] * s.dt;
            }
            if constexpr (LATE_F) load_F<D, T>(P, p, F);
            g2p_finish<D, T, VM>(P, s, p, x, vp, vpic, dvf, gv, dxs, Bn, F);
            int nb = 0;
            if constexpr (X64) {
                double xn[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    xn[d] = xd[d] + double(dxs[d]);
                    (P.x64_out[0] ? P.x64_out[d] : P.x64[d])[p] = xn[d];
                }
                if (next_bid) nb = findblock_x64<D, T>(M, xn);
            } else {
                if (next_bid) {
                    T xn[3] = {T(0), T(0), T(0)};
#pragma unroll
                    for (int d = 0; d < D; ++d) xn[d] = x[d] + dxs[d];  // the value g2p_finish stored
                    nb = findblock<D, T>(M, xn);
                }
            }
            if (next_bid) {
                // the next step's count pass: warp-aggregated, as bin_count_kernel
                next_bid[p] = nb;
                const unsigned act = __activemask();
                const unsigned peers = __match_any_sync(act, nb);
                if (nb > 0 && int(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&next_count[nb - 1], __popc(peers));
            }
        }
        __syncthreads();
    }
}

// Particle-parallel G2P reading the grid from global memory: the reference's own
// G2P schedule (one thread per particle, gpu.jl:226-232); needs no partition. The
// window is contracted as in the tiled kernel (x first, then the row's y and z
// factors; GEN as there), its rows read as three neighbouring nodes of a dense
// grid. 878 k particles, uGIMP, FP32: 0.180 ms with the weight of every node formed
// and the basis and transfer decided at run time, 0.119 ms here.
template <int D, class T, int GEN, bool VM = false>
__global__ void __launch_bounds__(128) g2p_direct_kernel(DMesh<D, T> M, GView<T> G, PView<T> P, Scalars<T> s,
                                                         int* err) {
    constexpr bool WLS = GEN == G_WLS || GEN == G_WLS_APIC, APIC = GEN == G_WLS_APIC || GEN == G_APIC;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P.n; p += (long long)gridDim.x * blockDim.x) {
        T x[3], vp[3];
        load_x<D, T>(P, p, x);
#pragma unroll
        for (int d = 0; d < D; ++d) vp[d] = P.v[d][p];
        const GimpLen<T> l = gimp_len(M, P, s, p);
        T vpic[3] = {T(0), T(0), T(0)}, dvf[3] = {T(0), T(0), T(0)}, dxs[3] = {T(0), T(0), T(0)};
        T gv[3][3] = {}, Bn[3][3] = {};
        Basis<D, T> B;
        if (prepare_basis<D, T, WLS>(M, s.basis, x, l, B, err)) {
            T dxh[3], rr[3][3] = {};
#pragma unroll
            for (int i = 0; i < 3; ++i) dxh[i] = B.ax[0].der[i] * M.h_inv;
            if constexpr (APIC) {
#pragma unroll
                for (int d = 0; d < D; ++d)
#pragma unroll
                    for (int k = 0; k < 3; ++k) rr[d][k] = node_coord(M, d, B.ax[d].lo + k) - x[d];
            }
            const bool cut = WLS && B.cut;
#pragma unroll
            for (int k = 0; k < (D == 3 ? 3 : 1); ++k)
#pragma unroll
                for (int jj = 0; jj < 3; ++jj) {
                    if (jj >= B.ax[1].cnt || (D == 3 && k >= B.ax[D - 1].cnt)) continue;
                    const int y = B.ax[1].lo + jj, z = D == 3 ? B.ax[D - 1].lo + k : 0;
                    const long long row = G.bnum ? 0 : grid_slot<D>(G, M, B.ax[0].lo, y, z);
                    T Av[3] = {T(0), T(0), T(0)}, Adv[3] = {T(0), T(0), T(0)}, Ag[3] = {T(0), T(0), T(0)};
                    T Agd[3] = {T(0), T(0), T(0)}, Ar[3] = {T(0), T(0), T(0)}, Agr[3] = {T(0), T(0), T(0)};
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        if (i >= B.ax[0].cnt) continue;
                        const long long lin = G.bnum ? grid_slot<D>(G, M, B.ax[0].lo + i, y, z) : row + i;
                        if (lin < 0) continue;  // not stored by a sparse grid: reads as zero
                        const T wx = B.ax[0].val[i], gx = dxh[i];
#pragma unroll
                        for (int r = 0; r < D; ++r) {
                            const T vi = __ldg(G.v[r] + lin);
                            Av[r] += wx * vi;
                            Ag[r] += gx * vi;
                            if constexpr (!APIC) {
                                const T dv = vi - __ldg(G.vn[r] + lin);
                                Adv[r] += wx * dv;
                                if constexpr (WLS) Agd[r] += gx * dv;
                            }
                            if constexpr (APIC) {
                                Ar[r] += (wx * rr[0][i]) * vi;
                                if constexpr (WLS) Agr[r] += (gx * rr[0][i]) * vi;
                            }
                        }
                    }
                    T wyz, dyz, wdz;
                    if constexpr (D == 3) {
                        wyz = B.ax[1].val[jj] * B.ax[D - 1].val[k];
                        dyz = (B.ax[1].der[jj] * M.h_inv) * B.ax[D - 1].val[k];
                        wdz = B.ax[1].val[jj] * (B.ax[D - 1].der[k] * M.h_inv);
                    } else {
                        wyz = B.ax[1].val[jj];
                        dyz = B.ax[1].der[jj] * M.h_inv;
                        wdz = T(0);
                    }
                    // the row's N_x = wx R + gx Q (WLS windows that the mesh cuts; else R = wyz, Q = 0)
                    T R = wyz, Q = T(0);
                    if (cut) {
                        R -= B.u[1] * dyz + (D == 3 ? B.u[D - 1] * wdz : T(0));
                        Q = -B.u[0] * wyz;
                    }
#pragma unroll
                    for (int r = 0; r < D; ++r) {
                        gv[r][0] += wyz * Ag[r];
                        gv[r][1] += dyz * Av[r];
                        if constexpr (D == 3) gv[r][2] += wdz * Av[r];
                        T Nv = R * Av[r];
                        if constexpr (WLS) Nv += Q * Ag[r];
                        vpic[r] += Nv;
                        if constexpr (!APIC) {
                            dvf[r] += R * Adv[r];
                            if constexpr (WLS) dvf[r] += Q * Agd[r];
                        }
                        if constexpr (APIC) {
                            Bn[r][0] += R * Ar[r];
                            if constexpr (WLS) Bn[r][0] += Q * Agr[r];
                            Bn[r][1] += Nv * rr[1][jj];
                            if constexpr (D == 3) Bn[r][2] += Nv * rr[2][k];
                        }
                    }
                }
#pragma unroll
            for (int d = 0; d < D; ++d) dxs[d] = vpic[d] * s.dt;
        }
        double F[3][3];
        load_F<D, T>(P, p, F);
        g2p_finish<D, T, VM>(P, s, p, x, vp, vpic, dvf, gv, dxs, Bn, F);
    }
}

// Particles outside the mesh (block id 0): empty window, so only the particle
// equations run (v and x keep their values under FLIP).
template <int D, class T, bool VM = false>
__global__ void __launch_bounds__(256) g2p_outside_kernel(PView<T> P, Scalars<T> s, const int* __restrict__ blockids,
                                                          const int* __restrict__ totals) {
    chain_wait();
    if ((long long)totals[1] >= P.n) return;  // every particle is inside a block
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P.n; p += (long long)gridDim.x * blockDim.x) {
        if (blockids[p] != 0) continue;
        T x[3], vp[3], z[3] = {T(0), T(0), T(0)};
        T gv[3][3] = {}, Bn[3][3] = {};
#pragma unroll
        for (int d = 0; d < D; ++d) {
            x[d] = P.x[0] ? P.x[d][p] : T(0);  // FP64 positions stay as they are
            vp[d] = P.v[d][p];
        }
        double F[3][3];
        load_F<D, T>(P, p, F);
        g2p_finish<D, T, VM>(P, s, p, x, vp, z, z, gv, z, Bn, F);
    }
}

// c = sqrt((lambda + 2 mu) / (m / V)) + |v| per particle, the Taylor impact's
// speed for its time step (docs/src/gpu.md:283-284); the maximum goes to *out
// as the bits of a non-negative double, which order as unsigned integers.
template <int D, class T>
__global__ void __launch_bounds__(256) wave_speed_kernel(PView<T> P, Scalars<T> s, unsigned long long* out) {
    double cmax = 0.0;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P.n; p += (long long)gridDim.x * blockDim.x) {
        const double mu = P.mu ? double(P.mu[p]) : s.mu;
        const double lam = P.lam ? double(P.lam[p]) : s.lam;
        const double m = P.m ? double(P.m[p]) : double(s.mass);
        double vv = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) vv += double(P.v[d][p]) * double(P.v[d][p]);
        const double c = sqrt((lam + 2.0 * mu) / (m / double(P.V[p]))) + sqrt(vv);
        cmax = fmax(cmax, c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cmax = fmax(cmax, __shfl_down_sync(0xffffffffu, cmax, o));
    if ((threadIdx.x & 31) == 0 && cmax > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(cmax));
}

// update!(weights, particles, mesh) with stored values (basis_weight.jl:714-752):
// w in (3,3,3,n) column-major, grad_w as Vec{D} per slot, window as 1-based
// (start, stop) Int64 pairs; slots outside a truncated window are zeroed.
template <int D, class T>
__global__ void __launch_bounds__(128) update_weights_kernel(DMesh<D, T> M, PView<T> P, Scalars<T> s, T* w_out,
                                                             T* gw_out, long long* win_out, int* err) {
    constexpr int NW = (D == 3) ? 27 : 9;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P.n; p += (long long)gridDim.x * blockDim.x) {
        T x[3];
        load_x<D, T>(P, p, x);
        const GimpLen<T> l = gimp_len(M, P, s, p);
        Basis<D, T> B;
        const bool ok = prepare_basis<D, T>(M, s.basis, x, l, B, err);
        for (int slot = 0; slot < NW; ++slot) {
            const int i = slot % 3, jj = (slot / 3) % 3, k = slot / 9;
            T w = T(0), dw[3] = {T(0), T(0), T(0)};
            if (ok && i < B.ax[0].cnt && jj < B.ax[1].cnt && (D == 2 || k < B.ax[D - 1].cnt)) {
                eval_node<D, T>(M, B, i, jj, k, w, dw);
            }
            w_out[p * NW + slot] = w;
#pragma unroll
            for (int d = 0; d < D; ++d) gw_out[(p * NW + slot) * D + d] = dw[d];
        }
#pragma unroll
        for (int d = 0; d < D; ++d) {
            win_out[p * 2 * D + 2 * d] = ok ? B.ax[d].lo + 1 : 1;
            win_out[p * 2 * D + 2 * d + 1] = ok ? B.ax[d].lo + B.ax[d].cnt : 0;
        }
    }
}

template <class K>
int occupancy_grid(K kernel, int threads, int num_sms) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
    return num_sms * (per_sm > 0 ? per_sm : 1);
}

}  // namespace

// m, mv and f of every stored node to zero, one launch at every size. Memsets would
// have to be one per array (adjoining arrays need not be one allocation, and a memset
// across two is an error), and seven of them measured slower than the kernel at every
// size: FP32, 1 M nodes 0.032 against 0.010 ms, 4.2 M 0.044 against 0.023 ms, 16.8 M
// 0.089 against 0.076 ms.
template <int D, class T>
cudaError_t launch_grid_zero(const DMesh<D, T>& M, const GView<T>& G, const LaunchCfg& cfg) {
    const long long nn = G.bnum ? G.cap : M.nnodes;  // a sparse grid's count is on the device
    KernelScope ks(cfg, "grid_zero");
    const int grid = int(std::min<long long>((nn + 31 + 255) / 256, (long long)cfg.num_sms * 16));
    launch_chained(grid_zero_kernel<D, T>, grid, 256, 0, cfg, G, nn);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T>
cudaError_t launch_grid_update(const DMesh<D, T>& M, const GView<T>& G, const Scalars<T>& s, const LaunchCfg& cfg) {
    KernelScope ks(cfg, "grid_update");
    if (G.bnum) {
        const int grid = int(std::min<long long>((G.cap + 255) / 256, (long long)cfg.num_sms * 16));
        grid_update_sparse_kernel<D, T><<<std::max(grid, 1), 256, 0, cfg.stream>>>(M, G, s);
    } else {
        const int grid = int(std::min<long long>((M.nnodes + 255) / 256, (long long)cfg.num_sms * 16));
        launch_chained(grid_update_kernel<D, T>, grid, 256, 0, cfg, M, G, s);
    }
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T, int BW, int GEN>
cudaError_t launch_g2p_kind(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                            const BinBuffers& b, const LaunchCfg& cfg, bool count_next, bool x64, bool vm) {
    auto kern = g2p_tile_kernel<D, T, BW, GEN, false>;
    if constexpr (D == 3) {
        if (vm) kern = g2p_tile_kernel<D, T, BW, GEN, false, true>;
    }
    if constexpr (sizeof(T) == 4) {
        if (x64) {
            kern = g2p_tile_kernel<D, T, BW, GEN, true>;
            if constexpr (D == 3) {
                if (vm) kern = g2p_tile_kernel<D, T, BW, GEN, true, true>;
            }
        }
    }
    const int grid = std::min(occupancy_grid(kern, 128, cfg.num_sms), 8 * M.nblocks);  // blocks may be split
    {
        // first: it reads this step's block ids, which the tiled pass below
        // replaces with the next step's when it counts
        KernelScope ks(cfg, "g2p_outside");
        const int og = int(std::min<long long>((P.n + 255) / 256, (long long)cfg.num_sms * 8));
        if (D == 3 && s.material == TB_MATERIAL_VONMISES)
            launch_chained(g2p_outside_kernel<D, T, D == 3>, og, 256, 0, cfg, P, s, b.blockids, b.totals);
        else
            launch_chained(g2p_outside_kernel<D, T>, og, 256, 0, cfg, P, s, b.blockids, b.totals);
    }
    KernelScope ks(cfg, "g2p");
    launch_chained(kern, grid, 128, 0, cfg, M, G, P, s, b.totals, b.blocklist, b.offsets, b.perm, cfg.err,
                   count_next ? b.blockids : nullptr, count_next ? b.counts : nullptr);
    *cfg.launches += 2;
    return cudaGetLastError();
}

template <int D, class T, int BW>
cudaError_t launch_g2p(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                       const BinBuffers& b, const LaunchCfg& cfg, bool count_next) {
    if (P.n == 0) return cudaSuccess;
    const bool wls = s.basis == TB_WLS_BSPLINE_QUADRATIC || s.basis == TB_WLS_UGIMP;
    const bool apic = s.transfer == TB_TRANSFER_APIC;
    const bool vm = s.material == TB_MATERIAL_VONMISES;  // 3D only (checked by the caller)
    const bool x64 = P.x64[0] != nullptr;  // FP64-position form: FP32 state only (checked by the caller)
    if (x64 && sizeof(T) != 4) return cudaErrorInvalidValue;
    if (!wls && !apic) return launch_g2p_kind<D, T, BW, G_PLAIN>(M, G, P, s, b, cfg, count_next, x64, vm);
    if (!apic) return launch_g2p_kind<D, T, BW, G_WLS>(M, G, P, s, b, cfg, count_next, x64, vm);
    if (wls) return launch_g2p_kind<D, T, BW, G_WLS_APIC>(M, G, P, s, b, cfg, count_next, x64, vm);
    return launch_g2p_kind<D, T, BW, G_APIC>(M, G, P, s, b, cfg, count_next, x64, vm);
}

template <int D, class T, int GEN>
void launch_g2p_direct_kind(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                            const LaunchCfg& cfg) {
    const int grid = int(std::min<long long>((P.n + 127) / 128, (long long)cfg.num_sms * 32));
    if (D == 3 && s.material == TB_MATERIAL_VONMISES)
        g2p_direct_kernel<D, T, GEN, D == 3><<<grid, 128, 0, cfg.stream>>>(M, G, P, s, cfg.err);
    else
        g2p_direct_kernel<D, T, GEN><<<grid, 128, 0, cfg.stream>>>(M, G, P, s, cfg.err);
}

template <int D, class T>
cudaError_t launch_g2p_direct(const DMesh<D, T>& M, const GView<T>& G, const PView<T>& P, const Scalars<T>& s,
                              const LaunchCfg& cfg) {
    if (P.n == 0) return cudaSuccess;
    const bool wls = s.basis == TB_WLS_BSPLINE_QUADRATIC || s.basis == TB_WLS_UGIMP;
    const bool apic = s.transfer == TB_TRANSFER_APIC;
    KernelScope ks(cfg, "g2p_direct");
    if (wls && apic) launch_g2p_direct_kind<D, T, G_WLS_APIC>(M, G, P, s, cfg);
    else if (wls) launch_g2p_direct_kind<D, T, G_WLS>(M, G, P, s, cfg);
    else if (apic) launch_g2p_direct_kind<D, T, G_APIC>(M, G, P, s, cfg);
    else launch_g2p_direct_kind<D, T, G_PLAIN>(M, G, P, s, cfg);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T, int BW>
cudaError_t launch_sparse_zero(const DMesh<D, T>& M, const GView<T>& G, const int* list, const int* count,
                               const LaunchCfg& cfg) {
    const int grid = int(std::max(1ll, std::min((M.nblocks * 32ll + 255) / 256, cfg.num_sms * 16ll)));
    KernelScope ks(cfg, "grid_zero");
    launch_chained(node_list_kernel<D, T, BW, 0>, grid, 256, 0, cfg, M, G, Scalars<T>{}, nullptr, list, count, 0);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T, int BW>
cudaError_t launch_sparse_grid_update(const DMesh<D, T>& M, const GView<T>& G, const Scalars<T>& s,
                                      const unsigned char* cur, const int* list, const int* count,
                                      const LaunchCfg& cfg, bool zero_after) {
    const int grid = int(std::max(1ll, std::min((M.nblocks * 32ll + 255) / 256, cfg.num_sms * 16ll)));
    KernelScope ks(cfg, "grid_update");
    launch_chained(node_list_kernel<D, T, BW, 1>, grid, 256, 0, cfg, M, G, s, cur, list, count, zero_after ? 1 : 0);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T>
cudaError_t launch_wave_speed(const PView<T>& P, const Scalars<T>& s, unsigned long long* out, const LaunchCfg& cfg) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), cfg.stream);
    if (e != cudaSuccess || P.n == 0) return e;
    const int grid = int(std::max<long long>(1, std::min<long long>((P.n + 255) / 256, (long long)cfg.num_sms * 8)));
    KernelScope ks(cfg, "wave_speed");
    wave_speed_kernel<D, T><<<grid, 256, 0, cfg.stream>>>(P, s, out);
    ++*cfg.launches;
    return cudaGetLastError();
}

template <int D, class T>
cudaError_t launch_update_weights(const DMesh<D, T>& M, const PView<T>& P, const Scalars<T>& s, T* w, T* gw,
                                  long long* win, const LaunchCfg& cfg) {
    if (P.n == 0) return cudaSuccess;
    const int grid = int(std::min<long long>((P.n + 127) / 128, (long long)cfg.num_sms * 16));
    KernelScope ks(cfg, "update_weights");
    update_weights_kernel<D, T><<<grid, 128, 0, cfg.stream>>>(M, P, s, w, gw, win, cfg.err);
    ++*cfg.launches;
    return cudaGetLastError();
}

#define TB_INST_T(D, T)                                                                                      \
    template cudaError_t launch_grid_update<D, T>(const DMesh<D, T>&, const GView<T>&, const Scalars<T>&,   \
                                                  const LaunchCfg&);                                         \
    template cudaError_t launch_grid_zero<D, T>(const DMesh<D, T>&, const GView<T>&, const LaunchCfg&);     \
    template cudaError_t launch_update_weights<D, T>(const DMesh<D, T>&, const PView<T>&, const Scalars<T>&, \
                                                     T*, T*, long long*, const LaunchCfg&);                  \
    template cudaError_t launch_g2p_direct<D, T>(const DMesh<D, T>&, const GView<T>&, const PView<T>&,       \
                                                 const Scalars<T>&, const LaunchCfg&);                     \
    template cudaError_t launch_wave_speed<D, T>(const PView<T>&, const Scalars<T>&, unsigned long long*,    \
                                                 const LaunchCfg&);
#define TB_INST_TB(D, T, BW)                                                                                 \
    template cudaError_t launch_sparse_zero<D, T, BW>(const DMesh<D, T>&, const GView<T>&, const int*,         \
                                                      const int*, const LaunchCfg&);                           \
    template cudaError_t launch_sparse_grid_update<D, T, BW>(const DMesh<D, T>&, const GView<T>&,              \
                                                             const Scalars<T>&, const unsigned char*,          \
                                                             const int*, const int*, const LaunchCfg&, bool);  \
    template cudaError_t launch_g2p<D, T, BW>(const DMesh<D, T>&, const GView<T>&, const PView<T>&,         \
                                              const Scalars<T>&, const BinBuffers&, const LaunchCfg&, bool);

TB_INST_T(3, double)
TB_INST_T(3, float)
TB_INST_T(2, double)
TB_INST_T(2, float)
TB_INST_TB(3, double, 4)
TB_INST_TB(3, float, 4)
TB_INST_TB(2, double, 8)
TB_INST_TB(2, float, 8)
TB_INST_TB(2, double, 4)
TB_INST_TB(2, float, 4)

}  // namespace tb
