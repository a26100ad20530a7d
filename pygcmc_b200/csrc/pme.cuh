// Ewald electrostatics by smooth particle-mesh Ewald (Essmann et al., J. Chem.
// Phys. 103 (1995) 8577), FP64 mesh; not in the reference, whose calcEnergy
// uses a plain cutoff.
//
// Each replica keeps its spread charges Q on the mesh: the fixed atoms and the
// occupied fragment atoms spread with order-4 cardinal B-splines once at
// set-up; afterwards the accept kernel spreads the change of every accepted
// move (-q at a molecule's old sites, +q at its new ones) and marks the mesh
// dirty.  Before a step's pose energies, a dirty mesh's potential is
// recomputed, phi_mesh = IFFT(G * FFT(Q)) with G(m) = K exp(-pi^2 m^2 /
// alpha^2) B(m) / (pi V m^2), B the B-spline moduli, by the hand-written FP64
// transforms of fft.cuh; after a step that accepted nothing every pass
// returns at once.  The potential at a point is the same B-spline
// interpolation of phi_mesh.
//
// Energy of a trial pose p (sites r_s, charges q_s) under Ewald:
//   E(p) = sum_{pairs in the group cutoff} [LJ + K q_s q_a erfc(alpha r) / r]
//        + sum_s q_s phi(r_s)
//        - [p replaces occupied group M]  K sum_{s, t in M} q_s q_t g(|r_s - x_t|)
//        (+ the neutralising-background change for insert / delete, added by
//         the accept kernel), g(r) = erf(alpha r) / r, g(0) = 2 alpha / sqrt(pi).
// The molecule's self and intramolecular terms cancel exactly for an insertion
// (its own Coulomb pairs are excluded); the g term removes a moving or
// leaving molecule's own field from phi.  Neglected: the molecule's
// interaction with its own periodic images beyond erf(alpha r)/r (a smooth
// term of order q^2 / L^3 for these box sizes).
#pragma once
#include "common.cuh"
#include "fft.cuh"

namespace gcmc {

// order-4 B-spline weights of the four mesh points floor(u) - j, j = 0..3
__device__ __forceinline__ void bspline4(double w, double m[4]) {
    const double w2 = w * w, w3 = w2 * w, c = 1.0 - w, sixth = 1.0 / 6.0;
    m[0] = w3 * sixth;
    m[1] = (-3.0 * w3 + 3.0 * w2 + 3.0 * w + 1.0) * sixth;
    m[2] = (3.0 * w3 - 6.0 * w2 + 4.0) * sixth;
    m[3] = c * c * c * sixth;
}

__device__ __forceinline__ int wrapm(int k, int n) {
    k %= n;
    return k < 0 ? k + n : k;
}

// mesh coordinate of x along axis a
__device__ __forceinline__ double mesh_u(const RepDev& R, double x, int a) {
    return ((x - (double)R.start[a]) / (double)R.L[a]) * (double)R.pme_n[a];
}

// derivatives of bspline4's weights with respect to w
__device__ __forceinline__ void bspline4_d(double w, double d[4]) {
    const double c = 1.0 - w;
    d[0] = 0.5 * w * w;
    d[1] = 0.5 * (-3.0 * w * w + 2.0 * w + 1.0);
    d[2] = 0.5 * (3.0 * w * w - 4.0 * w);
    d[3] = -0.5 * c * c;
}

// phi at a point by the same interpolation
__device__ __forceinline__ double pme_phi_at(const RepDev& R, double x, double y, double z) {
    double mx[4], my[4], mz[4];
    const double ux = mesh_u(R, x, 0), uy = mesh_u(R, y, 1), uz = mesh_u(R, z, 2);
    const double fx = floor(ux), fy = floor(uy), fz = floor(uz);
    bspline4(ux - fx, mx);
    bspline4(uy - fy, my);
    bspline4(uz - fz, mz);
    const int n0 = R.pme_n[0], n1 = R.pme_n[1], n2 = R.pme_n[2];
    double p = 0.0;
    for (int a = 0; a < 4; ++a) {
        const int i0 = wrapm((int)fx - a, n0);
        for (int b = 0; b < 4; ++b) {
            const int i1 = wrapm((int)fy - b, n1);
            const double* row = R.pme_phi + ((size_t)i0 * n1 + i1) * n2;
            double t = 0.0;
            for (int c = 0; c < 4; ++c) t += mz[c] * __ldg(row + wrapm((int)fz - c, n2));
            p += mx[a] * my[b] * t;
        }
    }
    return p;
}

// ---- the mesh transforms ----
//
// Planes (a context whose planes n1 x n2 fit, twice, in shared memory; 128 x 96
// and 81 x 96 do, 128 x 128 does not): three passes over the mesh,
//   1. k_pme_fwd_planes: a CTA per plane, rows real-to-complex, then axis 1;
//   2. k_pme_axis: axis 0 forward, times G, axis 0 inverse;
//   3. k_pme_inv_planes: a CTA per plane, axis 1 inverse, then rows to real.
// Otherwise passes 1 and 3 are two each (k_pme_rows_r2c + k_pme_axis along
// axis 1, and back).  Two real rows share one complex transform (one is the
// real, the other the imaginary part), which halves the row work for odd and
// even lengths alike.  All replicas of a launch are one list of items that the
// CTAs share (a replica whose mesh is current contributes none), so a batch
// takes as many launches as one replica.
// Bound: shared-memory passes and barriers per CTA (a 64 x 64 plane: four
// stages), then L2 traffic; the mesh of one replica stays in L2 between passes.
// Measured (average launch, about half of them of clean meshes): one 64^3 mesh
// 8.1 + 7.6 + 9.3 us, against 68 us for six launches with a sincospi per
// butterfly, radix 2 and 3 and a complex transform per real row; 4 replicas
// of a 128 x 128 x 96 mesh 75 + 73 + 78 us, against 4 x 228 us.
// Threads of a plane's CTA: one CTA fills an SM's shared memory from about 128 x 64 on, so
// large planes take more warps (16 replicas of 128 x 128 x 96: 926 -> 893 us a step with
// 768 threads; a 64 x 64 plane is slower with them).
constexpr int kPlaneThreads = 768;
inline int pme_plane_threads(size_t elems) { return elems >= 4096 ? kPlaneThreads : 512; }
constexpr int kAxisThreads = 256;
constexpr int kAxisLines = 16;   // columns (256 bytes of each row) per axis item
constexpr int kRowPairs = 8;     // row pairs per item of the separate row passes
constexpr int kPmeSmemMax = 220 * 1024;

// Complex elements of one of the plane passes' two buffers.
__host__ __device__ inline size_t pme_plane_elems(int n1, int n2) {
    const size_t rows = (size_t)n2 * (((n1 + 1) / 2) | 1), cols = (size_t)n1 * ((n2 / 2 + 1) | 1);
    return rows > cols ? rows : cols;
}
__host__ __device__ inline size_t pme_plane_smem(int n1, int n2) {
    return (2 * pme_plane_elems(n1, n2) + n1 + n2) * sizeof(double2);
}
__host__ __device__ inline size_t pme_axis_smem(int n) { return (size_t)(2 * kAxisLines + 1) * n * sizeof(double2); }
__host__ __device__ inline size_t pme_rows_smem(int n2) {
    return (size_t)(2 * (kRowPairs | 1) + 1) * n2 * sizeof(double2);
}

__device__ __forceinline__ bool pme_stale(const RepDev& R) {
    return R.pme && *reinterpret_cast<const volatile int*>(R.pme_dirty) != 0;
}

// The replica whose items hold `it` (pre[r] <= it < pre[r + 1]).
__device__ __forceinline__ int prefix_find(const int* pre, int nrep, int it) {
    int lo = 0, hi = nrep;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] <= it) lo = mid; else hi = mid;
    }
    return lo;
}

// The roots of axis a into shared memory (whole CTA, no barrier).
__device__ __forceinline__ void load_roots(const RepDev& R, int a, double2* tw) {
    const int off = a == 0 ? 0 : (a == 1 ? R.pme_n[0] : R.pme_n[0] + R.pme_n[1]);
    for (int i = threadIdx.x; i < R.pme_n[a]; i += blockDim.x) tw[i] = R.pme_tw[off + i];
}

// nrow real rows of length n2 from `src`, in pairs: pair j = row 2j + i row 2j + 1
// (0 past the last row), element i of pair j at b[i * ld + j].
__device__ __forceinline__ void load_row_pairs(const double* __restrict__ src, int nrow, int n2, double2* b, int ld) {
    const int np = (nrow + 1) >> 1;
    const FastDiv by_n2(n2);
#pragma unroll 4
    for (int e = threadIdx.x; e < np * n2; e += blockDim.x) {
        const int j = by_n2.quot(e), i = e - j * n2;
        const double* p = src + (size_t)(2 * j) * n2 + i;
        b[i * ld + j] = make_double2(p[0], 2 * j + 1 < nrow ? p[n2] : 0.0);
    }
}

// Half spectra of the two rows of a transformed pair, Z[k] and Z[n - k]:
// X_a = (Z[k] + conj Z[n - k]) / 2, X_b = (Z[k] - conj Z[n - k]) / 2i.
__device__ __forceinline__ void split_pair(double2 z, double2 w, double2& xa, double2& xb) {
    xa = make_double2(0.5 * (z.x + w.x), 0.5 * (z.y - w.y));
    xb = make_double2(0.5 * (z.y + w.y), 0.5 * (w.x - z.x));
}
// X_a + i X_b at k, from the half spectra (Hermitian extension past n / 2).
__device__ __forceinline__ double2 join_pair(double2 xa, double2 xb, bool mirrored) {
    return mirrored ? make_double2(xa.x + xb.y, xb.x - xa.y) : make_double2(xa.x - xb.y, xa.y + xb.x);
}

__global__ void __launch_bounds__(kPlaneThreads) k_pme_fwd_planes(const RepDev* __restrict__ reps, int nrep) {
    extern __shared__ __align__(16) double2 fbuf[];
    __shared__ int pre[257];
    __shared__ int wtot[32];
    items_prefix(nrep, pre, wtot, [&](int r) { return pme_stale(reps[r]) ? reps[r].pme_n[0] : 0; });
    for (int it = blockIdx.x; it < pre[nrep]; it += gridDim.x) {
        const int r = prefix_find(pre, nrep, it), i0 = it - pre[r];
        const RepDev& R = reps[r];
        const int n1 = R.pme_n[1], n2 = R.pme_n[2], M = n2 / 2 + 1, np = (n1 + 1) >> 1;
        const int ldp = np | 1, ldc = M | 1;
        const size_t S = pme_plane_elems(n1, n2);
        double2 *b0 = fbuf, *b1 = fbuf + S, *tw1 = fbuf + 2 * S, *tw2 = tw1 + n1;
        __syncthreads();
        load_roots(R, 1, tw1);
        load_roots(R, 2, tw2);
        load_row_pairs(R.pme_q + (size_t)i0 * n1 * n2, n1, n2, b0, ldp);
        double2* z = fft_lines_block(b0, b1, ldp, np, n2, tw2, -1);
        double2* c = z == b0 ? b1 : b0;
        const FastDiv by_np(np), by_M(M);
        for (int e = threadIdx.x; e < np * M; e += blockDim.x) {  // [i1][k2]
            const int k = by_np.quot(e), j = e - k * np;
            double2 xa, xb;
            split_pair(z[k * ldp + j], z[(k ? n2 - k : 0) * ldp + j], xa, xb);
            c[2 * j * ldc + k] = xa;
            if (2 * j + 1 < n1) c[(2 * j + 1) * ldc + k] = xb;
        }
        const double2* out = fft_lines_block(c, z, ldc, M, n1, tw1, -1);
        double2* dst = R.pme_spec + (size_t)i0 * n1 * M;
#pragma unroll 4
        for (int e = threadIdx.x; e < n1 * M; e += blockDim.x) {
            const int i = by_M.quot(e), k = e - i * M;
            dst[e] = out[i * ldc + k];
        }
    }
}

// After the last pass over the meshes of a launch: the last CTA to finish marks
// them current (every CTA has read the marks at its start).
__device__ __forceinline__ void pme_finish(const RepDev* __restrict__ reps, int nrep) {
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&reps[0].pme_dirty[1], 1) == (int)gridDim.x - 1) {
        for (int r = 0; r < nrep; ++r)
            if (reps[r].pme) reps[r].pme_dirty[0] = 0;
        reps[0].pme_dirty[1] = 0;
    }
}

__global__ void __launch_bounds__(kPlaneThreads) k_pme_inv_planes(const RepDev* __restrict__ reps, int nrep) {
    extern __shared__ __align__(16) double2 fbuf[];
    __shared__ int pre[257];
    __shared__ int wtot[32];
    items_prefix(nrep, pre, wtot, [&](int r) { return pme_stale(reps[r]) ? reps[r].pme_n[0] : 0; });
    for (int it = blockIdx.x; it < pre[nrep]; it += gridDim.x) {
        const int r = prefix_find(pre, nrep, it), i0 = it - pre[r];
        const RepDev& R = reps[r];
        const int n1 = R.pme_n[1], n2 = R.pme_n[2], M = n2 / 2 + 1, np = (n1 + 1) >> 1;
        const int ldp = np | 1, ldc = M | 1;
        const size_t S = pme_plane_elems(n1, n2);
        double2 *b0 = fbuf, *b1 = fbuf + S, *tw1 = fbuf + 2 * S, *tw2 = tw1 + n1;
        __syncthreads();
        load_roots(R, 1, tw1);
        load_roots(R, 2, tw2);
        const double2* src = R.pme_spec + (size_t)i0 * n1 * M;
        const FastDiv by_np(np), by_M(M), by_n2(n2);
#pragma unroll 4
        for (int e = threadIdx.x; e < n1 * M; e += blockDim.x) {
            const int i = by_M.quot(e), k = e - i * M;
            b0[i * ldc + k] = src[e];
        }
        double2* c = fft_lines_block(b0, b1, ldc, M, n1, tw1, 1);
        double2* z = c == b0 ? b1 : b0;
        for (int e = threadIdx.x; e < np * n2; e += blockDim.x) {
            const int k = by_np.quot(e), j = e - k * np;
            const bool mir = k >= M;
            const int kk = mir ? n2 - k : k;
            const double2 xb = 2 * j + 1 < n1 ? c[(2 * j + 1) * ldc + kk] : make_double2(0.0, 0.0);
            z[k * ldp + j] = join_pair(c[2 * j * ldc + kk], xb, mir);
        }
        const double2* out = fft_lines_block(z, c, ldp, np, n2, tw2, 1);
        double* phi = const_cast<double*>(R.pme_phi) + (size_t)i0 * n1 * n2;
#pragma unroll 4
        for (int e = threadIdx.x; e < np * n2; e += blockDim.x) {
            const int j = by_n2.quot(e), i = e - j * n2;
            const double2 v = out[i * ldp + j];
            phi[(size_t)(2 * j) * n2 + i] = v.x;
            if (2 * j + 1 < n1) phi[(size_t)(2 * j + 1) * n2 + i] = v.y;
        }
    }
    pme_finish(reps, nrep);
}

// Transforms along axis 0 or 1 of the half spectrum: the mesh is `outer`
// matrices of n rows and C contiguous columns (axis 0: one, n0 x (n1 M); axis
// 1: n0, n1 x M), an item is kAxisLines columns of one of them.  sign -1
// forward, +1 inverse; fuse_g: forward, times G, inverse.
__global__ void __launch_bounds__(kAxisThreads) k_pme_axis(const RepDev* __restrict__ reps, int nrep, int axis,
                                                           int sign, int fuse_g) {
    extern __shared__ __align__(16) double2 fbuf[];
    __shared__ int pre[257];
    __shared__ int wtot[32];
    auto columns = [&](const RepDev& R) { return (axis == 0 ? R.pme_n[1] : 1) * (R.pme_n[2] / 2 + 1); };
    items_prefix(nrep, pre, wtot, [&](int r) {
        if (!pme_stale(reps[r])) return 0;
        return (axis == 0 ? 1 : reps[r].pme_n[0]) * ((columns(reps[r]) + kAxisLines - 1) / kAxisLines);
    });
    for (int it = blockIdx.x; it < pre[nrep]; it += gridDim.x) {
        const int r = prefix_find(pre, nrep, it);
        const RepDev& R = reps[r];
        const int n = R.pme_n[axis], C = columns(R), cb = (C + kAxisLines - 1) / kAxisLines;
        const int o = (it - pre[r]) / cb, c0 = (it - pre[r] - o * cb) * kAxisLines;
        const int nl = min(kAxisLines, C - c0);
        const size_t base = (size_t)o * n * C + c0;
        double2 *b0 = fbuf, *b1 = fbuf + kAxisLines * n, *tw = b1 + kAxisLines * n;
        __syncthreads();
        load_roots(R, axis, tw);
#pragma unroll 4
        for (int e = threadIdx.x; e < n * kAxisLines; e += blockDim.x) {
            const int i = e / kAxisLines, b = e % kAxisLines;
            if (b < nl) b0[e] = R.pme_spec[base + (size_t)i * C + b];
        }
        double2* out = fft_lines_block(b0, b1, kAxisLines, nl, n, tw, fuse_g ? -1 : sign);
        if (fuse_g) {
            for (int e = threadIdx.x; e < n * kAxisLines; e += blockDim.x) {
                const int i = e / kAxisLines, b = e % kAxisLines;
                if (b < nl) {
                    const double g = R.pme_g[base + (size_t)i * C + b];
                    out[e] = make_double2(g * out[e].x, g * out[e].y);
                }
            }
            out = fft_lines_block(out, out == b0 ? b1 : b0, kAxisLines, nl, n, tw, 1);
        }
        for (int e = threadIdx.x; e < n * kAxisLines; e += blockDim.x) {
            const int i = e / kAxisLines, b = e % kAxisLines;
            if (b < nl) R.pme_spec[base + (size_t)i * C + b] = out[e];
        }
    }
}

// The row passes alone (planes that do not fit in shared memory): an item is
// kRowPairs pairs of consecutive rows.
__device__ __forceinline__ int row_items(const RepDev& R) {
    return (R.pme_n[0] * R.pme_n[1] + 2 * kRowPairs - 1) / (2 * kRowPairs);
}
__global__ void __launch_bounds__(kAxisThreads) k_pme_rows_r2c(const RepDev* __restrict__ reps, int nrep) {
    extern __shared__ __align__(16) double2 fbuf[];
    __shared__ int pre[257];
    __shared__ int wtot[32];
    items_prefix(nrep, pre, wtot, [&](int r) { return pme_stale(reps[r]) ? row_items(reps[r]) : 0; });
    for (int it = blockIdx.x; it < pre[nrep]; it += gridDim.x) {
        const int r = prefix_find(pre, nrep, it);
        const RepDev& R = reps[r];
        const int n2 = R.pme_n[2], M = n2 / 2 + 1, ld = kRowPairs | 1;
        const int r0 = (it - pre[r]) * 2 * kRowPairs, nrow = min(2 * kRowPairs, R.pme_n[0] * R.pme_n[1] - r0);
        const int np = (nrow + 1) >> 1;
        double2 *b0 = fbuf, *b1 = fbuf + ld * n2, *tw = b1 + ld * n2;
        __syncthreads();
        load_roots(R, 2, tw);
        load_row_pairs(R.pme_q + (size_t)r0 * n2, nrow, n2, b0, ld);
        const double2* z = fft_lines_block(b0, b1, ld, np, n2, tw, -1);
        const FastDiv by_M(M);
        for (int e = threadIdx.x; e < np * M; e += blockDim.x) {
            const int j = by_M.quot(e), k = e - j * M;
            double2 xa, xb;
            split_pair(z[k * ld + j], z[(k ? n2 - k : 0) * ld + j], xa, xb);
            double2* dst = R.pme_spec + (size_t)(r0 + 2 * j) * M + k;
            dst[0] = xa;
            if (2 * j + 1 < nrow) dst[M] = xb;
        }
    }
}
__global__ void __launch_bounds__(kAxisThreads) k_pme_rows_c2r(const RepDev* __restrict__ reps, int nrep) {
    extern __shared__ __align__(16) double2 fbuf[];
    __shared__ int pre[257];
    __shared__ int wtot[32];
    items_prefix(nrep, pre, wtot, [&](int r) { return pme_stale(reps[r]) ? row_items(reps[r]) : 0; });
    for (int it = blockIdx.x; it < pre[nrep]; it += gridDim.x) {
        const int r = prefix_find(pre, nrep, it);
        const RepDev& R = reps[r];
        const int n2 = R.pme_n[2], M = n2 / 2 + 1, ld = kRowPairs | 1;
        const int r0 = (it - pre[r]) * 2 * kRowPairs, nrow = min(2 * kRowPairs, R.pme_n[0] * R.pme_n[1] - r0);
        const int np = (nrow + 1) >> 1;
        double2 *b0 = fbuf, *b1 = fbuf + ld * n2, *tw = b1 + ld * n2;
        __syncthreads();
        load_roots(R, 2, tw);
        const FastDiv by_n2(n2);
        for (int e = threadIdx.x; e < np * n2; e += blockDim.x) {
            const int j = by_n2.quot(e), k = e - j * n2;
            const bool mir = k >= M;
            const double2* src = R.pme_spec + (size_t)(r0 + 2 * j) * M + (mir ? n2 - k : k);
            b0[k * ld + j] = join_pair(src[0], 2 * j + 1 < nrow ? src[M] : make_double2(0.0, 0.0), mir);
        }
        const double2* out = fft_lines_block(b0, b1, ld, np, n2, tw, 1);
        double* phi = const_cast<double*>(R.pme_phi) + (size_t)r0 * n2;
        for (int e = threadIdx.x; e < np * n2; e += blockDim.x) {
            const int j = by_n2.quot(e), i = e - j * n2;
            const double2 v = out[i * ld + j];
            phi[(size_t)(2 * j) * n2 + i] = v.x;
            if (2 * j + 1 < nrow) phi[(size_t)(2 * j + 1) * n2 + i] = v.y;
        }
    }
    pme_finish(reps, nrep);
}

__device__ __forceinline__ double sel4(const double m[4], int j) {
    return j & 2 ? (j & 1 ? m[3] : m[2]) : (j & 1 ? m[1] : m[0]);
}

// Mesh index of the spline's point j at mesh coordinate floor f (any period).
__device__ __forceinline__ int mesh_index(double f, int j, int n) {
    int k = (int)f;
    if ((unsigned)k >= (unsigned)n) k = wrapm(k, n);
    k -= j;
    return k < 0 ? wrapm(k, n) : k;
}

// Charge q at (x, y, z) spread onto Q by a whole warp: lane l adds the points
// (l / 8, (l / 2) % 4, 2 (l % 2) + {0, 1}); lane 4 a + j forms axis a's weight and
// index j, which the others fetch (with every lane forming all twelve weights the
// single SM's FP64 rate bounded it, 3.8 us a site).  One site per warp instead of
// one per lane: a lane's 64 adds in a row took 10 to 20 us of the accept kernel
// (3-site water, 64^3 mesh; 70 to 120 us in the slab's steps of 30 to 70 accepted
// moves).
__device__ __forceinline__ void pme_spread_warp(const RepDev& R, double* Q, float x, float y, float z, double q,
                                                int lane) {
    const int ax = (lane >> 2) % 3;
    const double u = mesh_u(R, ax == 0 ? x : (ax == 1 ? y : z), ax), f = floor(u);
    double m[4];
    bspline4(u - f, m);
    const double w = sel4(m, lane & 3);
    const int k = mesh_index(f, lane & 3, R.pme_n[ax]);
    const int a = lane >> 3, b = 4 + ((lane >> 1) & 3), c = 8 + (lane & 1) * 2;
    const double wab = q * __shfl_sync(kFull, w, a) * __shfl_sync(kFull, w, b);
    const double w0 = __shfl_sync(kFull, w, c), w1 = __shfl_sync(kFull, w, c + 1);
    const int ka = __shfl_sync(kFull, k, a), kb = __shfl_sync(kFull, k, b);
    const int k0 = __shfl_sync(kFull, k, c), k1 = __shfl_sync(kFull, k, c + 1);
    double* row = Q + ((size_t)ka * R.pme_n[1] + kb) * R.pme_n[2];
    atomicAdd(row + k0, wab * w0);
    atomicAdd(row + k1, wab * w1);
}

// phi at caller points (diagnostics)
__global__ void k_pme_phi_points(const RepDev* __restrict__ rep, const double* __restrict__ pts, int n,
                                 double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = pme_phi_at(*rep, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
}

__device__ __forceinline__ float ewald_g(float r, float alpha) {
    return r < 1e-6f ? 2.0f * alpha * 0.564189584f : erff(alpha * r) / r;
}

// Lanes that share one site's 16 mesh rows (of 4 points) when ns sites are
// interpolated by a warp: the largest power of two with ns lanes' groups in 32.
__device__ __forceinline__ int mesh_lanes(int ns) {
    return ns <= 2 ? 16 : (ns <= 4 ? 8 : (ns <= 8 ? 4 : (ns <= 16 ? 2 : 1)));
}

// Reciprocal-space and molecular terms of a pose, whole warp; the sum over the
// lanes of the results is
//   sum_s q_s phi(r_s) - K q_s sum_t q_t g(|r_s - x_t|)
// (the latter when the pose replaces group `self`).  Site s at sites[s]
// (absolute position, charge) in shared memory.  phi is interpolated by
// mesh_lanes lanes per site, each taking its share of the 16 mesh rows: with one
// lane per site a 3-site pose kept 3 lanes busy with 64 loads each.
__device__ __forceinline__ double pme_pose_warp(const RepDev& R, int ns, int lane, const float4* sites, int self) {
    const int P = mesh_lanes(ns), s = lane / P, sub = lane - s * P;
    double e = 0.0;
    if (s < ns) {
        const float4 p = sites[s];
        const double ux = mesh_u(R, p.x, 0), uy = mesh_u(R, p.y, 1), uz = mesh_u(R, p.z, 2);
        const double fx = floor(ux), fy = floor(uy), fz = floor(uz);
        double mx[4], my[4], mz[4];
        bspline4(ux - fx, mx);
        bspline4(uy - fy, my);
        bspline4(uz - fz, mz);
        const int n1 = R.pme_n[1], n2 = R.pme_n[2];
        const int z0 = mesh_index(fz, 0, n2), z1 = mesh_index(fz, 1, n2), z2 = mesh_index(fz, 2, n2),
                  z3 = mesh_index(fz, 3, n2);
        for (int r = sub; r < 16; r += P) {
            const int a = r >> 2, b = r & 3;
            const double* row = R.pme_phi + ((size_t)mesh_index(fx, a, R.pme_n[0]) * n1 + mesh_index(fy, b, n1)) * n2;
            const double t = mz[0] * row[z0] + mz[1] * row[z1] + mz[2] * row[z2] + mz[3] * row[z3];
            e += sel4(mx, a) * sel4(my, b) * t;
        }
        e *= (double)p.w;
    }
    if (self >= 0 && lane < ns) {
        const float4 p = sites[lane];
        const int2 sp = R.gspan[self];
        float m = 0.0f;
        for (int t = 0; t < sp.y; ++t) {
            const float4 a = R.xyzq[sp.x + t];
            float dx = p.x - a.x, dy = p.y - a.y, dz = p.z - a.z;
            dx -= rintf(dx * R.invL[0]) * R.L[0];
            dy -= rintf(dy * R.invL[1]) * R.L[1];
            dz -= rintf(dz * R.invL[2]) * R.L[2];
            m += a.w * ewald_g(sqrtf(dx * dx + dy * dy + dz * dz), R.pme_alpha);
        }
        e -= (double)kCoulomb * (double)p.w * (double)m;
    }
    return e;
}

// Gradient of pme_pose_warp's terms with respect to lane `lane`'s site position
// (lanes < ns; zero otherwise), whole warp: q grad phi(r_s) from the derivative of
// the B-spline interpolation (d/dx = (n / L) d/du), the mesh rows shared out as
// there, minus K q sum_t q_t g'(d) d/|d| over the replaced group's atoms
// (d = r_s - x_t, minimum image).
__device__ __forceinline__ void pme_grad_warp(const RepDev& R, int ns, int lane, const float4* sites, int self,
                                              float& gx, float& gy, float& gz) {
    const int P = mesh_lanes(ns), ms = lane / P, sub = lane - ms * P;
    double px = 0.0, py = 0.0, pz = 0.0;
    if (ms < ns) {
        const float4 p = sites[ms];
        const double ux = mesh_u(R, p.x, 0), uy = mesh_u(R, p.y, 1), uz = mesh_u(R, p.z, 2);
        const double fx = floor(ux), fy = floor(uy), fz = floor(uz);
        double mx[4], my[4], mz[4], dx[4], dy[4], dz[4];
        bspline4(ux - fx, mx);
        bspline4(uy - fy, my);
        bspline4(uz - fz, mz);
        bspline4_d(ux - fx, dx);
        bspline4_d(uy - fy, dy);
        bspline4_d(uz - fz, dz);
        const int n1 = R.pme_n[1], n2 = R.pme_n[2];
        const int z0 = mesh_index(fz, 0, n2), z1 = mesh_index(fz, 1, n2), z2 = mesh_index(fz, 2, n2),
                  z3 = mesh_index(fz, 3, n2);
        for (int r = sub; r < 16; r += P) {
            const int a = r >> 2, b = r & 3;
            const double* row = R.pme_phi + ((size_t)mesh_index(fx, a, R.pme_n[0]) * n1 + mesh_index(fy, b, n1)) * n2;
            const double v0 = row[z0], v1 = row[z1], v2 = row[z2], v3 = row[z3];
            const double t = mz[0] * v0 + mz[1] * v1 + mz[2] * v2 + mz[3] * v3;
            const double tz = dz[0] * v0 + dz[1] * v1 + dz[2] * v2 + dz[3] * v3;
            const double wx = sel4(mx, a), wy = sel4(my, b);
            px += sel4(dx, a) * wy * t;
            py += wx * sel4(dy, b) * t;
            pz += wx * wy * tz;
        }
    }
    for (int off = P >> 1; off > 0; off >>= 1) {
        px += __shfl_xor_sync(kFull, px, off);
        py += __shfl_xor_sync(kFull, py, off);
        pz += __shfl_xor_sync(kFull, pz, off);
    }
    const int from = min(lane * P, 31);  // lane s: the sum of the lanes of site s
    px = __shfl_sync(kFull, px, from);
    py = __shfl_sync(kFull, py, from);
    pz = __shfl_sync(kFull, pz, from);
    gx = gy = gz = 0.0f;
    if (lane >= ns || sites[lane].w == 0.0f) return;
    const float sx = sites[lane].x, sy = sites[lane].y, sz = sites[lane].z, q = sites[lane].w;
    double g0 = (double)q * px * R.pme_n[0] / (double)R.L[0];
    double g1 = (double)q * py * R.pme_n[1] / (double)R.L[1];
    double g2 = (double)q * pz * R.pme_n[2] / (double)R.L[2];
    if (self >= 0) {  // d/dr_s of -K q sum_t q_t g(|r_s - x_t|), g(r) = erf(alpha r) / r
        const int2 sp = R.gspan[self];
        const double al = (double)R.pme_alpha, c = 1.1283791670955126 * al;  // 2 alpha / sqrt(pi)
        for (int t = 0; t < sp.y; ++t) {
            const float4 at = R.xyzq[sp.x + t];
            double ex = (double)sx - at.x, ey = (double)sy - at.y, ez = (double)sz - at.z;
            ex -= rint(ex / (double)R.L[0]) * (double)R.L[0];
            ey -= rint(ey / (double)R.L[1]) * (double)R.L[1];
            ez -= rint(ez / (double)R.L[2]) * (double)R.L[2];
            const double r = sqrt(ex * ex + ey * ey + ez * ez);
            // g'(r) / r (a smooth even function: -(4/3) alpha^3 / sqrt(pi) at r = 0)
            const double gp = r < 1e-4 ? -(2.0 / 3.0) * c * al * al
                                       : (c * exp(-al * al * r * r) * r - erf(al * r)) / (r * r * r);
            const double w = -(double)kCoulomb * q * at.w * gp;
            g0 += w * ex;
            g1 += w * ey;
            g2 += w * ez;
        }
    }
    gx = (float)g0;
    gy = (float)g1;
    gz = (float)g2;
}

}  // namespace gcmc
