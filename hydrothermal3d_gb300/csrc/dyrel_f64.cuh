// The FP64 pseudo-iteration of k_dyrel_iter with every face flux evaluated once
// and the quotient by the diagonal from its reciprocal (include from
// -fmad=false translation units).  With the reciprocals at hand the values are
// those of the reference's statements, without them up to div_any's (fp64_div.cuh).
//
// Bound by the FP64 pipe, 2 results per clock and SM: at 63^3 the fields sit in
// L2 and at 255^3 an iteration moves 0.17 of the copy rate, so only the number
// of FP64 instructions and an even load of the SMs count.  A thread has two
// neighbouring cells of a row; a block has a run of such pairs of a plane, row
// after row without gaps, and marches through a chunk of planes.  A thread
// evaluates its cells' west and south fluxes and leaves them in shared memory
// for the pair to the west and the row to the south; the z flux stays in a
// register.  (Small grids: one cell per thread.)  What is left are 9 operations for
// the fluxes (15 in k_dyrel_iter), 9 or 11 for their sum, 3 for the quotient (9)
// and 5 for the update, and one more face at the block's end, at a wall and at a
// chunk's first plane.
//
// us per iteration, k_dyrel_iter and this kernel: 31 x 29 x 33 8.5 -> 4.7, 63^3
// 31.0 -> 18.8, 95^3 82 -> 58.2, 127 x 119 x 131 180 -> 130, 255^3 1440 -> 1009.
// Plain launches begin on a 2 us raster; launch_after saves the wait (63^3: 22.9).
#pragma once
#include "dyrel_common.cuh"
#include "fp64_div.cuh"

namespace {

// ghost value; the subtraction is not issued for a Neumann face
__device__ __forceinline__ double ghost_f64(const BC6<double>& bc, int f, double inner) {
    double v = inner;
    if (bc.dir[f]) v = bc.val2[f] - inner;
    return v;
}

// CX: cX != 0 (adding 0 * x changes no value).  INV: iPC holds 1 / PC.  NC: cells
// per thread, neighbours in x.
template <int MODE, bool CX, bool INV, int T, int NC>
__global__ void __launch_bounds__(T) k_dyrel_f64(const double* __restrict__ Xin, double* __restrict__ Xout,
                                                const double* __restrict__ R, const double* __restrict__ kx,
                                                const double* __restrict__ ky, const double* __restrict__ kz,
                                                const double* __restrict__ PC, const double* __restrict__ iPC,
                                                double* __restrict__ F0, double* __restrict__ F, DyrelScalT<double> s,
                                                BC6<double> bc, int nx, int ny, int nz, int zchunk,
                                                double* __restrict__ partials) {
    // west flux of the first cell and south fluxes, two planes deep: one barrier per plane
    __shared__ double west[2][T], south[2][NC][T];
    after_previous();
    const int np = (nx + NC - 1) / NC, tid = threadIdx.x;
    const int t = blockIdx.x * T + tid;
    // a warp past the plane: on thin grids most of them (with two cells per thread
    // the plane is wide, and the test cost 2 % at 200 x 190 x 200)
    if (NC == 1 && t - (tid & 31) >= np * ny) return;
    const int j = t / np, i = NC * (t - j * np);
    const bool row = j < ny;
    const int k0 = blockIdx.z * zchunk, k1 = min(nz, k0 + zchunk);
    const double h1 = s.h1, h2 = s.h2, dtau = s.dtau, _dx = s._dx, _dy = s._dy, _dz = s._dz;
    const int nc = min(NC, nx - i);                                          // cells of this thread
    const bool wall = i + NC == nx;                                          // its last face is the wall
    const bool east_here = wall || (tid == T - 1 && i + NC < nx);            // that face is no thread's west face
    const bool north_here = j >= ny - 1 || tid + np >= T;
    const int n1 = nx + 2, pl = n1 * (ny + 2), cpl = nx * ny;
    const int jc = min(j, ny - 1);  // threads past the plane read its last row and store nothing
    int e = (i + 1) + n1 * (jc + 1) + pl * (k0 + 1);
    int c = i + nx * jc + cpl * k0;
    int fx = i + (nx + 1) * (jc + ny * k0), fy = i + nx * (jc + (ny + 1) * k0);
    auto off = [&](int m) { return m < nc ? m : 0; };  // a missing cell reads the first one's values
    double xc[NC], xb[NC], qB[NC];
#pragma unroll
    for (int m = 0; m < NC; ++m) {
        xc[m] = Xin[e + off(m)];
        xb[m] = k0 == 0 ? ghost_f64(bc, 4, xc[m]) : Xin[e - pl + off(m)];
        qB[m] = -kz[c + off(m)] * (_dz * (xc[m] - xb[m]));
    }
    for (int k = k0; k < k1; ++k) {
        const int par = k & 1;
        // the plane's loads first: they are in flight while the fluxes wait for the FP64 pipe
        double xf[NC], xs[NC], kW[NC], kS[NC], kF[NC], pc[NC], ip[NC], mo[NC], fu[NC];
        double xw = Xin[e - 1];
#pragma unroll
        for (int m = 0; m < NC; ++m) {
            xf[m] = Xin[e + pl + off(m)];
            xs[m] = Xin[e - n1 + off(m)];
            kW[m] = kx[fx + (i + m <= nx ? m : 0)];
            kS[m] = ky[fy + off(m)];
            kF[m] = kz[c + cpl + off(m)];
            pc[m] = PC[c + off(m)];
            ip[m] = INV ? iPC[c + off(m)] : 0.0;
            mo[m] = F0[c + off(m)];
            fu[m] = R[c + off(m)];
        }
        if (k == nz - 1)
#pragma unroll
            for (int m = 0; m < NC; ++m) xf[m] = ghost_f64(bc, 5, xc[m]);
        if (j == 0)
#pragma unroll
            for (int m = 0; m < NC; ++m) xs[m] = ghost_f64(bc, 2, xc[m]);
        if (i == 0) xw = ghost_f64(bc, 0, xc[0]);
        // a cell after the row's last one stands for the wall's ghost, so the wall's flux is its west flux
        double a[NC + 1], xe = 0.0;
        a[0] = xw;
#pragma unroll
        for (int m = 0; m < NC; ++m) {
            a[m + 1] = xc[m];
            if (m > 0 && i + m == nx) a[m + 1] = xe = ghost_f64(bc, 1, xc[m - 1]);
        }
        double qx[NC + 1], qS[NC], qN[NC], qF[NC];
#pragma unroll
        for (int m = 0; m < NC; ++m) {
            qx[m] = -kW[m] * (_dx * (a[m + 1] - a[m]));
            qS[m] = -kS[m] * (_dy * (xc[m] - xs[m]));
            south[par][m][tid] = qS[m];
        }
        west[par][tid] = qx[0];
#pragma unroll
        for (int m = 0; m < NC; ++m) qF[m] = -kF[m] * (_dz * (xf[m] - xc[m]));
        __syncthreads();
        qx[NC] = 0.0;
        if (east_here) {
            xe = wall ? ghost_f64(bc, 1, xc[NC - 1]) : Xin[e + NC];
            qx[NC] = -kx[fx + NC] * (_dx * (xe - xc[NC - 1]));
        } else if (tid + 1 < T) {
            qx[NC] = west[par][tid + 1];
        }
        double xn[NC];
        if (north_here) {
#pragma unroll
            for (int m = 0; m < NC; ++m) {
                xn[m] = j >= ny - 1 ? ghost_f64(bc, 3, xc[m]) : Xin[e + n1 + off(m)];
                qN[m] = -ky[fy + nx + off(m)] * (_dy * (xn[m] - xc[m]));
            }
        } else {
#pragma unroll
            for (int m = 0; m < NC; ++m) qN[m] = south[par][m][tid + np];
        }
#pragma unroll
        for (int m = 0; m < NC; ++m) {
            if (CX) fu[m] = fu[m] + s.cX * xc[m];
            fu[m] = fu[m] + _dx * (qx[m + 1] - qx[m]) + _dy * (qN[m] - qS[m]) + _dz * (qF[m] - qB[m]);
            const double f = INV ? div_known(fu[m], pc[m], ip[m]) : div_any(fu[m], pc[m]);
            const double f0 = h1 * mo[m] + h2 * f;
            const double d = dtau * f0;
            const double o = xc[m] - d;
            if (!row || m >= nc) continue;
            F0[c + m] = f0;
            Xout[e + m] = o;
            if (MODE == MODE_CHECK) {  // per-cell terms of the check sums (canonical tree order)
                const long long n = (long long)cpl * nz;
                partials[c + m] = fabs(f * pc[m]);
                partials[c + m + n] = -d * (f - F[c + m]);
                partials[c + m + 2 * n] = d * d;
            }
            if (MODE >= MODE_STOREF) F[c + m] = f;
            // face ghosts of the output = BC of the input (reference state)
            if (i + m == 0) Xout[e - 1] = xw;
            if (i + m == nx - 1) Xout[e + m + 1] = xe;
            if (j == 0) Xout[e + m - n1] = xs[m];
            if (j == ny - 1) Xout[e + m + n1] = xn[m];
            if (k == 0) Xout[e + m - pl] = xb[m];
            if (k == nz - 1) Xout[e + m + pl] = xf[m];
        }
#pragma unroll
        for (int m = 0; m < NC; ++m) {
            xc[m] = xf[m];
            qB[m] = qF[m];
        }
        e += pl;
        c += cpl;
        fx += (nx + 1) * ny;
        fy += nx * (ny + 1);
    }
}

// 1 / PC of every cell
__global__ void k_reciprocal(double* __restrict__ iPC, const double* __restrict__ PC, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        iPC[t] = 1.0 / PC[t];
}

struct F64Launch {
    int cells, threads, zchunk;  // cells per thread, threads per block, planes per block
    dim3 grid;
    long long blocks() const { return (long long)grid.x * grid.z; }
};
// (a grid has at most 65535 blocks in z: longer columns take more planes a block)
inline F64Launch f64_shape(int cells, int threads, int zchunk, int nx, int ny, int nz) {
    zchunk = std::max(zchunk, (nz + 65534) / 65535);
    const long long runs = (long long)((nx + cells - 1) / cells) * ny;
    return F64Launch{cells, threads, zchunk,
                     dim3((unsigned)((runs + threads - 1) / threads), 1, (unsigned)((nz + zchunk - 1) / zchunk))};
}
// Below 2^19 cells the shape whose busiest SM is done first: an SM's share of the
// cell slots, times what a slot takes where the SM's blocks run together, and 1.2 us
// a plane of a block.  One cell per thread in blocks of 128 for the smallest grids
// (31 x 29 x 33: 4.6 us) and of 256 (72 x 70 x 75: 28.6, 29.9 with 128); two cells
// in blocks of 64 and two planes while an SM holds its share of them at once (56^3:
// 14.7, 15.3 with one cell; 63^3: 18.8, 20.4), and in blocks of 256 and two or three
// planes while an SM holds its two at once (80 x 70 x 75: 31.0, 32.6 with one cell;
// but 80^3, a second round of them: 42.1, 39.0).  From 2^19 cells on the rounds blend:
// three planes up to 2^22 (95^3: 58.2, 63.0 with one cell; 127 x 119 x 131: 130, two
// planes 137), eight above (255^3: 1009, three 1037).  A plane of less than two
// blocks of pairs is left to the small shapes, where its empty warps leave: per
// iteration 1 x 1 x 4096 56 us with them and 17 without (k_dyrel_iter 29), 2 x 2 x
// 60000 589 and 167 (566).
inline F64Launch f64_launch(int sms, int nx, int ny, int nz) {
    const long long n = (long long)nx * ny * nz;
    const int plane = nx * ny, pairs = (nx + 1) / 2 * ny;
    if (n >= (1LL << 19) && pairs >= 512) return f64_shape(2, 256, n < (1LL << 22) ? 3 : 8, nx, ny, nz);
    struct Shape { int cells, threads, planes, most, ps; };  // most: blocks that an SM may have; ps a slot
    const Shape shapes[] = {{1, 128, 1, 1 << 30, 11200}, {1, 256, 1, 1 << 30, 10800}, {2, 64, 2, 9, 9500},
                            {2, 256, 2, 2, 8800}, {2, 256, 3, 2, 8800}};
    F64Launch best{};
    long long least = -1;
    for (const Shape& h : shapes) {
        const F64Launch L = f64_shape(h.cells, h.threads, h.planes, nx, ny, nz);
        const long long share = (L.blocks() + sms - 1) / sms;
        if (share > h.most || (h.cells == 1 && h.threads > 128 && plane <= 128)) continue;
        const int busy = h.cells == 1 ? std::min(h.threads, (plane + 31) / 32 * 32) : h.threads;
        const long long cost = share * h.cells * busy * h.planes * h.ps + 1200000LL * h.planes;
        if (least < 0 || cost < least) least = cost, best = L;
    }
    return best;
}

template <int MODE>
struct F64Kernel {
    typedef void (*Fn)(const double*, double*, const double*, const double*, const double*, const double*, const double*,
                       const double*, double*, double*, DyrelScalT<double>, BC6<double>, int, int, int, int, double*);
    template <bool CX, bool INV>
    static Fn by_shape(const F64Launch& L) {
        if (L.cells == 1)
            return L.threads == 128 ? (Fn)k_dyrel_f64<MODE, CX, INV, 128, 1> : (Fn)k_dyrel_f64<MODE, CX, INV, 256, 1>;
        return L.threads == 64 ? (Fn)k_dyrel_f64<MODE, CX, INV, 64, 2> : (Fn)k_dyrel_f64<MODE, CX, INV, 256, 2>;
    }
    static Fn get(bool cx, bool inv, const F64Launch& L) {
        return cx ? (inv ? by_shape<true, true>(L) : by_shape<true, false>(L))
                  : (inv ? by_shape<false, true>(L) : by_shape<false, false>(L));
    }
};

}  // namespace
