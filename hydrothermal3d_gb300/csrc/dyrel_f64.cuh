// The FP64 pseudo-iteration of k_dyrel_iter with every face flux evaluated once
// and the quotient by the diagonal from its reciprocal (include from
// -fmad=false translation units: the same values as the reference's statements).
//
// Bound by the FP64 pipe, 2 results per clock and SM: at 63^3 the fields sit in
// L2 and at 255^3 an iteration moves 0.17 of the copy rate, so only the number
// of FP64 instructions and an even load of the SMs count.  A thread has two
// neighbouring cells of a row; a block has a run of such pairs of a plane, row
// after row without gaps, and marches through a chunk of planes.  A thread
// evaluates its cells' west and south fluxes and leaves them in shared memory
// for the pair to the west and the row to the south; the z flux stays in a
// register.  What is left are 9 operations for the fluxes (15 in k_dyrel_iter),
// 9 or 11 for their sum, 3 for the quotient (9) and 5 for the update, and one
// more face at the block's end, at a wall and at a chunk's first plane.
//
// us per iteration, k_dyrel_iter and this kernel: 31 x 29 x 33 8.5 -> 6.5, 63^3
// 31.0 -> 22.9, 95^3 82 -> 62, 127 x 119 x 131 180 -> 133, 255^3 1440 -> 1006.
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

// CX: cX != 0 (adding 0 * x changes no value).  INV: iPC holds 1 / PC.
template <int MODE, bool CX, bool INV, int T>
__global__ void __launch_bounds__(T) k_dyrel_f64(const double* __restrict__ Xin, double* __restrict__ Xout,
                                                const double* __restrict__ R, const double* __restrict__ kx,
                                                const double* __restrict__ ky, const double* __restrict__ kz,
                                                const double* __restrict__ PC, const double* __restrict__ iPC,
                                                double* __restrict__ F0, double* __restrict__ F, DyrelScalT<double> s,
                                                BC6<double> bc, int nx, int ny, int nz, int zchunk,
                                                double* __restrict__ partials) {
    // west flux of the first cell and south fluxes, two planes deep: one barrier per plane
    __shared__ double west[2][T];
    __shared__ double2 south[2][T];
    const int np = (nx + 1) / 2, tid = threadIdx.x;
    const int t = blockIdx.x * T + tid;
    const int j = t / np, i = 2 * (t - j * np);
    const bool row = j < ny, in1 = i + 1 < nx;
    const int k0 = blockIdx.z * zchunk, k1 = min(nz, k0 + zchunk);
    const double h1 = s.h1, h2 = s.h2, dtau = s.dtau, _dx = s._dx, _dy = s._dy, _dz = s._dz;
    const bool east_here = i + 2 == nx || (tid == T - 1 && i + 2 < nx);  // east face of cell 1: no thread's west face
    const bool north_here = j == ny - 1 || tid + np >= T;
    const int n1 = nx + 2, pl = n1 * (ny + 2), cpl = nx * ny;
    const int jc = min(j, ny - 1);  // threads past the plane read its last row and store nothing
    int e = (i + 1) + n1 * (jc + 1) + pl * (k0 + 1);
    int c = i + nx * jc + cpl * k0;
    int fx = i + (nx + 1) * (jc + ny * k0), fy = i + nx * (jc + (ny + 1) * k0);
    const int d1 = in1 ? 1 : 0;  // cell 1 from cell 0
    double c0 = Xin[e], c1 = Xin[e + d1];
    double xb0 = Xin[e - pl], xb1 = Xin[e - pl + d1];
    if (k0 == 0) {
        xb0 = ghost_f64(bc, 4, c0);
        xb1 = ghost_f64(bc, 4, c1);
    }
    double qB0 = -kz[c] * (_dz * (c0 - xb0)), qB1 = -kz[c + d1] * (_dz * (c1 - xb1));
    for (int k = k0; k < k1; ++k) {
        // the plane's loads first: they are in flight while the fluxes wait for the FP64 pipe
        double f0x = Xin[e + pl], f1x = Xin[e + pl + d1], xs0 = Xin[e - n1], xs1 = Xin[e - n1 + d1], xw = Xin[e - 1];
        const double kW0 = kx[fx], kW1 = kx[fx + 1], kS0 = ky[fy], kS1 = ky[fy + d1], kF0 = kz[c + cpl],
                     kF1 = kz[c + cpl + d1], p0 = PC[c], p1 = PC[c + d1], m0 = F0[c], m1 = F0[c + d1];
        double fu0 = R[c], fu1 = R[c + d1], y0 = 0.0, y1 = 0.0;
        if (INV) {
            y0 = iPC[c];
            y1 = iPC[c + d1];
        }
        if (k == nz - 1) {
            f0x = ghost_f64(bc, 5, c0);
            f1x = ghost_f64(bc, 5, c1);
        }
        if (j == 0) {
            xs0 = ghost_f64(bc, 2, c0);
            xs1 = ghost_f64(bc, 2, c1);
        }
        if (i == 0) xw = ghost_f64(bc, 0, c0);
        double a1 = c1, xe = 0.0;
        if (!in1) a1 = xe = ghost_f64(bc, 1, c0);  // cell 0 is the row's last: its east wall as cell 1's west face
        const double qW0 = -kW0 * (_dx * (c0 - xw)), qW1 = -kW1 * (_dx * (a1 - c0));
        const double qS0 = -kS0 * (_dy * (c0 - xs0)), qS1 = -kS1 * (_dy * (c1 - xs1));
        west[k & 1][tid] = qW0;
        south[k & 1][tid] = make_double2(qS0, qS1);
        const double z0 = -kF0 * (_dz * (f0x - c0)), z1 = -kF1 * (_dz * (f1x - c1));
        __syncthreads();
        double qE1 = 0.0, qN0, qN1, xn0 = 0.0, xn1 = 0.0;
        if (east_here) {
            xe = i + 2 == nx ? ghost_f64(bc, 1, c1) : Xin[e + 2];
            qE1 = -kx[fx + 2] * (_dx * (xe - c1));
        } else if (tid + 1 < T) {
            qE1 = west[k & 1][tid + 1];
        }
        if (north_here) {
            xn0 = j >= ny - 1 ? ghost_f64(bc, 3, c0) : Xin[e + n1];
            xn1 = j >= ny - 1 ? ghost_f64(bc, 3, c1) : Xin[e + n1 + d1];
            qN0 = -ky[fy + nx] * (_dy * (xn0 - c0));
            qN1 = -ky[fy + nx + d1] * (_dy * (xn1 - c1));
        } else {
            const double2 n = south[k & 1][tid + np];
            qN0 = n.x;
            qN1 = n.y;
        }
        if (CX) {
            fu0 = fu0 + s.cX * c0;
            fu1 = fu1 + s.cX * c1;
        }
        fu0 = fu0 + _dx * (qW1 - qW0) + _dy * (qN0 - qS0) + _dz * (z0 - qB0);
        fu1 = fu1 + _dx * (qE1 - qW1) + _dy * (qN1 - qS1) + _dz * (z1 - qB1);
        const double f0 = INV ? div_known(fu0, p0, y0) : div_any(fu0, p0);
        const double f1 = INV ? div_known(fu1, p1, y1) : div_any(fu1, p1);
        const double g0 = h1 * m0 + h2 * f0, g1 = h1 * m1 + h2 * f1;
        const double r0 = dtau * g0, r1 = dtau * g1;
        const double o0 = c0 - r0, o1 = c1 - r1;
        if (row) {
            F0[c] = g0;
            Xout[e] = o0;
            if (in1) {
                F0[c + 1] = g1;
                Xout[e + 1] = o1;
            }
            if (MODE == MODE_CHECK) {  // per-cell terms of the check sums (canonical tree order)
                const long long n = (long long)cpl * nz;
                partials[c] = fabs(f0 * p0);
                partials[c + n] = -r0 * (f0 - F[c]);
                partials[c + 2 * n] = r0 * r0;
                if (in1) {
                    partials[c + 1] = fabs(f1 * p1);
                    partials[c + 1 + n] = -r1 * (f1 - F[c + 1]);
                    partials[c + 1 + 2 * n] = r1 * r1;
                }
            }
            if (MODE >= MODE_STOREF) {
                F[c] = f0;
                if (in1) F[c + 1] = f1;
            }
            // face ghosts of the output = BC of the input (reference state)
            if (i == 0) Xout[e - 1] = xw;
            if (!in1) Xout[e + 1] = xe;
            if (i + 2 == nx) Xout[e + 2] = xe;
            if (j == 0) {
                Xout[e - n1] = xs0;
                if (in1) Xout[e - n1 + 1] = xs1;
            }
            if (j == ny - 1) {
                Xout[e + n1] = xn0;
                if (in1) Xout[e + n1 + 1] = xn1;
            }
            if (k == 0) {
                Xout[e - pl] = xb0;
                if (in1) Xout[e - pl + 1] = xb1;
            }
            if (k == nz - 1) {
                Xout[e + pl] = f0x;
                if (in1) Xout[e + pl + 1] = f1x;
            }
        }
        c0 = f0x;
        c1 = f1x;
        qB0 = z0;
        qB1 = z1;
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
    int threads, zchunk;
    dim3 grid;
};
// Chunks of planes so that the SMs carry about the same number of planes (a
// block's time is its planes' plus a tenth for the first one's extra flux).  256
// threads keep two warps per scheduler busy with one block per SM; small grids
// spread over more schedulers with 128.
inline F64Launch f64_launch(int sms, int nx, int ny, int nz) {
    F64Launch L;
    const long long pairs = (long long)((nx + 1) / 2) * ny;
    L.threads = pairs * nz >= 256LL * sms ? 256 : 128;
    const long long gx = (pairs + L.threads - 1) / L.threads;
    long long best = -1;
    for (int c = 1; c <= std::min(nz, 64); ++c) {
        const long long blocks = gx * ((nz + c - 1) / c);
        // blocks in a row on an SM, in halves; where there are many, the last wave is half full
        const long long deep = blocks >= 4LL * sms ? 2 * blocks / sms + 1 : 2 * ((blocks + sms - 1) / sms);
        const long long cost = deep * (10LL * c + 1);
        if (best < 0 || cost < best) best = cost, L.zchunk = c;
    }
    L.grid = dim3((unsigned)gx, 1, (nz + L.zchunk - 1) / L.zchunk);
    return L;
}

template <int MODE>
struct F64Kernel {
    typedef void (*Fn)(const double*, double*, const double*, const double*, const double*, const double*, const double*,
                       const double*, double*, double*, DyrelScalT<double>, BC6<double>, int, int, int, int, double*);
    template <bool CX, bool INV>
    static Fn by_size(int threads) {
        return threads == 256 ? (Fn)k_dyrel_f64<MODE, CX, INV, 256> : (Fn)k_dyrel_f64<MODE, CX, INV, 128>;
    }
    static Fn get(bool cx, bool inv, int threads) {
        return cx ? (inv ? by_size<true, true>(threads) : by_size<true, false>(threads))
                  : (inv ? by_size<false, true>(threads) : by_size<false, false>(threads));
    }
};

}  // namespace
