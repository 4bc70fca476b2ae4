// FP32 inner iterations of the mixed solver with the whole problem kept on the
// chip (included by dyrel_mixed.cu, which defines the padded layout, the
// scalars and the cell arithmetic).
//
// One cooperative launch runs a whole run of inner iterations (up to the next
// FP64 check or refresh).  A CTA keeps a block of complete x rows, `by` of
// them in y and BZ planes in z: both correction buffers in shared memory, the
// coefficients in shared memory and registers.  A thread owns one quad column
// (4 cells in x, BZ planes), so all of a cell's coefficients stay with one
// thread from the first iteration to the last, and an iteration moves only
// the blocks' faces: D of a face quad goes to its neighbour block through
// global memory (the L2) as 64-bit words that hold a value and the number of
// the iteration it belongs to.  A reader polls the words themselves, so a
// hand-over takes one store and one load that meet in the L2, without flags,
// fences or a grid barrier (64-bit accesses are single, so value and number
// cannot come apart).
//
// Two buffers of face words are enough: a block writes iteration n + 1's faces
// (over those of n - 1) after a CTA barrier behind which it held every
// neighbour's faces of n, and a neighbour's thread publishes its face quad of
// n after it has read the same face's quad of n - 1.
//
// Why: one launch per iteration costs about 4 us whatever the grid, and below
// 10^6 cells that is most of the iteration; above, each iteration reads 28
// bytes per cell from L2 or HBM, 24 of which never change.  What bounds it now:
// the hand-over (a face word takes about 0.45 us from L2, 0.9 with all of a
// CTA's faces in flight: 64 bytes per clock and SM) for low columns; for high
// ones half that and half the latency of the columns' own arithmetic at 12 to
// 16 warps per SM.  Measured, us per iteration, before (k_mixed_inner) and now:
// 33 x 29 x 31 4.0 -> 1.1, 63^3 4.1 -> 1.25, 79^3 6.1 -> 1.7, 95^3 6.2 -> 3.4,
// 100 x 110 x 120 8.2 -> 3.7, 127 x 119 x 131 9.7 -> 4.8.
//
// The cell arithmetic is mixed_cell's, operation for operation, two cells per
// instruction where the operands are neighbours in a quad (f32x2: each half
// rounds like the scalar operation).  The ghost rules are folded into the
// coefficients of the wall faces: D has homogeneous conditions, so a Neumann
// wall's flux is k (v - v) = 0 and its face gets k' = 0; a Dirichlet wall's is
// k (v - (-v)) = k (2 v) = (2 k) (v - 0), the same rounding, so its face gets
// k' = 2 k against a neighbour of 0.  The diagonals use the true k.  Cells
// outside the grid have 1 / diag = 0 and stay 0.  Results are equal to
// k_mixed_inner's, value for value.
#pragma once

typedef unsigned long long u64;
struct __align__(16) P4 {  // four floats as two packed pairs
    u64 a, b;
};
__device__ __forceinline__ u64 pk(float lo, float hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpk(u64 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 x, u64 y) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 x, u64 y) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 x, u64 y, u64 z) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ P4 sub4(const P4& x, const P4& y) { return P4{sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ P4 mul4(const P4& x, const P4& y) { return P4{mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ P4 fma4(const P4& x, const P4& y, const P4& z) {
    return P4{fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)};
}
__device__ __forceinline__ P4 fma4s(u64 s, const P4& y, const P4& z) {
    return P4{fma2(s, y.a, z.a), fma2(s, y.b, z.b)};
}
__device__ __forceinline__ P4 p4(const float (&v)[4]) { return P4{pk(v[0], v[1]), pk(v[2], v[3])}; }

constexpr int kResThreads = 512;               // at most (128 registers each)
constexpr size_t kResSmem = 226 * 1024;        // dynamic shared memory of a CTA
constexpr int kResThreads2 = 256;              // ... and of a CTA that shares its SM with another
constexpr size_t kResSmem2 = 112 * 1024;
constexpr unsigned kResWaitLimit = 1u << 20;   // polls of one face quad (about a second)
constexpr int kResMaxPerLaunch = 120;

// Where a thread keeps its column.  In shared memory a column's planes lie
// side by side at an odd pitch: every plane is an immediate offset from one
// address, and 16-byte accesses of neighbouring columns fall on all banks.
// Few planes fit the registers; from three planes on the x and y faces go to
// shared memory, with five the residual as well, and with seven planes (shared
// memory is full) the residual is read again from L2 in every iteration.
template <int BZ>
struct ResCfg {
    static constexpr int pitch = BZ | 1;
    static constexpr bool kShared = BZ >= 3;
    static constexpr bool rShared = BZ == 5;
    static constexpr bool rStream = BZ >= 6;
};
inline size_t res_smem(int bz, int nq, int by) {
    const size_t T = (size_t)nq * by, pitch = bz | 1;
    size_t cols = 2 * T + 2 * (size_t)nq;  // both corrections, the rows of the neighbour blocks
    if (bz >= 3) cols += T + T + nq;       // kx, ky
    if (bz == 5) cols += T;     // residual
    return (cols + 1) * pitch * 16;        // and one column of zeros before the first
}
// face words of one CTA, in quads per parity: S and N faces, B and F faces
__host__ __device__ inline int res_faces(int bz, int nq, int T) { return 2 * bz * nq + 2 * T; }

struct ResMember {
    const float *D, *Dp, *Rin, *kx, *ky, *kz;  // padded fields at the start of the run
    float *Dout, *Dpout;                       // ... and after it
    u64* xch;                                  // face words of the member's CTAs
    Pad P;
    MixScal s;
    int dir;  // bit f: face f is Dirichlet
    int nq, by, nby, T;
};
struct ResLaunch {
    int n, iters, prev0;
    unsigned tag;  // iteration it publishes tag + it + 1
    unsigned limit;
    int skip;      // test hook: CTA skip - 1 of each member does not publish its faces
    int* err;
    int block0[kResMaxPerLaunch + 1];
    ResMember rec[kResMaxPerLaunch];
};
static_assert(sizeof(ResLaunch) <= 32000, "launch parameters exceed the 32 KB kernel parameter space");

__device__ __forceinline__ void ld_words(const u64* p, u64& x, u64& y) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p));
}
__device__ __forceinline__ void st_words(u64* p, u64 x, u64 y) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y));
}
// shared memory by its 32-bit address
__device__ __forceinline__ P4 ld_sh(unsigned a) {
    P4 v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(a));
    return v;
}
__device__ __forceinline__ float ld_sh1(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_sh(unsigned a, const P4& v) {
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(v.a), "l"(v.b) : "memory");
}
// a face quad as loaded: words of cells 0, 1 at p and 2, 3 at p + half
struct FaceWords {
    u64 w[4];
};
__device__ __forceinline__ FaceWords face_ld(const u64* p, int half) {
    FaceWords f;
    ld_words(p, f.w[0], f.w[1]);
    ld_words(p + half, f.w[2], f.w[3]);
    return f;
}
__device__ __forceinline__ bool face_ready(const FaceWords& f, unsigned tag) {
    return (unsigned)(f.w[0] >> 32) == tag && (unsigned)(f.w[1] >> 32) == tag && (unsigned)(f.w[2] >> 32) == tag &&
           (unsigned)(f.w[3] >> 32) == tag;
}
__device__ __forceinline__ u64 low_halves(u64 x, u64 y) { return (x & 0xffffffffull) | (y << 32); }
// waits (bounded) until the quad is iteration `tag`'s; f: an earlier load of it
__device__ __forceinline__ bool face_wait(const u64* p, int half, unsigned tag, FaceWords f, const int* err,
                                          unsigned limit, P4& v) {
    for (unsigned c = 1; !face_ready(f, tag); ++c) {
        if (c > limit || ((c & 255u) == 0 && *(volatile const int*)err)) return false;
        f = face_ld(p, half);
    }
    v = P4{low_halves(f.w[0], f.w[1]), low_halves(f.w[2], f.w[3])};
    return true;
}
__device__ __forceinline__ void face_st(u64* p, int half, unsigned tag, const P4& v) {
    const u64 t = (u64)tag << 32;
    st_words(p, (v.a & 0xffffffffull) | t, (v.a >> 32) | t);
    st_words(p + half, (v.b & 0xffffffffull) | t, (v.b >> 32) | t);
}

template <int BZ>
__global__ void __launch_bounds__(kResThreads, 1) k_mixed_resident(const __grid_constant__ ResLaunch L) {
    using C = ResCfg<BZ>;
    constexpr bool KS = C::kShared, RM = C::rShared, RS = C::rStream;
    constexpr int PT = C::pitch;
    extern __shared__ __align__(16) unsigned char res_raw[];
    int lo = 0, hi = L.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((int)blockIdx.x >= L.block0[mid]) lo = mid;
        else hi = mid;
    }
    const ResMember& e = L.rec[lo];
    const Pad& P = e.P;
    const int cta = (int)blockIdx.x - L.block0[lo];
    const int zb = cta / e.nby, yb = cta - zb * e.nby;
    const int T = e.T, nq = e.nq;
    const int tid = min((int)threadIdx.x, T - 1);  // threads past the block repeat its last quad and store nothing
    const int jl = tid / nq, q = tid - jl * nq, i0 = 4 * q;
    const int j = yb * e.by + jl, z0 = zb * BZ;
    const int nk = min(BZ, P.nz - z0);  // planes inside the grid
    const bool own = (int)threadIdx.x < T, act = own && j < P.ny;
    const int pln = (int)P.plane, col = i0 + P.PX * min(j, P.ny - 1) + pln * z0;  // 32 bits: P.size < 2^31
    const float _dx2f = __fmul_rn(e.s._dx, e.s._dx), _dy2f = __fmul_rn(e.s._dy, e.s._dy),
                _dz2f = __fmul_rn(e.s._dz, e.s._dz);
    // 32-bit addresses of this thread's columns; a plane is 16 bytes
    const unsigned aD = (unsigned)__cvta_generic_to_shared(res_raw) + 16 * PT;  // [2][T] columns, behind one of zeros
    const unsigned bD = 16 * PT * T;                                            // bytes of one correction buffer
    const unsigned aY = aD + 2 * bD;  // [2][nq]: D of the rows before and after the block
    const unsigned me = 16 * PT * tid, row = 16 * PT * nq;
    const unsigned aKx = aY + 2 * row + me, aKy = aKx + bD, aR = aKy + bD + row;  // [T], [T + nq], [T]
    const P4 zero{0, 0};

    // ---- this thread's column
    P4 kz[BZ + 1], rd[BZ], R[RM || RS ? 1 : BZ], kx[KS ? 1 : BZ], kyS[KS ? 1 : BZ], kyN[KS ? 1 : BZ];
    float kE[KS ? 1 : BZ];
#pragma unroll
    for (int k = 0; k < BZ; ++k) {
        const int kg = z0 + k;
        const bool live = act && k < nk;
        const int b = col + pln * min(k, nk - 1);
        float w[5], s[4], n[4], bk[4], fr[4], r[4], dd[4], dp[4], rr[4];
        *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(e.kx + b);
        w[4] = i0 + 4 < P.PX ? e.kx[b + 4] : 0.f;
        *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(e.ky + b);
        *reinterpret_cast<float4*>(n) = *reinterpret_cast<const float4*>(e.ky + b + P.PX);
        *reinterpret_cast<float4*>(bk) = *reinterpret_cast<const float4*>(e.kz + b);
        *reinterpret_cast<float4*>(fr) = *reinterpret_cast<const float4*>(e.kz + b + pln);
        *reinterpret_cast<float4*>(r) = *reinterpret_cast<const float4*>(e.Rin + b);
        *reinterpret_cast<float4*>(dd) = *reinterpret_cast<const float4*>(e.D + b);
        *reinterpret_cast<float4*>(dp) = *reinterpret_cast<const float4*>(e.Dp + b);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const bool in = live && i0 + m < P.nx;
            rr[m] = in ? mixed_rdiag(w[m], w[m + 1], s[m], n[m], bk[m], fr[m], e.s.cX, _dx2f, _dy2f, _dz2f) : 0.f;
            if (!in) r[m] = dd[m] = dp[m] = 0.f;
            if (L.prev0) dp[m] = 0.f;
        }
        const float fW = (e.dir & 1) ? 2.f : 0.f, fE = (e.dir & 2) ? 2.f : 0.f, fS = (e.dir & 4) ? 2.f : 0.f,
                    fN = (e.dir & 8) ? 2.f : 0.f, fB = (e.dir & 16) ? 2.f : 0.f, fF = (e.dir & 32) ? 2.f : 0.f;
#pragma unroll
        for (int m = 0; m < 5; ++m) {
            if (i0 + m == 0) w[m] *= fW;
            if (i0 + m == P.nx) w[m] *= fE;
            if (!live) w[m] = 0.f;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (j == 0) s[m] *= fS;
            if (j == P.ny - 1) n[m] *= fN;
            if (kg == 0) bk[m] *= fB;
            if (kg == P.nz - 1) fr[m] *= fF;
            if (!live) s[m] = n[m] = bk[m] = fr[m] = 0.f;
        }
        if (k == 0) kz[0] = p4(bk);
        kz[k + 1] = p4(fr);
        rd[k] = p4(rr);
        const P4 kx4 = P4{pk(w[0], w[1]), pk(w[2], w[3])};
        if constexpr (!RM && !RS) R[k] = p4(r);
        if constexpr (RM) {
            if (own) st_sh(aR + 16 * k, p4(r));
        }
        if constexpr (KS) {
            if (own) {
                st_sh(aKx + 16 * k, kx4);
                // a row's north face is the next row's south face, but for the
                // block's last row and the grid's (row ny leaves its place to it)
                if (j != P.ny) st_sh(aKy + 16 * k, p4(s));
                if (jl == e.by - 1 || j == P.ny - 1) st_sh(aKy + row + 16 * k, p4(n));
            }
        } else {
            kx[k] = kx4;
            kE[k] = w[4];
            kyS[k] = p4(s);
            kyN[k] = p4(n);
        }
        if (own) {
            st_sh(aD + me + 16 * k, p4(dd));
            st_sh(aD + bD + me + 16 * k, p4(dp));
        }
    }
    // neighbours across the block's faces (other CTAs); none at the grid's
    // walls.  A block with a neighbour in y has two rows at least, so a thread
    // has at most one of them.
    const bool south = act && jl == 0 && yb > 0, north = act && jl == e.by - 1 && j < P.ny - 1;
    const bool back = act && zb > 0, front = act && z0 + BZ < P.nz, yedge = south || north;
    const int set = 4 * res_faces(BZ, nq, T);  // words of one parity
    // offsets in a set: per plane the S and the N face row, then the B and the F
    // face; each as the words of its quads' cells 0, 1 and then those of 2, 3
    const int xme = cta * 2 * set;
    const int oS = 2 * q, oN = 4 * BZ * nq + oS, oB = 8 * BZ * nq + 2 * tid, oF = oB + 4 * T;
    const int wY = xme + (south ? oS : oN), wB = xme + oB, wF = xme + oF;  // own faces, and the neighbours'
    const int xY = south ? xme - 2 * set + oN : xme + 2 * set + oS, xB = xme - 2 * set * e.nby + oF,
              xF = xme + 2 * set * e.nby + oB;
    // the rows to the south and north of this thread's: its block's (in D) or,
    // at the block's edge, the ones fetched from the neighbour block (0 at a wall)
    const unsigned hS = aY + 16 * PT * q, hN = hS + row;
    if (own)
#pragma unroll
        for (int k = 0; k < BZ; ++k) {
            if (jl == 0) st_sh(hS + 16 * k, zero);
            if (jl == e.by - 1) st_sh(hN + 16 * k, zero);
            if (tid == 0) st_sh(aD - 16 * PT + 16 * k, zero);
        }
    const int dY = south ? -P.PX : P.PX;
    const u64 mom = pk(e.s.mom, e.s.mom), ndh2 = pk(-e.s.dh2, -e.s.dh2), cX = pk(e.s.cX, e.s.cX),
              dx2 = pk(_dx2f, _dx2f), dy2 = pk(_dy2f, _dy2f), dz2 = pk(_dz2f, _dz2f);
    const float* const Rcol = e.Rin + col;
    const bool mute = L.skip == cta + 1, pubY = yedge && !mute, pubB = back && !mute, pubF = front && !mute;
    u64* const xch = e.xch;
    const unsigned hY = south ? hS : hN;
    // the neighbour blocks' cells next to this column: planes before and after
    // it in registers, the row beside it in shared memory
    P4 zB = zero, zF = zero;
    if (back) zB = *reinterpret_cast<const P4*>(e.D + col - pln);
    if (front) zF = *reinterpret_cast<const P4*>(e.D + col + pln * BZ);
    if (yedge)
#pragma unroll
        for (int k = 0; k < BZ; ++k)
            if (k < nk) st_sh(hY + 16 * k, *reinterpret_cast<const P4*>(e.D + col + pln * k + dY));
    __syncthreads();

    bool ok = true;
    auto take_y = [&](int par, unsigned tag) {  // the row is read by the thread that fetches it
        const u64* const w = xch + (xY + par);
        constexpr int G = BZ < 4 ? BZ : 4;  // loads in flight (registers)
#pragma unroll
        for (int g = 0; g < BZ; g += G) {
            FaceWords f[G];
#pragma unroll
            for (int u = 0; u < G; ++u)
                if (g + u < BZ) f[u] = face_ld(w + 4 * nq * (g + u), 2 * nq);
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const int k = g + u;
                if (k >= BZ || k >= nk) continue;
                P4 v = zero;
                ok = ok && face_wait(w + 4 * nq * k, 2 * nq, tag, f[u], L.err, L.limit, v);
                st_sh(hY + 16 * k, v);
            }
        }
    };
    unsigned Dc = aD + me, Dn = Dc + bD;
    for (int it = 0; it < L.iters; ++it) {
        const unsigned tag = L.tag + (unsigned)it + 1u;  // of the iteration's result
        const int par = (it & 1) ? 0 : set;              // its parity's set
        if (it > 0) {  // the neighbours' cells (the load after a barrier mostly finds the words at the first try)
            FaceWords fB, fF;
            if (back) fB = face_ld(xch + (xB + set - par), 2 * T);
            if (front) fF = face_ld(xch + (xF + set - par), 2 * T);
            if (yedge) take_y(set - par, tag - 1u);
            if (back) ok = ok && face_wait(xch + (xB + set - par), 2 * T, tag - 1u, fB, L.err, L.limit, zB);
            if (front) ok = ok && face_wait(xch + (xF + set - par), 2 * T, tag - 1u, fF, L.err, L.limit, zF);
        }
        const unsigned rS = jl > 0 ? Dc - row : hS, rN = jl < e.by - 1 ? Dc + row : hN;
        // D' of plane k from x_c, x_back, x_front
        auto plane = [&](int k, const P4& xc, const P4& xb, const P4& xf, const P4& Rk) {
            // The column west of a row's first quad is the last quad of the row
            // before (or the column of zeros), whose last cell is outside the grid
            // and 0; what lies east of a row's last quad only meets such a cell.
            const float xw = ld_sh1(Dc + 16 * (k - PT) + 12), xe = ld_sh1(Dc + 16 * (k + PT));
            const P4 xs = ld_sh(rS + 16 * k), xn = ld_sh(rN + 16 * k), xp = ld_sh(Dn + 16 * k);
            P4 kxk, ks, kn, r;
            float kEk;
            if constexpr (KS) {
                kxk = ld_sh(aKx + 16 * k);
                kEk = ld_sh1(aKx + 16 * (k + PT));
                ks = ld_sh(aKy + 16 * k);
                kn = ld_sh(aKy + row + 16 * k);
            } else {
                kxk = kx[k];
                kEk = kE[k];
                ks = kyS[k];
                kn = kyN[k];
            }
            if constexpr (RM) r = ld_sh(aR + 16 * k);
            else if constexpr (RS) r = Rk;
            else r = R[k];
            const float2 c01 = unpk(xc.a), c23 = unpk(xc.b), k01 = unpk(kxk.a), k23 = unpk(kxk.b);
            const P4 gy = fma4(ks, sub4(xc, xs), mul4(kn, sub4(xc, xn)));
            const P4 gz = fma4(kz[k], sub4(xc, xb), mul4(kz[k + 1], sub4(xc, xf)));
            // x: differences across the quad's five faces
            const float e0 = __fsub_rn(c01.x, xw), e1 = __fsub_rn(c01.y, c01.x), e2 = __fsub_rn(c23.x, c01.y),
                        e3 = __fsub_rn(c23.y, c23.x), e4 = __fsub_rn(xe, c23.y);
            const P4 gx{pk(__fmaf_rn(k01.x, e0, -__fmul_rn(k01.y, e1)), __fmaf_rn(k01.y, e1, -__fmul_rn(k23.x, e2))),
                        pk(__fmaf_rn(k23.x, e2, -__fmul_rn(k23.y, e3)), __fmaf_rn(k23.y, e3, -__fmul_rn(kEk, e4)))};
            P4 fu = fma4s(cX, xc, r);
            fu = fma4s(dx2, gx, fu);
            fu = fma4s(dy2, gy, fu);
            fu = fma4s(dz2, gz, fu);
            const P4 x1 = fma4s(mom, sub4(xc, xp), fma4s(ndh2, mul4(fu, rd[k]), xc));
            if (own) st_sh(Dn + 16 * k, x1);
            if (pubY) face_st(xch + (wY + par + 4 * nq * k), 2 * nq, tag, x1);
            return x1;
        };
        auto residual = [&](int k) {  // from L2, where it is not kept
            P4 v = zero;
            if (RS && k < nk) {
                const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(Rcol + pln * k));
                v = P4{w.x, w.y};
            }
            return v;
        };
        // first the planes that other blocks wait for ...
        const P4 Ra = residual(0), Rb = residual(BZ - 1);
        P4 R0 = residual(BZ > 2 ? 1 : 0), R1 = residual(BZ > 3 ? 2 : 0);  // and two planes ahead of the others
        const P4 x0 = ld_sh(Dc);
        P4 x1 = zF;
        if constexpr (BZ > 1) x1 = ld_sh(Dc + 16);
        {
            const P4 y0 = plane(0, x0, zB, x1, Ra);
            if (pubB) face_st(xch + (wB + par), 2 * T, tag, y0);
            if (BZ == 1 && pubF) face_st(xch + (wF + par), 2 * T, tag, y0);
        }
        if constexpr (BZ > 1) {
            const P4 xl = ld_sh(Dc + 16 * (BZ - 1)), xm = ld_sh(Dc + 16 * (BZ - 2));
            const P4 y0 = plane(BZ - 1, xl, xm, zF, Rb);
            if (pubF) face_st(xch + (wF + par), 2 * T, tag, y0);
        }
        // ... then the others, while the faces travel
        if constexpr (BZ > 2) {
            P4 xb = ld_sh(Dc), xc = ld_sh(Dc + 16);
#pragma unroll
            for (int k = 1; k < BZ - 1; ++k) {
                const P4 xf = ld_sh(Dc + 16 * (k + 1));
                const P4 Rk = R0;
                R0 = R1;
                if (k + 2 < BZ - 1) R1 = residual(k + 2);
                plane(k, xc, xb, xf, Rk);
                xb = xc;
                xc = xf;
            }
        }
        const unsigned t = Dc;
        Dc = Dn;
        Dn = t;
        if (__syncthreads_or(!ok)) {  // a wait gave up (here or, seen through *err, elsewhere): the CTA leaves together
            if (threadIdx.x == 0) atomicExch(L.err, HT3D_ERR_TIMEOUT);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < BZ; ++k)
        if (act && k < nk) {
            *reinterpret_cast<P4*>(e.Dout + col + pln * k) = ld_sh(Dc + 16 * k);
            *reinterpret_cast<P4*>(e.Dpout + col + pln * k) = ld_sh(Dn + 16 * k);
        }
}

// ------------------------------------------------------------------ host side
struct ResPlan {
    int bz = 0, nq = 0, by = 0, nby = 0, nbz = 0, T = 0;  // bz 0: does not fit
    int ctas() const { return nby * nbz; }
    int work() const { return bz * ((T + 31) / 32); }  // warp-wide quads of a CTA per iteration
};
inline ResPlan res_plan_with(const Pad& P, int bz, int by) {
    ResPlan r;
    r.nq = (P.nx + 4) / 4;  // quads that hold a row's nx + 1 faces
    r.bz = bz;
    r.by = by;
    r.nby = (P.ny + by - 1) / by;
    r.nbz = (P.nz + bz - 1) / bz;
    r.T = r.nq * by;
    return r;
}
constexpr int kResBZ[] = {1, 2, 3, 5, 7};  // the compiled column heights
// rows of the largest block with columns of bz planes (0: none fits)
inline int res_max_by(const Pad& P, int bz, int threads, size_t smem) {
    const int nq = (P.nx + 4) / 4;
    int by = std::min(P.ny, threads / nq);
    while (by > 0 && res_smem(bz, nq, by) > smem) --by;
    return by == 1 && P.ny > 1 ? 0 : by;  // a block with a neighbour in y has two rows at least
}
// The plan of one grid on a device of `sms` SMs.  An iteration's time goes with
// the height of the columns (1.1-1.3, 1.5-1.7, 1.9-2.6, 3.2-3.8 and 4.3-4.9 us
// for 1, 2, 3, 5 and 7 planes, against 4.0 us at 63^3, 6.2 at 95^3 and 9.7 at
// 127 x 119 x 131 for one launch per iteration), so the lowest that fit win.
// Columns of up to three planes wait for their neighbours most of the time: two
// CTAs share an SM (79^3, two planes: 1.62 us against 1.91 for three planes and
// one CTA) unless blocks can span the rows.  Fewer, larger row blocks are faster
// up to five planes (47^3, five planes: 2.6 us with 24 rows, 3.5 with 6), the
// smaller ones with seven (100 x 110 x 120: 4.3 us with 14 rows, 5.0 with 19).
inline ResPlan res_plan(const Pad& P, int sms) {
    for (int bz : kResBZ) {
        const int nbz = (P.nz + bz - 1) / bz, by1 = res_max_by(P, bz, kResThreads, kResSmem);
        if (by1 < 1) continue;
        const int nby1 = (P.ny + by1 - 1) / by1;
        if (bz <= 3) {
            if (nby1 == 1 && nbz <= sms) return res_plan_with(P, bz, P.ny);
            const int by2 = res_max_by(P, bz, kResThreads2, kResSmem2);
            const int nby2 = by2 ? (P.ny + by2 - 1) / by2 : 0;
            if (by2 && (long long)nbz * nby2 <= 2LL * sms) return res_plan_with(P, bz, (P.ny + nby2 - 1) / nby2);
        }
        if ((long long)nbz * nby1 > sms) continue;
        const int nby = bz == 7 ? sms / nbz : nby1;
        return res_plan_with(P, bz, std::min(by1, std::max(2, (P.ny + nby - 1) / nby)));
    }
    return ResPlan();
}
// The plan of one of many grids that share the chip: large blocks, one per SM
// (64 members of 31 to 95 cells a side, all iterations of a pass: 39.5 us per
// iteration with five planes first, 43.2 with seven, 47.0 with three and two
// CTAs per SM; 64.9 for the batched kernel with one launch per iteration).
inline ResPlan res_plan_full(const Pad& P, int sms) {
    for (int bz : {5, 7}) {
        const int by = res_max_by(P, bz, kResThreads, kResSmem);
        if (!by) continue;
        const int nby = (P.ny + by - 1) / by;
        const ResPlan r = res_plan_with(P, bz, (P.ny + nby - 1) / nby);
        if (r.ctas() <= sms) return r;
    }
    return ResPlan();
}
// The shortest run of a solve that pays for loading a block's fields and writing
// them back.  300 iterations, runs of two with a check behind each in one launch
// and single: 16^3 3.38 and 2.99 ms, 95^3 (five planes) 9.24 and 8.93, 127 x 119 x
// 131 15.9 and 15.7; of four 2.32 and 2.31, 6.83 and 6.46, 11.4 and 11.6; of six 1.79
// and 1.89, 5.29 and 5.33, 9.09 and 9.35.
inline int res_shortest(const ResPlan& r) { return r.bz == 5 ? 6 : 4; }
// us per iteration of a wave whose tallest plan this is (within a tenth or so of
// the figures above and of 31^3 to 127^3, thin and long grids as ensembles)
inline double res_time(const ResPlan& r, const Pad& P) {
    return 1.2 + 0.00095 * r.T * std::min(r.bz, P.nz) + (r.nby > 1 ? 0.0009 * r.bz * r.nq : 0.0);
}
inline size_t res_words(const ResPlan& r) { return (size_t)r.ctas() * 8 * res_faces(r.bz, r.nq, r.T); }

// Room for the face words of a launch; false where the device has none.  Numbers
// of earlier iterations may stand in them, so they are cleared only when they are
// allocated and when the numbers run out.
inline bool res_reserve(ht3d_ctx* ctx, size_t words) {
    if (ctx->slot_bytes[SLOT_RES] >= words * sizeof(u64)) return true;
    try {
        ht3d_scratch(ctx, SLOT_RES, words * sizeof(u64));
    } catch (const ht3d_error& e) {
        if (e.code != HT3D_ERR_NOMEM) throw;
        return false;
    }
    HT3D_CUDA(cudaMemsetAsync(ctx->slot_ptr[SLOT_RES], 0, ctx->slot_bytes[SLOT_RES], ctx->stream));
    ctx->res_tag = 0;
    return true;
}
inline u64* res_exchange(ht3d_ctx* ctx, int iters, unsigned& tag) {
    if (ctx->res_tag > 0xffffffffu - (unsigned)iters - 1u) {
        HT3D_CUDA(cudaMemsetAsync(ctx->slot_ptr[SLOT_RES], 0, ctx->slot_bytes[SLOT_RES], ctx->stream));
        ctx->res_tag = 0;
    }
    tag = ctx->res_tag;
    ctx->res_tag += (unsigned)iters;
    return (u64*)ctx->slot_ptr[SLOT_RES];
}

inline ResMember res_member(const ResPlan& r, const Pad& P, const float* D, const float* Dp, const float* Rin,
                            const float* kx, const float* ky, const float* kz, float* Dout, float* Dpout,
                            const MixScal& s, const BC6<float>& bc, u64* xch) {
    ResMember m{D, Dp, Rin, kx, ky, kz, Dout, Dpout, xch, P, s, 0, r.nq, r.by, r.nby, r.T};
    for (int f = 0; f < 6; ++f) m.dir |= bc.dir[f] ? 1 << f : 0;
    return m;
}

// The launch's limit of polls and, for HT3D_TUNE_WAIT_TEST, the CTA of each member
// that stays silent; a launch in which no other CTA waits for one leaves the test
// armed.  (Counted by member, as the kernel does at hand: with the launch's own count
// 127 x 119 x 131, whose registers are full, took 1.6 % longer.)
inline void res_wait(ht3d_ctx* ctx, ResLaunch& L) {
    L.skip = 0;
    L.limit = kResWaitLimit;
    const int v = ctx->wait_test;
    for (int m = 0; m < L.n; ++m) {
        const int blocks = L.block0[m + 1] - L.block0[m];
        if (v > 0 && v <= blocks && blocks > 1) {
            L.skip = v;
            L.limit = 1u << 12;
            ctx->wait_test = 0;
        }
    }
}

inline const void* res_kernel(int bz) {
    static void (*const kern[])(ResLaunch) = {k_mixed_resident<1>, k_mixed_resident<2>, k_mixed_resident<3>,
                                              k_mixed_resident<5>, k_mixed_resident<7>};
    for (size_t c = 0; c < std::size(kResBZ); ++c)
        if (kResBZ[c] == bz) return (const void*)kern[c];
    throw ht3d_error(HT3D_ERR_ARG, "no kernel for columns of this height");
}
// Whether the device holds `blocks` CTAs of columns of bz planes at once (asked
// when a run is planned: a launch that it then refuses is an error).
inline bool res_fits(ht3d_ctx* ctx, int bz, int threads, size_t smem, long long blocks) {
    const void* f = res_kernel(bz);
    int coop = 0, optin = 0, per_sm = 0;
    HT3D_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
    HT3D_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    if (!coop || (size_t)optin < kResSmem) return false;
    HT3D_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem));
    HT3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, (threads + 31) / 32 * 32, smem));
    return blocks <= (long long)per_sm * ctx->num_sms;
}
inline bool res_fits(ht3d_ctx* ctx, const ResPlan& r) {
    return r.bz > 0 && res_fits(ctx, r.bz, r.T, res_smem(r.bz, r.nq, r.by), r.ctas());
}

inline void res_launch(ht3d_ctx* ctx, int bz, const ResLaunch& L, int threads, size_t smem) {
    void* args[] = {(void*)&L};
    HT3D_CUDA(cudaLaunchCooperativeKernel(res_kernel(bz), dim3((unsigned)L.block0[L.n]),
                                          dim3((unsigned)((threads + 31) / 32 * 32)), args, smem, ctx->stream));
    ctx->launches++;
}
