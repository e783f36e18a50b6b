// Pressure projection: boundary reset, Poisson coefficients + divergence, Jacobi-preconditioned
// CG with FP64 reductions, pressure/density update and the velocity correction.
// Follows pressureProject / calculatePressureProject (Game/environment.cu:851-987).
#include "skt_internal.cuh"
#include "skt_tma.cuh"

namespace skt {

namespace {

constexpr int TX = 32, TY = 8, NT = TX * TY;

struct Tiles {
    int tx, ty, n;  // tiles along x, along y, total (including z)
};
inline Tiles tiles_of(const Grid& g) {
    Tiles t;
    t.tx = (g.X + TX - 1) / TX;
    t.ty = (g.Y + TY - 1) / TY;
    t.n = t.tx * t.ty * g.Z;
    return t;
}
__device__ __forceinline__ void tile_cell(const Grid& g, const Tiles& T, int t, int& x, int& y, int& z) {
    const int txy = T.tx * T.ty;
    z = t / txy;
    const int r = t - z * txy;
    const int ty = r / T.tx;
    const int tx = r - ty * T.tx;
    x = tx * TX + (threadIdx.x & (TX - 1));
    y = ty * TY + (threadIdx.x / TX);
}

__device__ __forceinline__ float char_trunc(float a) {  // (char) of a float: truncate, saturate (Q3)
    const float t = truncf(a);
    return fminf(fmaxf(t, -128.0f), 127.0f);
}
// The face coefficient -max(1, 1.225 / hm) of two cells (initAMatrix Game/kernelSky.cu:1372), hm =
// 2 / (1/c + 1/n) the harmonic mean of their densities; 0 across a zero density (a ground cell)
__device__ __forceinline__ float coef_of(float c, float n) {
    return n == 0.0f ? 0.0f : -fmaxf(1.0f, 1.225f / (2.0f / (1.0f / c + 1.0f / n)));
}
// The same from the sum s of the reciprocal densities without its two divisions: 1.225 / hm is 0.6125 s up
// to rounding, and differs from it by one unit in the last place at most (checked for every significand:
// both scale with powers of two). The setup stores that difference, 0 to 2 for -1 to 1.
__device__ __forceinline__ unsigned coef_delta(float s) {
    return unsigned(__float_as_int(__fdiv_rn(1.225f, __fdiv_rn(2.0f, s))) - __float_as_int(0.6125f * s) + 1) & 3u;
}
__device__ __forceinline__ float coef_of_sum(float s, unsigned delta) {
    return -fmaxf(1.0f, __int_as_float(__float_as_int(0.6125f * s) + int(delta) - 1));
}
__device__ __forceinline__ float precon_of(float w) { return w == 0.0f ? 1.0f : 1.0f / w; }  // initPrecon :1409

// What the matrix-free operator needs of a cell besides its reciprocal density, one word: the three upper
// faces' coefficients as Q3 has them when they are another cell's lower ones, (char) of the float, their
// magnitudes 0 to 128 in a byte each (right, up, front), and four coef_deltas of two bits: the same
// faces' and that of a lower face that leaves the grid (the own density on both sides).
__device__ __forceinline__ unsigned pack_faces(float cr, float cu, float cf, float sr, float su, float sf, float sown) {
    return unsigned(-char_trunc(cr)) | unsigned(-char_trunc(cu)) << 8 | unsigned(-char_trunc(cf)) << 16 | coef_delta(sr) << 24 |
           coef_delta(su) << 26 | coef_delta(sf) << 28 | coef_delta(sown) << 30;
}
// a truncated coefficient as a float again (the byte under the exponent of 2^23, which is then taken off:
// two full-rate instructions, where the conversion runs at an eighth of that)
template <int BYTE>
__device__ __forceinline__ float trunc_of(unsigned w) {
    return 8388608.0f - __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440 + BYTE));
}
enum { FACE_R = 24, FACE_U = 26, FACE_F = 28, FACE_OWN = 30 };  // the deltas' places
template <int FACE>
__device__ __forceinline__ unsigned delta_of(unsigned w) { return (w >> FACE) & 3u; }

// resetVelPressProj Game/kernelSky.cu:1648-1682: the faces on the far sides and against ground cells.
// reference=1 stops a column (x,y) at its first ground cell along z (Q8).
// Flat terrain: the far sides of rows y >= 1 only, a thread per face; as a march of every column along z, a
// chain of Z loads, it took 33 us at 64x32x64 and 153 at 256x128x256, now 3.4 and 3.6.
__global__ void __launch_bounds__(256) k_reset_faces(Grid g, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                                                     const float* __restrict__ defU, const float* __restrict__ defW) {
    after_previous();
    const int X = g.X, Y = g.Y, Z = g.Z;
    unsigned i = blockIdx.x * 256u + threadIdx.x;  // may exceed 2^31 (far_faces)
    if (i < unsigned(X * Y)) {
        if (i >= unsigned(X)) w[int(i) + (Z - 1) * g.XY] = defW[int(i) / X];
        return;
    }
    i -= unsigned(X * Y);
    if (i < unsigned(X * Z)) {
        if (Y > 1) v[cidx(g, int(i) % X, Y - 1, int(i) / X)] = 0.0f;
        return;
    }
    i -= unsigned(X * Z);
    if (i < unsigned(Y * Z) && int(i) % Y > 0) u[cidx(g, X - 1, int(i) % Y, int(i) / Y)] = defU[int(i) % Y];
}
// Over terrain: one thread per (x,y) marching z, RVZ planes' heights loaded at a time (one at a time
// 63 us at 128x64x128, now 19)
constexpr int RVZ = 8;
__global__ void __launch_bounds__(128) k_reset_vel(Grid g, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                                                   const float* __restrict__ defU, const float* __restrict__ defW, int reference) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.XY) return;
    const int x = t % g.X, y = t / g.X, X = g.X, Z = g.Z;
    const int right = x + 1 < X ? 1 : 0;
    for (int z0 = 0; z0 < Z; z0 += RVZ) {
        int h[RVZ + 1], hr[RVZ];
#pragma unroll
        for (int i = 0; i <= RVZ; ++i) h[i] = __ldg(g.gh + x + min(z0 + i, Z - 1) * X);
#pragma unroll
        for (int i = 0; i < RVZ; ++i) hr[i] = __ldg(g.gh + x + right + min(z0 + i, Z - 1) * X);
#pragma unroll
        for (int i = 0; i < RVZ; ++i) {
            const int z = z0 + i;
            if (z >= Z) return;
            if (y <= h[i]) {
                if (reference) return;
                continue;
            }
            const int c = t + z * g.XY;
            if (y == g.Y - 1) v[c] = 0.0f;
            if (x == X - 1) u[c] = defU[y];
            if (right && y <= hr[i]) u[c] = 0.0f;
            if (z == Z - 1) w[c] = defW[y];
            else if (y <= h[i + 1]) w[c] = 0.0f;
        }
    }
}

// initAMatrix (Game/kernelSky.cu:1320-1393, density bounds NEUMANN sides / DIRICHLET ground)
// fused with calculateDivergenceGPU (:780-860, velocity bounds CUSTOM sides / DIRICHLET ground),
// the preconditioned start z = r/diag, s = z, sigma0 = z.r and the first max residual.
__global__ void __launch_bounds__(NT) k_build(Grid g, Tiles T, const float* __restrict__ rho, const float* __restrict__ u,
                                              const float* __restrict__ v, const float* __restrict__ w,
                                              const float* __restrict__ defU, const float* __restrict__ defW, float dt,
                                              float* __restrict__ ax, float* __restrict__ ay, float* __restrict__ az, float* __restrict__ aw,
                                              float* __restrict__ r, float* __restrict__ s, float* __restrict__ pp, float* __restrict__ As,
                                              int faces, int reference, Scalars* sc, double* partials) {
    Sum dsum;
    float mx = 0.0f;
    for (int t = blockIdx.x; t < T.n; t += gridDim.x) {
        int x, y, z;
        tile_cell(g, T, t, x, y, z);
        if (x >= g.X || y >= g.Y) continue;
        const int c = cidx(g, x, y, z);
        pp[c] = 0.0f;
        if (faces) As[c] = 0.0f;
        if (is_ground(g, x, y, z)) {
            ax[c] = ay[c] = aw[c] = 0.0f;
            if (faces) az[c] = 0.0f;
            r[c] = 0.0f;
            s[c] = 0.0f;
            continue;
        }
        const float cur = rho[c];
        const float nr = ghost(g, rho, x + 1, y, z, NEUMANN, DIRICHLET, nullptr);
        const float nl = ghost(g, rho, x - 1, y, z, NEUMANN, DIRICHLET, nullptr);
        const float nu = ghost(g, rho, x, y + 1, z, NEUMANN, DIRICHLET, nullptr);
        const float nd = ghost(g, rho, x, y - 1, z, NEUMANN, DIRICHLET, nullptr);
        const float nf = ghost(g, rho, x, y, z + 1, NEUMANN, DIRICHLET, nullptr);
        const float nb = ghost(g, rho, x, y, z - 1, NEUMANN, DIRICHLET, nullptr);
        const float cr = coef_of(cur, nr), cl = coef_of(cur, nl), cu = coef_of(cur, nu);
        const float cd = coef_of(cur, nd), cf = coef_of(cur, nf), cb = coef_of(cur, nb);
        if (faces) {
            ax[c] = cr;
            ay[c] = cu;
            az[c] = cf;
        } else {
            const float ri = 1.0f / cur;
            ax[c] = ri;  // the matrix-free operator's inputs
            reinterpret_cast<unsigned*>(ay)[c] = pack_faces(cr, cu, cf, ri + 1.0f / nr, ri + 1.0f / nu, ri + 1.0f / nf, ri + ri);
        }
        float wd = 0.0f;
        wd -= cr; wd -= cl; wd -= cu; wd -= cd; wd -= cf; wd -= cb;
        aw[c] = wd;
        // divergence
        const float ur = u[c], ul = face_nb(g, u, x, y, z, -1, 0, 0, CUSTOM, DIRICHLET, defU[y]);
        const float uu = v[c], ud = face_nb(g, v, x, y, z, 0, -1, 0, CUSTOM, DIRICHLET, 0.0f);
        const float uf = w[c], ub = face_nb(g, w, x, y, z, 0, 0, -1, CUSTOM, DIRICHLET, defW[y]);
        auto hm = [&](float d) { return d == 0.0f ? 0.0f : 2.0f / (1.0f / cur + 1.0f / d); };
        const float dr = hm(nr), dl = hm(nl), du = hm(nu), dd = hm(nd), df = hm(nf), db = hm(nb);
        const float mfd = ((dr * ur - dl * ul) + (du * uu - dd * ud) + (df * uf - db * ub));
        const float dch = (cur - rho[c]) / dt;  // the reference's old density is a copy of rho
        const float rv = mfd - dch;
        r[c] = rv;
        const float zv = rv * precon_of(wd);
        s[c] = zv;
        dsum.add_prod(zv, rv);
        const float m = (!reference || z == 0) ? fabsf(rv) : rv;
        if (m > mx) mx = m;
    }
    double tot;
    float mall;
    if (grid_sum_max<NT, true>(sc, partials, blockIdx.x, gridDim.x, threadIdx.x, dsum, mx, tot, mall)) {
        sc->sigma0 = tot;
        sc->sigma1 = 0.0;
        sc->iters = 0;
        sc->residual = mall;
        sc->converged = (mall == 0.0f) ? 1 : 0;
    }
}

// As = A s and s.As (applyAGPU Game/kernelSky.cu:719-778 + dotProductGPU :675-717), any X.
// reference=1: lower coefficients pass through a char (Q3) and the denominator keeps accumulating (Q1).
// A lane owns MR rows of one x cell and marches a run of z planes with the planes of s in registers and the
// next plane's loads in flight; x neighbours come from the lanes beside. Ground cells hold s = 0 and
// coefficients 0, as does the face to one, so no neighbour is tested. Blocks take their (x, y, z run) tiles
// in turn, whatever their number.
// What bounds it: HBM (24 bytes a cell) and the loads' instructions. A thread per cell that asked the
// heights about every neighbour took 77 us at 251x118x275, now
// 59 (52 with the sums in pairs of floats; then one or two rows a lane 62 and 65, eight warps a block 58).
constexpr int MR = 4, MW = 4;  // rows per lane, warps per block
struct Runs {
    int nx, ny, n, zlen;  // tiles along x and y, all of them, planes per tile
};
inline Runs matvec_runs(const Grid& g, int sms) {
    Runs t;
    t.nx = (g.X + 31) / 32;
    t.ny = (g.Y + MR * MW - 1) / (MR * MW);
    int zc = std::max(1, std::min(g.Z, (sms * 8 + t.nx * t.ny - 1) / (t.nx * t.ny)));
    t.zlen = (g.Z + zc - 1) / zc;
    t.n = t.nx * t.ny * ((g.Z + t.zlen - 1) / t.zlen);
    return t;
}
__global__ void __launch_bounds__(32 * MW, 4) k_matvec(Grid g, Runs T, const float* __restrict__ ax, const float* __restrict__ ay,
                                                    const float* __restrict__ az, const float* __restrict__ aw, const float* __restrict__ s,
                                                    float* __restrict__ As, int reference, Scalars* sc, double* partials) {
    if (sc->converged) return;
    const int X = g.X, Y = g.Y, Z = g.Z, XY = g.XY, lane = threadIdx.x;
    // the thread's sum waits in shared memory: four blocks an SM leave the march 128 registers and none for it
    // (141 registers and three blocks 69 us at 251x118x275, spills 62, this 59)
    constexpr int NTH = 32 * MW;
    __shared__ float part[3][NTH];
    __shared__ double far[NTH];
    const int tid = threadIdx.y * 32 + lane;
    volatile float* const mine = &part[0][tid];
    mine[0] = mine[NTH] = mine[2 * NTH] = 0.0f;
    far[tid] = 0.0;
    struct Plane {
        float cx[MR], cy[MR], cz[MR], cw[MR], es[MR], ea[MR], up, down, cd;
    };
    for (int t = blockIdx.x; t < T.n; t += gridDim.x) {
        const int xo = (t % T.nx) * 32 + lane, y0 = ((t / T.nx) % T.ny * MW + threadIdx.y) * MR;
        const int zs = t / (T.nx * T.ny) * T.zlen, ze = min(zs + T.zlen, Z);
        if (y0 >= Y) continue;  // a whole warp
        const int x = min(xo, X - 1);  // the lanes beyond a row follow its last cell, the rows beyond the top the top one
        const int rows = xo < X ? min(MR, Y - y0) : 0;
        const bool el = lane == 0 && x > 0, er = lane == 31 && x + 1 < X, first = x == 0, last = x + 1 == X;
        int ro[MR];
#pragma unroll
        for (int r = 0; r < MR; ++r) ro[r] = min(r, Y - 1 - y0) * X;
        int c = x + y0 * X + zs * XY;
        auto load = [&](int cc, Plane& P) {
            P.up = y0 + MR < Y ? s[cc + MR * X] : 0.0f;
            P.down = y0 > 0 ? s[cc - X] : 0.0f;
            P.cd = y0 > 0 ? ay[cc - X] : 0.0f;
#pragma unroll
            for (int r = 0; r < MR; ++r) {
                const int q = cc + ro[r];
                P.cx[r] = ax[q]; P.cy[r] = ay[q]; P.cz[r] = az[q]; P.cw[r] = aw[q];
                P.es[r] = el || er ? s[q + (el ? -1 : 1)] : 0.0f;
                P.ea[r] = el ? ax[q - 1] : 0.0f;
            }
        };
        float q[MR], n[MR], b[MR], zb[MR];
        Plane P;
        load(c, P);
#pragma unroll
        for (int r = 0; r < MR; ++r) {
            q[r] = s[c + ro[r]];
            n[r] = zs + 1 < Z ? s[c + ro[r] + XY] : 0.0f;
            b[r] = zs > 0 ? s[c + ro[r] - XY] : 0.0f;
            zb[r] = zs > 0 ? az[c + ro[r] - XY] : 0.0f;
        }
        for (int z = zs; z < ze; ++z, c += XY) {
            Plane N;
            float n2[MR], o[MR];
            if (z + 1 < ze) load(c + XY, N);
#pragma unroll
            for (int r = 0; r < MR; ++r) n2[r] = z + 2 <= ze && z + 2 < Z ? s[c + ro[r] + 2 * XY] : 0.0f;
#pragma unroll
            for (int r = 0; r < MR; ++r) {
                const float v = q[r];
                float sl = __shfl_up_sync(0xffffffffu, v, 1), sr = __shfl_down_sync(0xffffffffu, v, 1), AL = __shfl_up_sync(0xffffffffu, P.cx[r], 1);
                if (el) { sl = P.es[r]; AL = P.ea[r]; }
                if (er) sr = P.es[r];
                if (first) sl = AL = 0.0f;
                if (last) sr = 0.0f;
                const float sd = r > 0 ? q[r > 0 ? r - 1 : 0] : P.down;
                float AD = r > 0 ? P.cy[r > 0 ? r - 1 : 0] : P.cd, AB = zb[r];
                const float su = y0 + r + 1 < Y ? (r + 1 < MR ? q[r + 1 < MR ? r + 1 : r] : P.up) : 0.0f;
                if (reference) { AL = char_trunc(AL); AD = char_trunc(AD); AB = char_trunc(AB); }
                const float ld = fmaf(AL, sl, __fmul_rn(AD, sd));
                const float out = fmaf(P.cw[r], v, fmaf(P.cz[r], n[r], fmaf(P.cy[r], su, fmaf(P.cx[r], sr, fmaf(AB, b[r], ld)))));
                const bool sky = r < rows && P.cw[r] != 0.0f;
                if (sky) As[c + r * X] = out;  // As of ground cells stays 0
                o[r] = sky ? out : 0.0f;
            }
            Sum dsum;
            dsum.h = mine[0]; dsum.l = mine[NTH]; dsum.t = mine[2 * NTH];
            dsum.add_prods(o, q);
            mine[0] = dsum.h; mine[NTH] = dsum.l; mine[2 * NTH] = dsum.t;
            if (dsum.far != 0.0) far[tid] += dsum.far;
#pragma unroll
            for (int r = 0; r < MR; ++r) {
                b[r] = q[r];
                q[r] = n[r];
                n[r] = n2[r];
                zb[r] = P.cz[r];
            }
            P = N;
        }
    }
    double tot;
    float mall;
    Sum dsum;
    dsum.h = mine[0]; dsum.l = mine[NTH]; dsum.t = mine[2 * NTH];
    dsum.far = far[tid];
    if (grid_sum_max<NTH, true>(sc, partials, blockIdx.x, gridDim.x, tid, dsum, 0.0f, tot, mall)) {
        const double s1 = reference ? sc->sigma1 + tot : tot;
        sc->sigma1 = s1;
        sc->alpha = float(sc->sigma0 / s1);
    }
}

// The arrays as float4 streams and a scalar rest (any X; ground cells hold 0, which every formula keeps):
// fn(value, place) for value in float4 or float form
template <class F4, class F1>
__device__ __forceinline__ void stream4(int n, F4 four, F1 one) {
    const int n4 = n / 4, t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = t; i < n4; i += gridDim.x * blockDim.x) four(i);
    if (t < n - 4 * n4) one(4 * n4 + t);
}

// p += alpha s; r -= alpha As (updatePandDiv :955-985), then the stop test on the max residual
// (getMaxDivergence, Q4 in reference mode: |r| on the z = 0 plane only), z = r/diag and z.r for the next search
// direction. HBM-bound, 28 bytes a cell: 115 us at 251x118x275 cell by cell in tiles, 43 as float4 streams.
__global__ void __launch_bounds__(NT) k_update(int n, int XY, const float* __restrict__ aw, const float* __restrict__ s,
                                               const float* __restrict__ As, float* __restrict__ pp, float* __restrict__ r,
                                               int reference, float tol, int max_iter, Scalars* sc, double* partials) {
    if (sc->converged) return;
    const float alpha = sc->alpha;
    Sum dsum;
    float mx = 0.0f;
    auto cell = [&](float a, float sv, float av, float& pv, float& rv, int c) {
        pv += alpha * sv;
        rv = rv - alpha * av;
        const float m = (!reference || c < XY) ? fabsf(rv) : rv;
        if (m > mx) mx = m;
        return rv * precon_of(a);
    };
    stream4(n,
            [&](int i) {
                const float4 a = reinterpret_cast<const float4*>(aw)[i], sv = reinterpret_cast<const float4*>(s)[i];
                const float4 av = reinterpret_cast<const float4*>(As)[i];
                float4 pv = reinterpret_cast<float4*>(pp)[i], rv = reinterpret_cast<float4*>(r)[i];
                const float z0 = cell(a.x, sv.x, av.x, pv.x, rv.x, 4 * i), z1 = cell(a.y, sv.y, av.y, pv.y, rv.y, 4 * i + 1);
                const float z2 = cell(a.z, sv.z, av.z, pv.z, rv.z, 4 * i + 2), z3 = cell(a.w, sv.w, av.w, pv.w, rv.w, 4 * i + 3);
                reinterpret_cast<float4*>(pp)[i] = pv;
                reinterpret_cast<float4*>(r)[i] = rv;
                const float z[4] = {z0, z1, z2, z3}, q[4] = {rv.x, rv.y, rv.z, rv.w};
                dsum.add_prods(z, q);
            },
            [&](int c) {
                float pv = pp[c], rv = r[c];
                const float z = cell(aw[c], s[c], As[c], pv, rv, c);
                pp[c] = pv;
                r[c] = rv;
                dsum.add_prod(z, rv);
            });
    double tot;
    float mall;
    if (grid_sum_max<NT, true>(sc, partials, blockIdx.x, gridDim.x, threadIdx.x, dsum, mx, tot, mall)) {
        sc->iters += 1;
        sc->residual = mall;
        if (mall <= tol) {
            sc->converged = 1;
        } else if (sc->iters >= max_iter) {
            sc->converged = 2;  // stopped at the iteration cap (the reference falls through, :986)
        } else {
            sc->sigma1 = tot;
            sc->beta_f = float(tot / sc->sigma0);
            sc->sigma0 = tot;
        }
    }
}

// s = z + beta s (endIteration :987-1014), z recomputed from r and the diagonal; 16 bytes a cell, 72 us at
// 251x118x275 in tiles, now 24
__global__ void __launch_bounds__(NT) k_search(int n, const float* __restrict__ aw, const float* __restrict__ r, float* __restrict__ s,
                                               const Scalars* sc) {
    if (sc->converged) return;
    const float beta = sc->beta_f;
    auto cell = [&](float a, float rv, float sv) {
        return fmaf(beta, sv, __fmul_rn(rv, precon_of(a)));
    };
    stream4(n,
            [&](int i) {
                const float4 a = reinterpret_cast<const float4*>(aw)[i], rv = reinterpret_cast<const float4*>(r)[i];
                const float4 sv = reinterpret_cast<float4*>(s)[i];
                reinterpret_cast<float4*>(s)[i] = make_float4(cell(a.x, rv.x, sv.x), cell(a.y, rv.y, sv.y), cell(a.z, rv.z, sv.z), cell(a.w, rv.w, sv.w));
            },
            [&](int c) { s[c] = cell(aw[c], r[c], s[c]); });
}

// ---- vectorised PCG iteration (X % 4 == 0): float4 streams, FP32-compensated per-thread sums,
// FP64 across warps and blocks --------------------------------------------------------------

struct Kahan {  // compensated FP32 running sum of one thread
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float v) {
        const float y = v - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ Sum sum() const { return sum_of(s, c); }
};

constexpr int UT = 256;

// p += alpha s, r -= alpha As, z = r/diag, z.r and the max residual, over all cells as float4
// (ground cells hold s = As = r = 0 and diag 0, so they contribute nothing and stay zero).
__global__ void __launch_bounds__(UT) k_update4(int n4, int xy4, const float4* __restrict__ aw, const float4* __restrict__ s,
                                                const float4* __restrict__ As, float4* __restrict__ pp, float4* __restrict__ r,
                                                int reference, float tol, int max_iter, Scalars* sc, double* partials) {
    if (sc->converged) return;
    const float alpha = sc->alpha;
    Kahan acc;
    float mx = 0.0f;
    for (int i = blockIdx.x * UT + threadIdx.x; i < n4; i += gridDim.x * UT) {
        const float4 a = aw[i], sv = s[i], av = As[i];
        float4 pv = pp[i], rv = r[i];
        pv.x += alpha * sv.x; pv.y += alpha * sv.y; pv.z += alpha * sv.z; pv.w += alpha * sv.w;
        rv.x = rv.x - alpha * av.x; rv.y = rv.y - alpha * av.y; rv.z = rv.z - alpha * av.z; rv.w = rv.w - alpha * av.w;
        pp[i] = pv;
        r[i] = rv;
        const float z0 = rv.x * precon_of(a.x), z1 = rv.y * precon_of(a.y), z2 = rv.z * precon_of(a.z), z3 = rv.w * precon_of(a.w);
        acc.add(z0 * rv.x);
        acc.add(z1 * rv.y);
        acc.add(z2 * rv.z);
        acc.add(z3 * rv.w);
        const bool absv = !reference || i < xy4;  // the reference takes |r| on the z = 0 plane only (Q4)
        const float m0 = absv ? fabsf(rv.x) : rv.x, m1 = absv ? fabsf(rv.y) : rv.y;
        const float m2 = absv ? fabsf(rv.z) : rv.z, m3 = absv ? fabsf(rv.w) : rv.w;
        if (m0 > mx) mx = m0;
        if (m1 > mx) mx = m1;
        if (m2 > mx) mx = m2;
        if (m3 > mx) mx = m3;
    }
    double tot;
    float mall;
    if (grid_sum_max<UT, false>(sc, partials, blockIdx.x, gridDim.x, threadIdx.x, acc.sum(), mx, tot, mall)) {
        sc->iters += 1;
        sc->residual = mall;
        if (mall <= tol) {
            sc->converged = 1;
        } else if (sc->iters >= max_iter) {
            sc->converged = 2;
        } else {
            sc->sigma1 = tot;
            sc->beta_f = float(tot / sc->sigma0);
            sc->sigma0 = tot;
        }
    }
}

// s = r/diag + beta s over all cells as float4
__global__ void __launch_bounds__(UT) k_search4(int n4, const float4* __restrict__ aw, const float4* __restrict__ r, float4* __restrict__ s,
                                                const Scalars* sc) {
    if (sc->converged) return;
    const float beta = sc->beta_f;
    for (int i = blockIdx.x * UT + threadIdx.x; i < n4; i += gridDim.x * UT) {
        const float4 a = aw[i], rv = r[i];
        float4 sv = s[i];
        sv.x = rv.x * precon_of(a.x) + beta * sv.x;
        sv.y = rv.y * precon_of(a.y) + beta * sv.y;
        sv.z = rv.z * precon_of(a.z) + beta * sv.z;
        sv.w = rv.w * precon_of(a.w) + beta * sv.w;
        s[i] = sv;
    }
}

constexpr int MVY = 32;           // y rows per block (neighbour rows of s mostly from L1)
constexpr int MVT = 32 * MVY;     // threads per block

__device__ __forceinline__ float4 ld4(const float* p, int c) { return *reinterpret_cast<const float4*>(p + c); }
__device__ __forceinline__ float4 f4zero() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }

// As = A s and s.As with 4 cells per thread along x and a march along z that keeps the planes
// z-1, z, z+1 of s and the previous plane's z-coefficient in registers. Neighbours outside the
// domain read as 0; ground neighbours need no test because their s and coefficients are 0.
// FLAT: the ground is the row y = 0 only (no heightfield reads).
template <bool FLAT>
__global__ void __launch_bounds__(MVT) k_matvec4(Grid g, int zlen, const float* __restrict__ ax, const float* __restrict__ ay,
                                                 const float* __restrict__ az, const float* __restrict__ aw, const float* __restrict__ s,
                                                 float* __restrict__ As, int reference, Scalars* sc, double* partials) {
    if (sc->converged) return;
    const int lane = threadIdx.x, tid = threadIdx.x + 32 * threadIdx.y;
    const int x0 = (blockIdx.x * 32 + lane) * 4;
    const int y = blockIdx.y * MVY + threadIdx.y;
    const int zs = blockIdx.z * zlen, ze = min(zs + zlen, g.Z);
    const bool act = x0 < g.X && y < g.Y;
    const int X = g.X, XY = g.XY;
    const int row = x0 + y * X;
    Kahan acc;
    float4 sb = f4zero(), scur = f4zero(), azb = f4zero();
    if (act) {
        const int c = row + zs * XY;
        scur = ld4(s, c);
        if (zs > 0) { sb = ld4(s, c - XY); azb = ld4(az, c - XY); }
    }
    for (int z = zs; z < ze; ++z) {
        const int c = row + z * XY;
        float4 sf = f4zero(), sd = f4zero(), su = f4zero(), ayd = f4zero(), cx = f4zero(), cy = f4zero(), cz = f4zero(), cw = f4zero();
        int4 gh4 = make_int4(0, 0, 0, 0);
        if (act) {
            if (z + 1 < g.Z) sf = ld4(s, c + XY);
            if (y > 0) { sd = ld4(s, c - X); ayd = ld4(ay, c - X); }
            if (y + 1 < g.Y) su = ld4(s, c + X);
            cx = ld4(ax, c); cy = ld4(ay, c); cz = ld4(az, c); cw = ld4(aw, c);
            if (!FLAT) gh4 = *reinterpret_cast<const int4*>(g.gh + x0 + z * X);
        }
        // x neighbours through the neighbouring lanes; the warp's edge lanes load them
        float sl = __shfl_up_sync(0xffffffffu, scur.w, 1);
        float axl = __shfl_up_sync(0xffffffffu, cx.w, 1);
        float sr = __shfl_down_sync(0xffffffffu, scur.x, 1);
        if (act && lane == 0) {
            if (x0 > 0) { sl = s[c - 1]; axl = ax[c - 1]; } else { sl = 0.0f; axl = 0.0f; }
        }
        if (act && (lane == 31 || x0 + 4 >= X)) sr = (x0 + 4 < X) ? s[c + 4] : 0.0f;
        if (act) {
            float AL0 = axl, AL1 = cx.x, AL2 = cx.y, AL3 = cx.z;
            float AD0 = ayd.x, AD1 = ayd.y, AD2 = ayd.z, AD3 = ayd.w;
            float AB0 = azb.x, AB1 = azb.y, AB2 = azb.z, AB3 = azb.w;
            if (reference) {
                AL0 = char_trunc(AL0); AL1 = char_trunc(AL1); AL2 = char_trunc(AL2); AL3 = char_trunc(AL3);
                AD0 = char_trunc(AD0); AD1 = char_trunc(AD1); AD2 = char_trunc(AD2); AD3 = char_trunc(AD3);
                AB0 = char_trunc(AB0); AB1 = char_trunc(AB1); AB2 = char_trunc(AB2); AB3 = char_trunc(AB3);
            }
            float4 o;
            o.x = cw.x * scur.x + ((AL0 * sl + AD0 * sd.x + AB0 * sb.x + cx.x * scur.y + cy.x * su.x + cz.x * sf.x));
            o.y = cw.y * scur.y + ((AL1 * scur.x + AD1 * sd.y + AB1 * sb.y + cx.y * scur.z + cy.y * su.y + cz.y * sf.y));
            o.z = cw.z * scur.z + ((AL2 * scur.y + AD2 * sd.z + AB2 * sb.z + cx.z * scur.w + cy.z * su.z + cz.z * sf.z));
            o.w = cw.w * scur.w + ((AL3 * scur.z + AD3 * sd.w + AB3 * sb.w + cx.w * sr + cy.w * su.w + cz.w * sf.w));
            if (FLAT) {
                if (y == 0) o = f4zero();
            } else {
                if (y <= gh4.x) o.x = 0.0f;
                if (y <= gh4.y) o.y = 0.0f;
                if (y <= gh4.z) o.z = 0.0f;
                if (y <= gh4.w) o.w = 0.0f;
            }
            *reinterpret_cast<float4*>(As + c) = o;
            acc.add(o.x * scur.x);
            acc.add(o.y * scur.y);
            acc.add(o.z * scur.z);
            acc.add(o.w * scur.w);
        }
        sb = scur;
        scur = sf;
        azb = cz;
    }
    double tot;
    float mall;
    if (grid_sum_max<MVT, false>(sc, partials, linear_block(), linear_blocks(), tid, acc.sum(), 0.0f, tot, mall)) {
        const double s1 = reference ? sc->sigma1 + tot : tot;
        sc->sigma1 = s1;
        sc->alpha = float(sc->sigma0 / s1);
    }
}

// ---- fused PCG iteration (X % 4 == 0): two launches per iteration instead of three --------
// The search step (endIteration :987-1014) and the next matrix product share one z march
// (k_pcg_operator4); the residual kernel stores z = r/diag (it forms z for z.r in any case), so the
// operator forms s_new = z + beta s_old from two arrays wherever it needs a neighbour's value. Every
// value is formed as in k_search4 / k_update4 (the search direction as fma(beta, s_old, z), the
// pressure as fma(alpha, s, p)); only the dot products' summation order differs.

constexpr int kDirs = 4;  // direction buffers: iteration k's direction is in buffer k % kDirs
struct Dirs {
    const float* d[kDirs];
};

// s_new = z + beta s_old, As = A s_new, s_new.As -> alpha. Matrix-free: a face's coefficient comes
// from the reciprocal densities of its two cells (0 in ground cells) and its delta in the cell's word
// (pack_faces), bit for bit the stored coefficient. REF: the lower coefficients as Q3 truncates them, from
// the word too.
// A block covers 128 x cells (a warp of four-cell lanes) by OPR rows and marches a run of z planes. The
// four inputs stream through a ring of OPSLOTS shared-memory slots, each plane's boxes (the block's
// cells, 4 more on either side so that the copies start on 16-byte boundaries, a row above and
// below) filled by TMA copies of one thread, OPSLOTS planes ahead, on one mbarrier per slot; outside
// the grid they read 0, which is the direction's value there. A lane carries its direction and
// densities of the planes behind and at hand in registers and takes its neighbours from the slot; one
// barrier a plane frees the slot. s_old and s_new are distinct buffers (a block's halo rows are another
// block's own rows). FIRST: the direction is z itself.
// What bounds it: HBM, 24 bytes a cell where the stored coefficients and the pressure made 40 (421 us a
// launch at 512x512x256 then, 247 now: 6.5 TB/s, 23.5 bytes of DRAM traffic a cell). An iteration with its
// residual and a quarter of the pressure's update went from 635 to 514 us, at 256x256x128 from 103 to 82. Loading the planes into registers instead of the ring left the
// lanes waiting (400 us, DRAM 48 % busy; with a plane's loads ahead and 512 threads a block 460). Tiles
// of 16 rows with 4 or 5 slots: 516 and 518 us an iteration, 20 rows 527, 24 rows 550, 12 rows two blocks
// per SM 531, 8 rows with 5 slots 532.
constexpr int OPR = 8, OPT = 32 * OPR;   // rows and threads per block; two blocks per SM
constexpr int OPW = 136;                 // box width in cells: 4 + 128 + 4
constexpr int OPSLOTS = 4;
constexpr int OPBOX = (OPW * (OPR + 2) * 4 + 127) / 128 * 32;  // floats per box, slots 128-byte aligned
constexpr int op_smem_bytes() { return OPSLOTS * 4 * OPBOX * 4 + OPSLOTS * 8; }
struct OpMaps {
    CUtensorMap z, s, r, w;
};

template <bool FLAT, bool FIRST, bool REF>
__global__ void __launch_bounds__(OPT, 2) k_pcg_operator4(const __grid_constant__ OpMaps maps, Grid g, int zlen, float* __restrict__ snew,
                                                          float* __restrict__ As, int slot, Scalars* sc, double* partials) {
    if (sc->converged) return;
    extern __shared__ __align__(128) unsigned char op_smem[];
    float* const ring = reinterpret_cast<float*>(op_smem);
    uint64_t* const bar = reinterpret_cast<uint64_t*>(ring + OPSLOTS * 4 * OPBOX);
    constexpr unsigned BYTES = OPW * (OPR + 2) * 4 * (3 + !FIRST);
    const float beta = sc->beta_f;
    const int tid = threadIdx.x, lane = tid & 31, wy = tid >> 5;
    const int X = g.X, Y = g.Y, Z = g.Z, XY = g.XY;
    const int bx = int(blockIdx.x) * 128, yb = int(blockIdx.y) * OPR;
    const int x0 = bx + 4 * lane, y = yb + wy;
    const int zs = int(blockIdx.z) * zlen, ze = min(zs + zlen, Z);
    const int p0 = max(zs - 1, 0), p1 = min(ze, Z - 1);  // planes read
    const bool act = x0 < X && y < Y;
    const bool below = FLAT ? y > 1 : y > 0;  // a row that may be sky lies below
    const bool lend = x0 == 0, rend = x0 + 4 >= X, top = y + 1 >= Y;
    const int own = (wy + 1) * OPW + 4 + 4 * lane;  // the lane's cells in a box

    auto issue = [&](int q) {
        const int s = (q - p0) % OPSLOTS;
        float* const d = ring + s * 4 * OPBOX;
        mbar_expect_tx(&bar[s], BYTES);
        tma_load_3d(d, &maps.z, &bar[s], bx - 4, yb - 1, q);
        if (!FIRST) tma_load_3d(d + OPBOX, &maps.s, &bar[s], bx - 4, yb - 1, q);
        tma_load_3d(d + 2 * OPBOX, &maps.r, &bar[s], bx - 4, yb - 1, q);
        tma_load_3d(d + 3 * OPBOX, &maps.w, &bar[s], bx - 4, yb - 1, q);
    };
    if (tid == 0) {
        for (int s = 0; s < OPSLOTS; ++s) mbar_init(&bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int issued = p0;  // thread 0: the next plane to copy
    if (tid == 0)
        for (; issued <= min(p1, p0 + OPSLOTS - 1); ++issued) issue(issued);
    bool ok = true;
    auto wait_plane = [&](int q) {
        const int i = q - p0, s = i % OPSLOTS;
        const unsigned par = unsigned(i / OPSLOTS) & 1u;
        if (!mbar_try_wait(&bar[s], par)) ok = mbar_wait(&bar[s], par) && ok;
        return ring + s * 4 * OPBOX;
    };
    // the direction and the densities at an offset of a plane's slot
    auto dir4 = [&](const float* d, int o) {
        const float4 z = ld4(d, o);
        if (FIRST) return z;
        const float4 s = ld4(d + OPBOX, o);
        return make_float4(__fmaf_rn(beta, s.x, z.x), __fmaf_rn(beta, s.y, z.y), __fmaf_rn(beta, s.z, z.z), __fmaf_rn(beta, s.w, z.w));
    };
    auto dir1 = [&](const float* d, int o) { return FIRST ? d[o] : __fmaf_rn(beta, d[OPBOX + o], d[o]); };
    auto rho4 = [&](const float* d, int o) { return ld4(d + 2 * OPBOX, o); };
    auto word4 = [&](const float* d, int o) { return *reinterpret_cast<const uint4*>(d + 3 * OPBOX + o); };
    // the coefficient between a cell of reciprocal density a and its neighbour b; 0 where one is ground
    auto coef = [&](float a, float b, unsigned delta) {
        const float c = coef_of_sum(a + b, delta);
        return FLAT || (a != 0.0f && b != 0.0f) ? c : 0.0f;
    };

    Kahan acc;
    float4 vb = f4zero(), cB;
    uint4 wb = make_uint4(0, 0, 0, 0);  // the plane before: its front faces are this plane's back ones
    float4 rb;
    const float* d0 = wait_plane(p0);
    if (zs > 0) {
        vb = dir4(d0, own);
        rb = rho4(d0, own);
        wb = word4(d0, own);
        d0 = wait_plane(zs);
    }
    float4 vc = dir4(d0, own), rc = rho4(d0, own);
    if (zs == 0) {  // outside the grid: the own density (NEUMANN)
        const uint4 w = word4(d0, own);
        rb = rc;
        cB = make_float4(coef(rc.x, rb.x, delta_of<FACE_OWN>(w.x)), coef(rc.y, rb.y, delta_of<FACE_OWN>(w.y)),
                         coef(rc.z, rb.z, delta_of<FACE_OWN>(w.z)), coef(rc.w, rb.w, delta_of<FACE_OWN>(w.w)));
    } else {
        cB = make_float4(coef(rc.x, rb.x, delta_of<FACE_F>(wb.x)), coef(rc.y, rb.y, delta_of<FACE_F>(wb.y)),
                         coef(rc.z, rb.z, delta_of<FACE_F>(wb.z)), coef(rc.w, rb.w, delta_of<FACE_F>(wb.w)));
    }
    bool stuck = false;
    for (int z = zs; z < ze; ++z) {
        float4 vf = f4zero(), rf = rc;
        const float* d1 = d0;
        if (z + 1 < Z) {
            d1 = wait_plane(z + 1);
            vf = dir4(d1, own);
            rf = rho4(d1, own);
        }
        if (y < Y) {
            const float4 vd = dir4(d0, own - OPW), rd = rho4(d0, own - OPW), vu = dir4(d0, own + OPW);
            const float4 ru = top ? rc : rho4(d0, own + OPW);
            const uint4 w = word4(d0, own), wd4 = word4(d0, own - OPW);
            const unsigned wl = reinterpret_cast<const unsigned*>(d0 + 3 * OPBOX)[own - 1];
            const float sl = dir1(d0, own - 1), sr = rend ? 0.0f : dir1(d0, own + 4);
            const float rl = lend ? rc.x : d0[2 * OPBOX + own - 1], rr = rend ? rc.w : d0[2 * OPBOX + own + 4];
            const float4 cR = make_float4(coef(rc.x, rc.y, delta_of<FACE_R>(w.x)), coef(rc.y, rc.z, delta_of<FACE_R>(w.y)),
                                          coef(rc.z, rc.w, delta_of<FACE_R>(w.z)), coef(rc.w, rr, delta_of<FACE_R>(w.w)));
            const float cl = coef(rc.x, rl, lend ? delta_of<FACE_OWN>(w.x) : delta_of<FACE_R>(wl));
            auto cell = [&](float v, float r, unsigned wo, float vl, float cL, unsigned wL, float vr, float cr, float vdn, float rdn,
                            unsigned wD, float vup, float rup, float vbk, float& cb, unsigned wB, float vfr, float rfr) {
                const float cU = coef(r, rup, delta_of<FACE_U>(wo)), cF = coef(r, rfr, delta_of<FACE_F>(wo));
                const float cD = below ? coef(r, rdn, delta_of<FACE_U>(wD)) : 0.0f;
                float wd = 0.0f;
                wd -= cr; wd -= cL; wd -= cU; wd -= cD; wd -= cF; wd -= cb;
                const float aL = REF ? trunc_of<0>(wL) : cL, aD = REF ? trunc_of<1>(wD) : cD, aB = REF ? trunc_of<2>(wB) : cb;
                cb = cF;
                return wd * v + ((aL * vl + aD * vdn + aB * vbk + cr * vr + cU * vup + cF * vfr));
            };
            float4 o;
            o.x = cell(vc.x, rc.x, w.x, sl, cl, wl, vc.y, cR.x, vd.x, rd.x, wd4.x, vu.x, ru.x, vb.x, cB.x, wb.x, vf.x, rf.x);
            o.y = cell(vc.y, rc.y, w.y, vc.x, cR.x, w.x, vc.z, cR.y, vd.y, rd.y, wd4.y, vu.y, ru.y, vb.y, cB.y, wb.y, vf.y, rf.y);
            o.z = cell(vc.z, rc.z, w.z, vc.y, cR.y, w.y, vc.w, cR.z, vd.z, rd.z, wd4.z, vu.z, ru.z, vb.z, cB.z, wb.z, vf.z, rf.z);
            o.w = cell(vc.w, rc.w, w.w, vc.z, cR.z, w.z, sr, cR.w, vd.w, rd.w, wd4.w, vu.w, ru.w, vb.w, cB.w, wb.w, vf.w, rf.w);
            if (FLAT) {
                if (y == 0) o = f4zero();
            } else {
                if (rc.x == 0.0f) o.x = 0.0f;
                if (rc.y == 0.0f) o.y = 0.0f;
                if (rc.z == 0.0f) o.z = 0.0f;
                if (rc.w == 0.0f) o.w = 0.0f;
            }
            if (act) {
                const int c = x0 + y * X + z * XY;
                *reinterpret_cast<float4*>(snew + c) = vc;
                *reinterpret_cast<float4*>(As + c) = o;
                acc.add(o.x * vc.x);
                acc.add(o.y * vc.y);
                acc.add(o.z * vc.z);
                acc.add(o.w * vc.w);
            }
            wb = w;
        }
        vb = vc;
        vc = vf;
        rc = rf;
        d0 = d1;
        // every warp has read plane z: its slot takes the plane OPSLOTS further (a stuck copy stops the block)
        if (__syncthreads_or(!ok)) {
            stuck = true;
            break;
        }
        if (tid == 0)
            for (; issued <= p1 && issued - OPSLOTS <= z; ++issued) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue(issued);
            }
    }
    if (stuck) {
        // record the timeout, then let the copies still in flight land before the block's shared memory
        // goes away (each wait again bounded); the block's partial is still published, so that the
        // reduction ends
        if (tid == 0) {
            sc->status = SKT_TIMEOUT;
            for (int q = max(issued - OPSLOTS, p0); q < issued; ++q)
                (void)mbar_wait(&bar[(q - p0) % OPSLOTS], unsigned((q - p0) / OPSLOTS) & 1u);
        }
        __syncthreads();
    }
    double tot;
    float mall;
    if (grid_sum_max<OPT, false>(sc, partials, linear_block(), linear_blocks(), tid, acc.sum(), 0.0f, tot, mall)) {
        const double s1 = REF ? sc->sigma1 + tot : tot;
        sc->sigma1 = s1;
        sc->alpha = float(sc->sigma0 / s1);
        sc->alpha_of[slot] = sc->alpha;
    }
}

// r -= alpha As, z = r/diag (stored), z.r and the max residual: k_update4 without the pressure
// update, which k_pressure4 applies. It runs through the cells
// backwards: the operator left the end of As and of the diagonal in L2, and finds the start of z there.
__global__ void __launch_bounds__(UT) k_residual4(int n4, int xy4, const float4* __restrict__ aw, const float4* __restrict__ As,
                                                  float4* __restrict__ r, float4* __restrict__ zout, int reference, float tol,
                                                  int max_iter, Scalars* sc, double* partials) {
    if (sc->converged) return;
    const float alpha = sc->alpha;
    Kahan acc;
    float mx = 0.0f;
    for (int i = n4 - 1 - (blockIdx.x * UT + threadIdx.x); i >= 0; i -= gridDim.x * UT) {
        const float4 a = aw[i], av = As[i];
        float4 rv = r[i];
        rv.x = rv.x - alpha * av.x; rv.y = rv.y - alpha * av.y; rv.z = rv.z - alpha * av.z; rv.w = rv.w - alpha * av.w;
        r[i] = rv;
        const float z0 = rv.x * precon_of(a.x), z1 = rv.y * precon_of(a.y), z2 = rv.z * precon_of(a.z), z3 = rv.w * precon_of(a.w);
        zout[i] = make_float4(z0, z1, z2, z3);
        acc.add(z0 * rv.x);
        acc.add(z1 * rv.y);
        acc.add(z2 * rv.z);
        acc.add(z3 * rv.w);
        const bool absv = !reference || i < xy4;  // the reference takes |r| on the z = 0 plane only (Q4)
        const float m0 = absv ? fabsf(rv.x) : rv.x, m1 = absv ? fabsf(rv.y) : rv.y;
        const float m2 = absv ? fabsf(rv.z) : rv.z, m3 = absv ? fabsf(rv.w) : rv.w;
        if (m0 > mx) mx = m0;
        if (m1 > mx) mx = m1;
        if (m2 > mx) mx = m2;
        if (m3 > mx) mx = m3;
    }
    double tot;
    float mall;
    if (grid_sum_max<UT, false>(sc, partials, blockIdx.x, gridDim.x, threadIdx.x, acc.sum(), mx, tot, mall)) {
        sc->iters += 1;
        sc->residual = mall;
        if (mall <= tol) {
            sc->converged = 1;
        } else if (sc->iters >= max_iter) {
            sc->converged = 2;
        } else {
            sc->sigma1 = tot;
            sc->beta_f = float(tot / sc->sigma0);
            sc->sigma0 = tot;
        }
    }
}

// The pressure updates p += alpha s (updatePandDiv :955-985), four iterations' at a time and in their
// order: before the iteration that overwrites the oldest direction (TAIL false), and after the last one
// to four (TAIL). The pressure is read and written once for four iterations, 6 bytes a cell and
// iteration instead of 8 and none of them in the operator.
template <bool TAIL>
__global__ void __launch_bounds__(UT) k_pressure4(int n4, Dirs dirs, float4* __restrict__ pp, const Scalars* sc) {
    if (!TAIL && sc->converged) return;  // the tail does these too
    const int it = sc->iters;
    if (it <= 0) return;
    const int n = TAIL ? it - (it - 1) / kDirs * kDirs : kDirs;
    float al[kDirs];
#pragma unroll
    for (int j = 0; j < kDirs; ++j) al[j] = sc->alpha_of[j];
    for (int i = blockIdx.x * UT + threadIdx.x; i < n4; i += gridDim.x * UT) {
        float4 pv = pp[i];
#pragma unroll
        for (int j = 0; j < kDirs; ++j) {
            if (TAIL && j >= n) break;
            const float4 sv = reinterpret_cast<const float4*>(dirs.d[j])[i];
            pv.x = __fmaf_rn(al[j], sv.x, pv.x);
            pv.y = __fmaf_rn(al[j], sv.y, pv.y);
            pv.z = __fmaf_rn(al[j], sv.z, pv.z);
            pv.w = __fmaf_rn(al[j], sv.w, pv.w);
        }
        pp[i] = pv;
    }
}

// graph mode, PCG loop: run (another) chunk of iterations while the solver has not stopped and no
// NaN was met; loop >= 0 counts a completed trip
__global__ void k_pcg_cond(cudaGraphConditionalHandle h, Scalars* sc, int loop) {
    if (loop >= 0) note_trip(sc, loop);
    cudaGraphSetConditional(h, (sc->converged == 0 && sc->status == 0) ? 1u : 0u);
}

// ---- the whole PCG in one launch (grids whose solver state fits the chip) ---------------------
// One cooperative launch of at most one 512-thread block per SM runs every iteration. A block owns
// K*512 consecutive cells; thread t holds cells t, t+512, ...: r, the pressure, the diagonal and
// the direction in registers, the six face coefficients (the lower ones truncated as Q3 wants, 0
// where there is no neighbour) in shared memory. Only the direction's halo crosses blocks: as in
// k_pcg_operator4 every block forms s_new = z + beta s_old for itself and, outside its own cells,
// from the neighbours' z and s_old in global memory (L2), so an iteration needs two grid-wide
// reductions and no third barrier. Each reduction is its own barrier: a block publishes its partial
// and arrives, waits until all have arrived, and sums all partials in the same order, so every
// block holds the same step lengths and takes the same decisions.
// What bounds it: the two exchanges of an iteration (2 to 3 us together, the second behind a fence for
// the direction's halo) and the block's own loads and sums. Measured per iteration, with streaming launches
// (two, or three for 90x51x75) and in one: 32^3 12.7 and 5.3 us, 64x32x64 14 and 6.9 us, 90x51x75 27 and
// 9.4 us, 128x64x128 30 and 12.5 us. Sums in pairs of floats, FP32's range and products: 4.8, 7.2, 8.8 and
// 12.9 us; FP64 trees and divisions in their place 5.5 at 32^3, exact products tested one by one 10.6 at
// 90x51x75.
// The cells of a thread depend on the grid's size alone, so a member of an ensemble gets the bits
// of the same grid alone. Every wait is bounded; one that runs out makes the block return and
// SKT_TIMEOUT be recorded (the other blocks' waits then run out too).
constexpr int GCT = 512;                      // threads per block
constexpr int kGridCells[4] = {2, 4, 8, 14};  // cells per thread of the variants (14: 200 KB of shared memory)
constexpr unsigned kGridSpinLimit = 1u << 21;
constexpr int kMaxGridBlocks = 256;           // blocks of the launch at most
template <int K>
int pcg_grid_smem(int X) { return (7 * K * GCT + 2 * X) * 4; }

// one block's partial of a reduction: its sum (Fixed's number), its maximum, and in one word the low 20 bits of
// the reduction's tag and the sum's unit; read and written as one 16-byte access so that a reader that sees
// the tag has the values with it
struct alignas(16) GridPart {
    long long v;
    float mx;
    unsigned word;
};
__device__ __forceinline__ unsigned part_word(unsigned tag, int u) { return tag << 12 | unsigned(u + 2048); }
__device__ __forceinline__ void put_part(GridPart* p, long long v, float mx, unsigned word) {
    asm volatile("{\n\t.reg .b64 hi;\n\t.reg .b128 v;\n\tmov.b64 hi, {%2, %3};\n\tmov.b128 v, {%1, hi};\n\t"
                 "st.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p), "l"(v), "f"(mx), "r"(word) : "memory");
}
__device__ __forceinline__ GridPart get_part(const GridPart* p) {
    GridPart r;
    asm volatile("{\n\t.reg .b64 hi;\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%3];\n\tmov.b128 {%0, hi}, v;\n\t"
                 "mov.b64 {%1, %2}, hi;\n\t}" : "=l"(r.v), "=f"(r.mx), "=r"(r.word) : "l"(p) : "memory");
    return r;
}

// (fence.acq_rel, not __threadfence, which is the sequentially consistent fence and slower)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// what the threads of a block share of the solver's scalars; thread 0 writes between a reduction's barriers
enum GridState { GRID_GO, GRID_DONE, GRID_CAP, GRID_NAN, GRID_STUCK, GRID_FAR };
struct GridScalars {
    double sigma0, sigma1;  // the dot products of the last iteration
    float len, residual;    // the step length that the last reduction gave, the last max residual
    int state;
};

// Reduces sum and maximum over the grid; a barrier too: every block writes its partial into every
// block's inbox and waits for all partials in its own, one hop through L2 (1.5 us for 128 blocks,
// 1.1 for 32; an arrival counter and then the partials 1.8 and 1.6, one block that sums for all 2.3
// and 1.4, every block polling one set of partials 2.9 and 1.2). The partials are summed in the same
// order everywhere, so every block gets the same totals; its first warp forms the step length from
// them in fin(total, maximum, whether no wait ran out), one lane of which stores. The FP64 work is the
// polling warps' and the first one's alone. THIRD: sums of Sum::add_near; FAR: sums of Sum::add_far. FENCE: the block's stores before the reduction are visible to
// every block after it. Inboxes alternate by the tag's parity: a block may send the next partial while
// another still reads these, but not the one after that.
template <bool FENCE, bool THIRD, bool FAR, class Fin>
__device__ __forceinline__ void grid_reduce(GridPart* inbox, int nb, unsigned tag, const Sum& sum, float mx, Fin fin) {
    constexpr int W = GCT / 32, B = kMaxGridBlocks / 32;
    __shared__ int4 ws[W];
    __shared__ float wm[W], tm[B];
    __shared__ double wf[FAR ? W : 1], ts[B];
    __shared__ int tk[B];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, par = tag & 1u, nw = (nb + 31) >> 5;
    {
        const WarpSum v = warp_sum<THIRD>(sum);
        const float m = warp_max(mx);
        const double f = FAR ? warp_far(sum.far) : 0.0;
        if (lane == 0) {
            ws[warp] = make_int4(v.a, v.b, v.c, int(v.e));
            wm[warp] = m;
            if (FAR) wf[warp] = f;
        }
    }
    __syncthreads();
    double tot = 0.0;
    float mall = 0.0f;
    bool ok = true;
    if (warp < nw) {
        const Fixed s = warps_total<log2_of(W), FAR>(ws, wf, lane);
        const float m = warp_max(lane < W ? wm[lane % W] : 0.0f);
        if (FENCE) fence_gpu();
        GridPart v{0, 0.0f, part_word(tag, -2048)};
        if (tid < nb) {
            put_part(inbox + (size_t(par) * nb + tid) * nb + blockIdx.x, s.v, m, part_word(tag, s.u));
            const GridPart* const mine = inbox + (size_t(par) * nb + blockIdx.x) * nb + tid;
            v = get_part(mine);
            for (unsigned i = 0; (v.word ^ tag << 12) >> 12 && ok; ++i) {
                ok = i < kGridSpinLimit;
                v = get_part(mine);
            }
        }
        if (FENCE) fence_gpu();
        tot = value(lanes_total<5>(Fixed{v.v, int(v.word & 0xfffu) - 2048}));
        mall = warp_max(v.mx);
        ok = __all_sync(0xffffffffu, ok);
    }
    if (nw > 1) {
        if (warp < nw && lane == 0) {
            ts[warp] = tot;
            tm[warp] = mall;
            tk[warp] = ok;
        }
        __syncthreads();
        if (warp == 0) {
            const bool in = lane < nw;
            tot = in ? ts[in ? lane : 0] : 0.0;
            for (int o = 1; o < nw; o <<= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            mall = warp_max(in ? tm[in ? lane : 0] : 0.0f);
            ok = __all_sync(0xffffffffu, !in || tk[in ? lane : 0]);
        }
    }
    if (warp == 0) fin(tot, mall, ok);
    __syncthreads();
}

// EXACT: the dot products' terms as k_matvec and k_update take them (X % 4 != 0), exact products summed to
// FP64's precision; otherwise as k_matvec4 and k_update4 do, FP32 products summed with compensation.
template <int K, bool EXACT>
__global__ void __launch_bounds__(GCT, 1) k_pcg_grid(Grid g, const float* __restrict__ ax, const float* __restrict__ ay,
                                                     const float* __restrict__ az, const float* __restrict__ aw, float* __restrict__ rg,
                                                     float* s_even, float* s_odd, float* zg, float* __restrict__ pg, int reference,
                                                     float tol, int max_iter, Scalars* sc, GridPart* inbox) {
    extern __shared__ float pcg_smem[];
    constexpr int LEN = K * GCT;
    float* const C = pcg_smem;  // the six face coefficients
    float* const S = pcg_smem + 6 * LEN + g.X;  // the direction with a row's halo on either side; between the phases z
    if (sc->converged) return;  // the setup found a zero residual
    const int tid = threadIdx.x, nb = gridDim.x, X = g.X, XY = g.XY, N = g.N;
    const int base = blockIdx.x * LEN;
    unsigned tag = sc->grid_tag;
    float r[K], p[K], w[K], s[K];  // (14 cells: some spill; the pressure in global memory instead was slower, 13.8 against 12.9 us)
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int l = tid + k * GCT, i = base + l;
        float cl = 0.0f, cr = 0.0f, cd = 0.0f, cu = 0.0f, cb = 0.0f, cf = 0.0f;
        r[k] = p[k] = w[k] = s[k] = 0.0f;
        if (i < N) {
            const int z = i / XY, xy = i - z * XY, y = xy / X, x = xy - y * X;
            if (x > 0) cl = ax[i - 1];
            if (x + 1 < X) cr = ax[i];
            if (y > 0) cd = ay[i - X];
            if (y + 1 < g.Y) cu = ay[i];
            if (z > 0) cb = az[i - XY];
            if (z + 1 < g.Z) cf = az[i];
            if (reference) { cl = char_trunc(cl); cd = char_trunc(cd); cb = char_trunc(cb); }
            r[k] = rg[i];
            w[k] = aw[i];
            s[k] = s_even[i];
        }
        C[l] = cl; C[LEN + l] = cr; C[2 * LEN + l] = cd; C[3 * LEN + l] = cu; C[4 * LEN + l] = cb; C[5 * LEN + l] = cf;
    }
    __shared__ GridScalars G;
    if (tid == 0) {
        G.sigma0 = sc->sigma0;
        G.sigma1 = sc->sigma1;
        G.residual = sc->residual;
    }
    float alpha = 0.0f, beta = 0.0f;
    int iters = 0;
    const bool whole = base + LEN <= N, inner = base >= XY && base + LEN + XY <= N;
    for (;;) {
        // the first direction is the setup's z itself: z + 0 times itself
        float* const snew = (iters & 1) ? s_odd : s_even;
        const float* const sold = iters == 0 ? s_even : ((iters & 1) ? s_even : s_odd);
        const float* const zold = iters == 0 ? s_even : zg;
        // outside the block's cells the direction is formed from global memory: the planes before and
        // behind for every cell (no test whether one lies inside), the rows above and below and the x
        // neighbours from the halo. A neighbour that does not exist has coefficient 0: its index is
        // clamped into the grid, which only the blocks at the grid's ends have to do.
        auto form = [&](int j) { return __fmaf_rn(beta, __ldcg(sold + j), __ldcg(zold + j)); };
        auto clamped = [&](int j) { return min(max(j, 0), N - 1); };
        float sb[K], sf[K];
        if (inner) {
            const float *so = sold + base + tid, *zo = zold + base + tid;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                sb[k] = __fmaf_rn(beta, __ldcg(so - XY + k * GCT), __ldcg(zo - XY + k * GCT));
                sf[k] = __fmaf_rn(beta, __ldcg(so + XY + k * GCT), __ldcg(zo + XY + k * GCT));
            }
        } else {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                sb[k] = form(clamped(base + tid + k * GCT - XY));
                sf[k] = form(clamped(base + tid + k * GCT + XY));
            }
        }
        for (int h = tid; h < 2 * X; h += GCT) {
            const int l = h < X ? h - X : LEN + h - X;
            S[l] = form(clamped(base + l));
        }
        float* const sn = snew + base + tid;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int l = tid + k * GCT;
            if (iters > 0) {
                s[k] = __fmaf_rn(beta, s[k], S[l]);
                if (whole || base + l < N) __stcg(sn + k * GCT, s[k]);
            }
            S[l] = s[k];
        }
        __syncthreads();
        float As[K];
        Kahan acc;
        Sum exact;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int l = tid + k * GCT;
            const float o = w[k] * s[k] + ((C[l] * S[l - 1] + C[2 * LEN + l] * S[l - X] + C[4 * LEN + l] * sb[k] + C[LEN + l] * S[l + 1] +
                                            C[3 * LEN + l] * S[l + X] + C[5 * LEN + l] * sf[k]));
            As[k] = o;
            if (!EXACT) acc.add(o * s[k]);
        }
        if (EXACT) exact.add_near(As, s);
        // (no fence: the next reads of another block's stores come after the second reduction)
        auto operator_done = [&](double tot, float, bool ok, bool again) {
            const double s1 = reference ? G.sigma1 + tot : tot;  // Q1
            const float a = quotient(G.sigma0, s1);
            __syncwarp();
            if (tid == 0) {
                G.state = !ok ? GRID_STUCK : again && !Sum::total_holds(tot) ? GRID_FAR : !isfinite(tot) ? GRID_NAN : GRID_GO;
                if (G.state != GRID_FAR) G.sigma1 = s1;
                G.len = a;
            }
        };
        grid_reduce<false, EXACT, false>(inbox, nb, ++tag, EXACT ? exact : acc.sum(), 0.0f,
                                         [&](double tot, float m, bool ok) { operator_done(tot, m, ok, EXACT); });
        if (EXACT && G.state == GRID_FAR) {  // the same for every block
            Sum far;
            far.add_far(As, s);
            grid_reduce<false, false, true>(inbox, nb, ++tag, far, 0.0f, [&](double tot, float m, bool ok) { operator_done(tot, m, ok, false); });
        }
        if (G.state != GRID_GO) break;
        alpha = G.len;
        Kahan zr;
        Sum zx;
        float zs[K], mx = 0.0f;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int l = tid + k * GCT, i = base + l;
            p[k] = __fmaf_rn(alpha, s[k], p[k]);
            r[k] = r[k] - alpha * As[k];
            const float z = r[k] * precon_of(w[k]);
            S[l] = z;  // every read of the direction lies before the reduction's barrier
            if (whole || i < N) __stcg(zg + base + tid + k * GCT, z);
            if (EXACT) zs[k] = z;
            else zr.add(z * r[k]);
            const float m = (!reference || i < XY) ? fabsf(r[k]) : r[k];  // Q4
            if (m > mx) mx = m;
        }
        if (EXACT) zx.add_near(zs, r);
        auto residual_done = [&](double tot, float mall, bool ok, bool again) {
            const float b = quotient(tot, G.sigma0);
            __syncwarp();
            if (tid == 0) {
                G.state = !ok ? GRID_STUCK : again && !Sum::total_holds(tot) ? GRID_FAR : !isfinite(tot) ? GRID_NAN : mall <= tol ? GRID_DONE
                          : iters + 1 >= max_iter ? GRID_CAP : GRID_GO;
                if (G.state != GRID_FAR) G.sigma0 = G.sigma1 = tot;
                G.len = b;
                G.residual = mall;
            }
        };
        grid_reduce<true, EXACT, false>(inbox, nb, ++tag, EXACT ? zx : zr.sum(), mx,
                                        [&](double tot, float m, bool ok) { residual_done(tot, m, ok, EXACT); });
        if (EXACT && G.state == GRID_FAR) {
            Sum far;
            far.add_far(zs, r);
            grid_reduce<true, false, true>(inbox, nb, ++tag, far, mx, [&](double tot, float m, bool ok) { residual_done(tot, m, ok, false); });
        }
        if (G.state == GRID_STUCK) break;
        ++iters;
        beta = G.len;
        if (G.state != GRID_GO) break;
    }
    const int state = G.state;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = base + tid + k * GCT;
        if (i < N) {
            rg[i] = r[k];
            pg[i] = p[k];
        }
    }
    if (tid == 0) {
        if (state == GRID_STUCK) sc->status = SKT_TIMEOUT;
        if (blockIdx.x == 0) {
            if (state == GRID_NAN) sc->status = SKT_NAN_DETECTED;
            sc->alpha = alpha;
            sc->beta_f = beta;
            sc->residual = G.residual;
            sc->iters = iters;
            sc->converged = state == GRID_DONE ? 1 : state == GRID_CAP ? 2 : 0;
            sc->grid_tag = tag_after(tag, state == GRID_STUCK);
        }
    }
}

// k_build for flat terrain and X % 4 == 0: four cells per thread, a march along z in blocks of
// MVY rows. Each cell's reciprocal density is formed once (the x neighbours' by shuffle, the next
// plane's carried), and each face once: a cell forms its right, up and front faces; the left face
// is the right face of the cell before (a shuffle across lanes), the back face the front face of
// the previous plane, the down face is formed again from the row below. coef_of and the harmonic
// mean are symmetric in their two densities (IEEE addition commutes), so every value equals
// k_build's; z.r is summed in a different order.
__device__ __forceinline__ float fcomp(const float4& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w)); }
__device__ __forceinline__ void fset(float4& v, int k, float a) {
    if (k == 0) v.x = a; else if (k == 1) v.y = a; else if (k == 2) v.z = a; else v.w = a;
}
__device__ __forceinline__ void face_of(float c, float rc, float n, float rn, float& h, float& coef) {
    // hm(n) = 2/(1/c + 1/n) and coef_of(c, n), both 0 across a zero density
    if (n == 0.0f) { h = 0.0f; coef = 0.0f; return; }
    h = 2.0f / (rc + rn);
    coef = -fmaxf(1.0f, 1.225f / h);
    (void)c;
}
// FACES: the three face coefficients are stored; otherwise, in the places of the first two,
// what k_pcg_operator4 reads: the reciprocal densities and the words of pack_faces.
template <bool FACES>
__global__ void __launch_bounds__(MVT) k_build4(Grid g, int zlen, const float* __restrict__ rho, const float* __restrict__ u,
                                                const float* __restrict__ v, const float* __restrict__ w,
                                                const float* __restrict__ defU, const float* __restrict__ defW, float dt,
                                                float* __restrict__ ax, float* __restrict__ ay, float* __restrict__ az,
                                                float* __restrict__ aw, float* __restrict__ r, float* __restrict__ s,
                                                float* __restrict__ pp, float* __restrict__ As, int reference, Scalars* sc,
                                                double* partials) {
    const int lane = threadIdx.x, tid = threadIdx.x + 32 * threadIdx.y;
    const int x0 = (blockIdx.x * 32 + lane) * 4;
    const int y = blockIdx.y * MVY + threadIdx.y;
    const int zs = blockIdx.z * zlen, ze = min(zs + zlen, g.Z);
    const bool act = x0 < g.X && y < g.Y;
    const bool sky = act && y >= 1;
    const int X = g.X, XY = g.XY, Z = g.Z;
    const int row = x0 + y * X;
    const float4 z4 = make_float4(0, 0, 0, 0);
    Sum dsum;
    float mx = 0.0f;
    const float du_ = sky ? defU[y] : 0.0f, dw_ = sky ? defW[y] : 0.0f;
    // own plane: density and reciprocal; the back face (front face of the plane before) and w there
    float4 pc = z4, rc = z4, hB = z4, cB = z4, wB = z4;
    if (sky) {
        pc = ld4(rho, row + zs * XY);
        rc = make_float4(1.0f / pc.x, 1.0f / pc.y, 1.0f / pc.z, 1.0f / pc.w);
        float4 pb = pc, rb = rc;  // outside at z = 0: the own density (NEUMANN)
        if (zs > 0) {
            pb = ld4(rho, row + (zs - 1) * XY);
            rb = make_float4(1.0f / pb.x, 1.0f / pb.y, 1.0f / pb.z, 1.0f / pb.w);
            wB = ld4(w, row + (zs - 1) * XY);
        } else {
            wB = make_float4(dw_, dw_, dw_, dw_);
        }
        face_of(pc.x, rc.x, pb.x, rb.x, hB.x, cB.x);
        face_of(pc.y, rc.y, pb.y, rb.y, hB.y, cB.y);
        face_of(pc.z, rc.z, pb.z, rb.z, hB.z, cB.z);
        face_of(pc.w, rc.w, pb.w, rb.w, hB.w, cB.w);
    }
    for (int z = zs; z < ze; ++z) {
        const int c = row + z * XY;
        float4 pf = pc, rf = rc, pd = z4, rd = z4, pu = pc, ru = rc, uo = z4, vo = z4, wo = z4, vd = z4;
        if (sky) {
            if (z + 1 < Z) {
                pf = ld4(rho, c + XY);
                rf = make_float4(1.0f / pf.x, 1.0f / pf.y, 1.0f / pf.z, 1.0f / pf.w);
            }
            if (y > 1) {  // the row below (y = 1 has the ground below: density 0, v 0)
                pd = ld4(rho, c - X);
                rd = make_float4(1.0f / pd.x, 1.0f / pd.y, 1.0f / pd.z, 1.0f / pd.w);
                vd = ld4(v, c - X);
            }
            if (y + 1 < g.Y) {
                pu = ld4(rho, c + X);
                ru = make_float4(1.0f / pu.x, 1.0f / pu.y, 1.0f / pu.z, 1.0f / pu.w);
            }
            uo = ld4(u, c);
            vo = ld4(v, c);
            wo = ld4(w, c);
        }
        // the right neighbour of the last cell and the left neighbour of the first
        float pr = __shfl_down_sync(0xffffffffu, pc.x, 1), rr = __shfl_down_sync(0xffffffffu, rc.x, 1);
        float ul = __shfl_up_sync(0xffffffffu, uo.w, 1);
        if (sky && (lane == 31 || x0 + 4 >= X)) {
            if (x0 + 4 < X) { pr = rho[c + 4]; rr = 1.0f / pr; }
            else { pr = pc.w; rr = rc.w; }  // outside: the own density (NEUMANN)
        }
        float hR[4], cR[4];
        face_of(pc.x, rc.x, pc.y, rc.y, hR[0], cR[0]);
        face_of(pc.y, rc.y, pc.z, rc.z, hR[1], cR[1]);
        face_of(pc.z, rc.z, pc.w, rc.w, hR[2], cR[2]);
        face_of(pc.w, rc.w, pr, rr, hR[3], cR[3]);
        float hL0 = __shfl_up_sync(0xffffffffu, hR[3], 1), cL0 = __shfl_up_sync(0xffffffffu, cR[3], 1);
        if (sky && lane == 0) {
            float pl = pc.x, rl = rc.x;
            if (x0 > 0) { pl = rho[c - 1]; rl = 1.0f / pl; ul = u[c - 1]; }
            else ul = du_;
            face_of(pc.x, rc.x, pl, rl, hL0, cL0);
        }
        if (sky) {
            const float hL[4] = {hL0, hR[0], hR[1], hR[2]}, cL[4] = {cL0, cR[0], cR[1], cR[2]};
            const float uL[4] = {ul, uo.x, uo.y, uo.z};
            float4 oax, oay, oaz, oaw, orr, oss;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float cur = fcomp(pc, k);
                float hU, cU, hD, cD, hF, cF;
                face_of(cur, fcomp(rc, k), fcomp(pu, k), fcomp(ru, k), hU, cU);
                face_of(cur, fcomp(rc, k), fcomp(pd, k), fcomp(rd, k), hD, cD);
                face_of(cur, fcomp(rc, k), fcomp(pf, k), fcomp(rf, k), hF, cF);
                float wd = 0.0f;
                wd -= cR[k]; wd -= cL[k]; wd -= cU; wd -= cD; wd -= cF; wd -= fcomp(cB, k);
                const float mfd = ((hR[k] * fcomp(uo, k) - hL[k] * uL[k]) + (hU * fcomp(vo, k) - hD * fcomp(vd, k)) +
                                   (hF * fcomp(wo, k) - fcomp(hB, k) * fcomp(wB, k)));
                const float dch = (cur - cur) / dt;  // the reference's old density is a copy of rho
                const float rv = mfd - dch;
                const float zv = rv * precon_of(wd);
                fset(oax, k, cR[k]); fset(oay, k, cU); fset(oaz, k, cF); fset(oaw, k, wd);
                fset(orr, k, rv); fset(oss, k, zv);
                dsum.add_prod(zv, rv);
                const float m = (!reference || z == 0) ? fabsf(rv) : rv;
                if (m > mx) mx = m;
                fset(hB, k, hF); fset(cB, k, cF);
            }
            *reinterpret_cast<float4*>(ax + c) = FACES ? oax : rc;
            if (FACES) {
                *reinterpret_cast<float4*>(ay + c) = oay;
                *reinterpret_cast<float4*>(az + c) = oaz;
                *reinterpret_cast<float4*>(As + c) = z4;
            } else {
                *reinterpret_cast<uint4*>(ay + c) =
                    make_uint4(pack_faces(oax.x, oay.x, oaz.x, rc.x + rc.y, rc.x + ru.x, rc.x + rf.x, rc.x + rc.x),
                               pack_faces(oax.y, oay.y, oaz.y, rc.y + rc.z, rc.y + ru.y, rc.y + rf.y, rc.y + rc.y),
                               pack_faces(oax.z, oay.z, oaz.z, rc.z + rc.w, rc.z + ru.z, rc.z + rf.z, rc.z + rc.z),
                               pack_faces(oax.w, oay.w, oaz.w, rc.w + rr, rc.w + ru.w, rc.w + rf.w, rc.w + rc.w));
            }
            *reinterpret_cast<float4*>(aw + c) = oaw;
            *reinterpret_cast<float4*>(r + c) = orr;
            *reinterpret_cast<float4*>(s + c) = oss;
            *reinterpret_cast<float4*>(pp + c) = z4;
        } else if (act) {  // the ground row
            *reinterpret_cast<float4*>(ax + c) = z4;
            *reinterpret_cast<float4*>(ay + c) = z4;
            if (FACES) {
                *reinterpret_cast<float4*>(az + c) = z4;
                *reinterpret_cast<float4*>(As + c) = z4;
            }
            *reinterpret_cast<float4*>(aw + c) = z4;
            *reinterpret_cast<float4*>(r + c) = z4;
            *reinterpret_cast<float4*>(s + c) = z4;
            *reinterpret_cast<float4*>(pp + c) = z4;
        }
        pc = pf;
        rc = rf;
        wB = wo;
    }
    double tot;
    float mall;
    if (grid_sum_max<MVT, true>(sc, partials, linear_block(), linear_blocks(), tid, dsum, mx, tot, mall)) {
        sc->sigma0 = tot;
        sc->sigma1 = 0.0;
        sc->iters = 0;
        sc->residual = mall;
        sc->converged = (mall == 0.0f) ? 1 : 0;
    }
}

// updatePressure (:1016-1030) followed by initDensity (:1432-1452)
__global__ void __launch_bounds__(256) k_press_dens(Grid g, float* __restrict__ p, const float* __restrict__ pp, float* __restrict__ rho,
                                                    const float* __restrict__ th, const float* __restrict__ qv, const float* __restrict__ Pg) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z = blockIdx.z;
    if (x >= g.X || y >= g.Y) return;
    if (is_ground(g, x, y, z)) return;
    const int c = cidx(g, x, y, z);
    const float pn = p[c] - pp[c] / 100.0f;
    p[c] = pn;
    const float Tt = th[c] * powf(pn / Pg[x + z * g.X], KC::KAPPA);
    const float Tv = Tt * (0.608f * qv[c] + 1);
    rho[c] = pn * 100 / (KC::Rsd * Tv);
}

// applyPresProjGPU Game/kernelSky.cu:862-908 (pressure bounds DIRICHLET sides / NEUMANN ground,
// density bounds NEUMANN sides / DIRICHLET ground)
__global__ void __launch_bounds__(256) k_apply_proj(Grid g, const float* __restrict__ pp, const float* __restrict__ rho, float* __restrict__ u,
                                                    float* __restrict__ v, float* __restrict__ w) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z = blockIdx.z;
    if (x >= g.X || y >= g.Y) return;
    if (is_ground(g, x, y, z)) return;
    const int c = cidx(g, x, y, z);
    const float cp = pp[c], cd = rho[c];
    const float pr = face_nb(g, pp, x, y, z, 1, 0, 0, DIRICHLET, NEUMANN, 0.0f);
    const float pu = face_nb(g, pp, x, y, z, 0, 1, 0, DIRICHLET, NEUMANN, 0.0f);
    const float pf = face_nb(g, pp, x, y, z, 0, 0, 1, DIRICHLET, NEUMANN, 0.0f);
    float dr = face_nb(g, rho, x, y, z, 1, 0, 0, NEUMANN, DIRICHLET, 0.0f);
    float du = face_nb(g, rho, x, y, z, 0, 1, 0, NEUMANN, DIRICHLET, 0.0f);
    float df = face_nb(g, rho, x, y, z, 0, 0, 1, NEUMANN, DIRICHLET, 0.0f);
    dr = dr == 0.0f ? cd : 2.0f / (1.0f / cd + 1.0f / dr);
    du = du == 0.0f ? cd : 2.0f / (1.0f / cd + 1.0f / du);
    df = df == 0.0f ? cd : 2.0f / (1.0f / cd + 1.0f / df);
    u[c] += (pr - cp) / dr;
    v[c] += (pu - cp) / du;
    w[c] += (pf - cp) / df;
}

// k_apply_proj for flat terrain and X % 4 == 0: four cells per thread and a march along z over the
// sky rows (the next plane's pressure correction and density are the front neighbours and become
// the next step's own values); each cell's reciprocal density is formed once. Flat ground is
// the row y = 0, so the +x, +y and +z neighbours of a sky cell are never ground: outside the
// domain the correction is 0 (DIRICHLET) and the density the cell's own (NEUMANN). Same
// arithmetic as k_apply_proj.
__global__ void __launch_bounds__(256) k_apply_proj4(Grid g, int zlen, const float* __restrict__ pp, const float* __restrict__ rho,
                                                     float* __restrict__ u, float* __restrict__ v, float* __restrict__ w) {
    const int lane = threadIdx.x;
    const int x0 = (blockIdx.x * 32 + lane) * 4;
    const int y = blockIdx.y * 8 + threadIdx.y + 1;  // sky rows start at y = 1
    const int zs = blockIdx.z * zlen, ze = min(zs + zlen, g.Z);
    const bool act = x0 < g.X && y < g.Y;
    const int X = g.X, XY = g.XY;
    const int row = x0 + y * X;
    float4 pc = f4zero(), dc = f4zero();
    if (act) {
        pc = ld4(pp, row + zs * XY);
        dc = ld4(rho, row + zs * XY);
    }
    for (int z = zs; z < ze; ++z) {
        const int c = row + z * XY;
        float4 pf = f4zero(), df = dc, pu = f4zero(), du = dc;
        if (act) {
            if (z + 1 < g.Z) { pf = ld4(pp, c + XY); df = ld4(rho, c + XY); }
            if (y + 1 < g.Y) { pu = ld4(pp, c + X); du = ld4(rho, c + X); }
        }
        float pr3 = __shfl_down_sync(0xffffffffu, pc.x, 1), dr3 = __shfl_down_sync(0xffffffffu, dc.x, 1);
        if (act && (lane == 31 || x0 + 4 >= X)) {
            if (x0 + 4 < X) { pr3 = pp[c + 4]; dr3 = rho[c + 4]; }
            else { pr3 = 0.0f; dr3 = dc.w; }
        }
        if (act) {
            const float prx[4] = {pc.y, pc.z, pc.w, pr3}, drx[4] = {dc.y, dc.z, dc.w, dr3};
            float4 uo = ld4(u, c), vo = ld4(v, c), wo = ld4(w, c);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float cp = fcomp(pc, k), cd = fcomp(dc, k), rc = 1.0f / cd;
                float dr = drx[k], dU = fcomp(du, k), dF = fcomp(df, k);
                dr = dr == 0.0f ? cd : 2.0f / (rc + 1.0f / dr);
                dU = dU == 0.0f ? cd : 2.0f / (rc + 1.0f / dU);
                dF = dF == 0.0f ? cd : 2.0f / (rc + 1.0f / dF);
                fset(uo, k, fcomp(uo, k) + (prx[k] - cp) / dr);
                fset(vo, k, fcomp(vo, k) + (fcomp(pu, k) - cp) / dU);
                fset(wo, k, fcomp(wo, k) + (fcomp(pf, k) - cp) / dF);
            }
            *reinterpret_cast<float4*>(u + c) = uo;
            *reinterpret_cast<float4*>(v + c) = vo;
            *reinterpret_cast<float4*>(w + c) = wo;
        }
        pc = pf;
        dc = df;
    }
}

}  // namespace

namespace {

template <int K>
const void* pcg_grid_kernel(const Env& e) {
    return e.g.X % 4 != 0 ? (const void*)k_pcg_grid<K, true> : (const void*)k_pcg_grid<K, false>;
}
// whether the blocks of this launch are resident at once (asked once per environment and variant)
template <int K>
bool pcg_grid_fits(Env& e, int slot, int nb) {
    const int smem = pcg_grid_smem<K>(e.g.X);
    if (e.pcg_grid_cap[slot] < 0) {
        // the limit set on the kernel is the device's, not this grid's need: other environments launch it too
        int coop = 0, most = 0, per_sm = 0;
        cudaFuncAttributes fa{};
        const void* const kernel = pcg_grid_kernel<K>(e);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, e.device);
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, e.device);
        if (!coop || cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || smem + int(fa.sharedSizeBytes) > most ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - int(fa.sharedSizeBytes)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, GCT, smem) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 0;
        }
        e.pcg_grid_cap[slot] = per_sm * e.num_sms;
    }
    return nb <= e.pcg_grid_cap[slot];
}
template <int K>
void launch_pcg_grid(Env& e, int nb) {
    int reference = e.cfg.semantics == 0;
    void* args[] = {&e.g, &e.ax, &e.ay, &e.az, &e.aw, &e.r, &e.s, &e.tB, &e.tA, &e.pp, &reference, &e.cfg.pcg_tol, &e.cfg.pcg_max_iter,
                    &e.sc, &e.grid_parts};
    // an error is the step's to report (its check finds it)
    (void)cudaLaunchCooperativeKernel(pcg_grid_kernel<K>(e), dim3(nb), dim3(GCT), args, pcg_grid_smem<K>(e.g.X), e.stream);
    e.launches += 1;
}

// The launch shape for a grid: the variant with the fewest cells per thread that needs at most 96
// blocks (the reductions' exchange grows with the blocks: 64x32x64 took 7.5 us an iteration as 128
// blocks of 2 cells a thread, 7.0 as 64 of 4 and 7.6 as 32 of 8), else the fewest whose blocks fit
// one per SM (1.09M cells on 152 SMs); nb = 0 above that, where the solver state does not fit the
// SMs' registers and shared memory and two streaming launches per iteration are used instead.
void pcg_grid_shape(const Env& e, int& slot, int& nb) {
    for (const int most : {std::min(96, e.num_sms), std::min(e.num_sms, kMaxGridBlocks)})
        for (slot = 0; slot < 4; ++slot) {
            nb = blocks_for(e.g.N, kGridCells[slot] * GCT);
            if (nb <= most) return;
        }
    nb = 0;
}

// How the plain PCG runs: in one cooperative launch where the grid fits, else matrix-free in two
// launches per iteration (X % 4 == 0), else from stored coefficients in three (any X; pcg_fused = 0).
// Rows of less than 24 cells leave the matrix-free operator's warps, each across 128 cells of a row, too few
// lanes to form coefficients with (us an iteration matrix-free and stored at 2.1M cells: X = 4 250 and 152, 8 146
// and 100, 16 88 and 73; 1.8M cells, 20 68 and 64; 1.6M, 24 58 and 59; 1.9M, 48 47 and 53).
constexpr int kFreeMinX = 24;
enum class PcgPath { GRID, FREE, STORED };
PcgPath pcg_path(Env& e, int& slot, int& nb, OpMaps* maps, float* const* dirs, const float* zbuf) {
    pcg_grid_shape(e, slot, nb);
    if (!e.cfg.pcg_fused || e.cfg.pcg_max_iter <= 0) return PcgPath::STORED;
    if (nb > 0 && (slot == 0 ? pcg_grid_fits<2>(e, slot, nb) : slot == 1 ? pcg_grid_fits<4>(e, slot, nb)
                   : slot == 2 ? pcg_grid_fits<8>(e, slot, nb) : pcg_grid_fits<14>(e, slot, nb)))
        return PcgPath::GRID;
    if (e.g.X % 4 != 0 || e.g.X < kFreeMinX || (long long)((e.g.X + 127) / 128) * ((e.g.Y + OPR - 1) / OPR) > kMaxPartials) return PcgPath::STORED;
    // one set of tensor maps per direction buffer that an iteration reads; without an encoder: stored
    for (int j = 0; j < kDirs; ++j) {
        if (!field_tensor_map(e.g, zbuf, OPW, OPR + 2, &maps[j].z) || !field_tensor_map(e.g, dirs[j], OPW, OPR + 2, &maps[j].s) ||
            !field_tensor_map(e.g, e.ax, OPW, OPR + 2, &maps[j].r) || !field_tensor_map(e.g, e.ay, OPW, OPR + 2, &maps[j].w))
            return PcgPath::STORED;
    }
    return PcgPath::FREE;
}
// the operator's instance (its shared memory allowed)
template <bool FLAT, bool FIRST, bool REF>
auto pcg_operator_of() {
    cudaFuncSetAttribute(k_pcg_operator4<FLAT, FIRST, REF>, cudaFuncAttributeMaxDynamicSharedMemorySize, op_smem_bytes());
    return k_pcg_operator4<FLAT, FIRST, REF>;
}
template <bool FLAT>
auto pcg_operator(bool first, bool ref) {
    return first ? (ref ? pcg_operator_of<FLAT, true, true>() : pcg_operator_of<FLAT, true, false>())
                 : (ref ? pcg_operator_of<FLAT, false, true>() : pcg_operator_of<FLAT, false, false>());
}
// z runs of the operator: the fewest planes in a row on one SM (two blocks per SM at a time; a run reads
// a plane more on either side and fills its ring first), within the partials' storage
int operator_runs(const Env& e, int columns, int& zlen) {
    long long best = -1;
    int runs = 1;
    for (int zc = 1; zc <= e.g.Z && (long long)columns * zc <= kMaxPartials; ++zc) {
        const int len = (e.g.Z + zc - 1) / zc;
        const long long waves = ((long long)columns * zc + 2 * e.num_sms - 1) / (2 * e.num_sms), cost = waves * (len + 3);
        if (best < 0 || cost < best) {
            best = cost;
            runs = zc;
        }
    }
    zlen = (e.g.Z + runs - 1) / runs;
    return (e.g.Z + zlen - 1) / zlen;
}

}  // namespace

size_t pcg_grid_bytes(const Env& e) {
    int slot, nb;
    pcg_grid_shape(e, slot, nb);
    return e.cfg.precision == 1 ? 0 : sizeof(GridPart) * 2 * size_t(nb) * nb;
}

// As = A s and s.As -> alpha (textbook operator, vectorised; X % 4 == 0)
void launch_matvec_textbook(Env& e, const float* s, float* As) {
    const Grid& g = e.g;
    const dim3 mvb(32, MVY);
    const int gx = (g.X / 4 + 31) / 32, gy = (g.Y + MVY - 1) / MVY;
    int zc = std::max(1, std::min(g.Z, (e.num_sms * 8 + gx * gy - 1) / (gx * gy)));
    while (gx * gy * zc > kMaxPartials && zc > 1) --zc;
    const int zlen = (g.Z + zc - 1) / zc;
    zc = (g.Z + zlen - 1) / zlen;
    if (e.flat)
        k_matvec4<true><<<dim3(gx, gy, zc), mvb, 0, e.stream>>>(g, zlen, e.ax, e.ay, e.az, e.aw, s, As, 0, e.sc, e.partials);
    else
        k_matvec4<false><<<dim3(gx, gy, zc), mvb, 0, e.stream>>>(g, zlen, e.ax, e.ay, e.az, e.aw, s, As, 0, e.sc, e.partials);
    e.launches += 1;
}

void launch_project(Env& e, float dtS) {
    const Grid& g = e.g;
    const Tiles T = tiles_of(g);
    const int ref = e.cfg.semantics == 0;
    const int nblk = std::min(std::min(T.n, e.num_sms * 4), kMaxPartials);
    int slot = 0, gridblocks = 0;
    // matrix-free: z = r/diag in e.tA, the directions in the free fields (the advection's scratch and
    // the mixed solve's fields)
    float* zbuf = e.tA;
    float* dirs[kDirs] = {e.s, e.tB, reinterpret_cast<float*>(e.xd), reinterpret_cast<float*>(e.xd) + size_t(g.N)};
    OpMaps maps[kDirs];
    const PcgPath path = e.cfg.precision == 1 ? PcgPath::STORED : pcg_path(e, slot, gridblocks, maps, dirs, zbuf);
    const bool faces = path != PcgPath::FREE;
    {
    ProfScope ps(e, "proj_setup");
    e.launches += 2;
    if (e.flat) launch_next(e, k_reset_faces, far_faces(g.X, g.Y, g.Z) / 256u + 1u, 256, 0, g, e.u, e.v, e.w, e.defU, e.defW);
    else launch_next(e, k_reset_vel, (g.XY + 127) / 128, 128, 0, g, e.u, e.v, e.w, e.defU, e.defW, ref);
    float* z0 = faces ? e.s : zbuf;
    if (e.flat && (g.X % 4) == 0) {
        const int gx = (g.X / 4 + 31) / 32, gy = (g.Y + MVY - 1) / MVY;
        int zc = std::max(1, std::min(g.Z, (e.num_sms * 4 + gx * gy - 1) / (gx * gy)));
        while (gx * gy * zc > kMaxPartials && zc > 1) --zc;
        const int zlen = (g.Z + zc - 1) / zc;
        zc = (g.Z + zlen - 1) / zlen;
        const auto build = faces ? k_build4<true> : k_build4<false>;
        build<<<dim3(gx, gy, zc), dim3(32, MVY), 0, e.stream>>>(g, zlen, e.rho, e.u, e.v, e.w, e.defU, e.defW, dtS, e.ax, e.ay, e.az, e.aw,
                                                                e.r, z0, e.pp, e.As, ref, e.sc, e.partials);
    } else {
        k_build<<<nblk, NT, 0, e.stream>>>(g, T, e.rho, e.u, e.v, e.w, e.defU, e.defW, dtS, e.ax, e.ay, e.az, e.aw, e.r, z0, e.pp, e.As,
                                          faces, ref, e.sc, e.partials);
    }
    }
    if (e.cfg.precision == 1) {
        mg_solve(e);
    } else if (path == PcgPath::GRID) {
        {
            ProfScope ps(e, "pcg_grid");
            switch (slot) {
                case 0: launch_pcg_grid<2>(e, gridblocks); break;
                case 1: launch_pcg_grid<4>(e, gridblocks); break;
                case 2: launch_pcg_grid<8>(e, gridblocks); break;
                default: launch_pcg_grid<14>(e, gridblocks); break;
            }
        }
        if (!e.capturing) {
            fetch_scalars(e);
            e.last_iters = e.host_sc->iters;
            e.last_residual = e.host_sc->residual;
            e.last_converged = e.host_sc->converged == 1;
        }
    } else {
    const int chunk = 8;  // a multiple of kDirs: a chunk's iterations use the direction buffers as the chunk before
    const bool vec = (g.X % 4) == 0;
    // vectorised launch shapes: streams at 16 blocks/SM (several waves of the grid-stride loop:
    // 8 per SM, 1.3 waves, left the second wave a third full), the matvec's z chunks sized to fill
    // the GPU
    const int n4 = g.N / 4;
    const int nstream = std::min(std::min((n4 + UT - 1) / UT, e.num_sms * 16), kMaxPartials);
    const int nany = std::max(1, std::min(std::min((n4 + NT - 1) / NT, e.num_sms * 16), kMaxPartials));
    const Runs MT = matvec_runs(g, e.num_sms);
    const dim3 mvb(32, MVY);
    const int gx = (g.X / 4 + 31) / 32, gy = (g.Y + MVY - 1) / MVY;
    // k_matvec4 (pcg_fused = 0): about 4 blocks of 1024 threads per SM (one resident at a time), 251 us a launch
    // at 512x256x512 and 50.0 at 256x128x256; 6 blocks 256 and 51.8, 8 blocks 261 and 54.8, 12 blocks 266 and
    // 54.6, all four 20.6 to 20.7 at 128x100x128
    int zc = std::max(1, std::min(g.Z, (e.num_sms * 4 + gx * gy - 1) / (gx * gy)));
    while (gx * gy * zc > kMaxPartials && zc > 1) --zc;
    const int zlen = (g.Z + zc - 1) / zc;
    zc = (g.Z + zlen - 1) / zlen;
    const dim3 mvg(gx, gy, zc);
    const Dirs dp{{dirs[0], dirs[1], dirs[2], dirs[3]}};
    const int ox = (g.X + 127) / 128, oy = (g.Y + OPR - 1) / OPR;
    int ozlen;
    const dim3 og(ox, oy, operator_runs(e, ox * oy, ozlen));
    const auto op_first = e.flat ? pcg_operator<true>(true, ref) : pcg_operator<false>(true, ref);
    const auto op_next = e.flat ? pcg_operator<true>(false, ref) : pcg_operator<false>(false, ref);
    // iteration kk of the PCG (kk == 0: the first; others by their place in the chunks after it)
    auto iterate = [&](int kk) {
            if (path == PcgPath::FREE) {
                const int slot = kk % kDirs;
                if (slot == 0 && kk > 0) {
                    ProfScope ps(e, "pcg_update"); e.launches += 1;
                    k_pressure4<false><<<nstream, UT, 0, e.stream>>>(n4, dp, (float4*)e.pp, e.sc);
                }
                { ProfScope ps(e, "pcg_matvec"); e.launches += 1;
                  (kk == 0 ? op_first : op_next)<<<og, OPT, op_smem_bytes(), e.stream>>>(maps[(kk + kDirs - 1) % kDirs], g, ozlen, dirs[slot],
                                                                                       e.As, slot, e.sc, e.partials); }
                { ProfScope ps(e, "pcg_update"); e.launches += 1;
                  k_residual4<<<nstream, UT, 0, e.stream>>>(n4, g.XY / 4, (const float4*)e.aw, (const float4*)e.As, (float4*)e.r,
                                                            (float4*)zbuf, ref, e.cfg.pcg_tol, e.cfg.pcg_max_iter, e.sc, e.partials); }
            } else if (vec) {
                { ProfScope ps(e, "pcg_matvec"); e.launches += 1;
                  if (e.flat) k_matvec4<true><<<mvg, mvb, 0, e.stream>>>(g, zlen, e.ax, e.ay, e.az, e.aw, e.s, e.As, ref, e.sc, e.partials);
                  else k_matvec4<false><<<mvg, mvb, 0, e.stream>>>(g, zlen, e.ax, e.ay, e.az, e.aw, e.s, e.As, ref, e.sc, e.partials); }
                { ProfScope ps(e, "pcg_update"); e.launches += 1;
                  k_update4<<<nstream, UT, 0, e.stream>>>(n4, g.XY / 4, (const float4*)e.aw, (const float4*)e.s, (const float4*)e.As,
                                                          (float4*)e.pp, (float4*)e.r, ref, e.cfg.pcg_tol, e.cfg.pcg_max_iter, e.sc, e.partials); }
                { ProfScope ps(e, "pcg_search"); e.launches += 1;
                  k_search4<<<nstream, UT, 0, e.stream>>>(n4, (const float4*)e.aw, (const float4*)e.r, (float4*)e.s, e.sc); }
            } else {
                { ProfScope ps(e, "pcg_matvec"); e.launches += 1; k_matvec<<<std::min(MT.n, kMaxPartials), dim3(32, MW), 0, e.stream>>>(g, MT, e.ax, e.ay, e.az, e.aw, e.s, e.As, ref, e.sc, e.partials); }
                { ProfScope ps(e, "pcg_update"); e.launches += 1; k_update<<<nany, NT, 0, e.stream>>>(g.N, g.XY, e.aw, e.s, e.As, e.pp, e.r, ref, e.cfg.pcg_tol, e.cfg.pcg_max_iter, e.sc, e.partials); }
                { ProfScope ps(e, "pcg_search"); e.launches += 1; k_search<<<nany, NT, 0, e.stream>>>(g.N, e.aw, e.r, e.s, e.sc); }
            }
    };
    auto tail = [&]() {  // the last directions' pressure updates (no later operator launch carries them)
        if (path != PcgPath::FREE) return;
        ProfScope ps(e, "pcg_update");
        e.launches += 1;
        k_pressure4<true><<<nstream, UT, 0, e.stream>>>(n4, dp, (float4*)e.pp, e.sc);
    };
    if (e.capturing) {
        // graph mode: iteration 0, then chunks of `chunk` iterations as a WHILE loop that runs while
        // the solver has not stopped; the kernels of iterations past the stop return at once, as in
        // the stream-ordered form
        if (e.cfg.pcg_max_iter > 0) {
            iterate(0);
            graph_while(
                e, [&](cudaGraphConditionalHandle h) {
                    k_pcg_cond<<<1, 1, 0, e.stream>>>(h, e.sc, -1);
                    e.launches += 1;
                },
                [&](cudaGraphConditionalHandle h, int loop) {
                    for (int kk = 1; kk <= chunk; ++kk) iterate(kk);
                    k_pcg_cond<<<1, 1, 0, e.stream>>>(h, e.sc, loop);
                    e.launches += 1;
                });
            tail();
        }
    } else {
    for (int it = 0; it < e.cfg.pcg_max_iter; it += chunk) {
        const int n = std::min(chunk, e.cfg.pcg_max_iter - it);
        for (int k = 0; k < n; ++k) iterate(it + k);
        fetch_scalars(e);
        if (e.host_sc->converged || e.host_sc->status != 0) break;
    }
    if (e.cfg.pcg_max_iter > 0) tail();
    e.last_iters = e.host_sc->iters;
    e.last_residual = e.host_sc->residual;
    e.last_converged = e.host_sc->converged == 1;
    }
    }
    const dim3 grd((g.X + 31) / 32, (g.Y + 7) / 8, g.Z), blk(32, 8);
    ProfScope ps(e, "proj_apply");
    e.launches += 2;
    k_press_dens<<<grd, blk, 0, e.stream>>>(g, e.p, e.pp, e.rho, e.th, e.qv, e.Pg);
    if (e.flat && (g.X % 4) == 0) {
        const int ax = (g.X / 4 + 31) / 32, ay = (g.Y - 1 + 7) / 8;
        int az = std::max(1, std::min(g.Z, (stencil_sms(e) * 16 + ax * ay - 1) / (ax * ay)));
        const int alen = (g.Z + az - 1) / az;
        az = (g.Z + alen - 1) / alen;
        k_apply_proj4<<<dim3(ax, ay, az), dim3(32, 8), 0, e.stream>>>(g, alen, e.pp, e.rho, e.u, e.v, e.w);
    } else {
        k_apply_proj<<<grd, blk, 0, e.stream>>>(g, e.pp, e.rho, e.u, e.v, e.w);
    }
}

}  // namespace skt
