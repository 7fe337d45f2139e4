// Coulomb and D4 pair terms, every pair once, with a register tile of pairs per lane.
// Included inside namespace gfnff by engine.cu (one translation unit); k_pairs
// (k_nonbonded.cuh) evaluates the same pairs by rows and describes the terms.
//
// A warp owns 32 rows i and walks 8 partners j per step: lane (g, t) = (lane / 4, lane % 4)
// holds the pairs of rows g, g+8, g+16, g+24 with the partners 2t and 2t+1, which is the
// accumulator layout of mma.m16n8k4 (FP64).  That layout decides everything else:
//  * the C6 of the pairs and both dC6/dCN, which are dot products of per-atom vectors (half
//    contraction of one atom against the reference weights of the other), come from the FP64
//    tensor instruction, 32 x 8 pairs at a time over the packed references of all elements
//    present (5 -> 8 for water, 17 -> 20 for C/H/N/O), from operands that a warp reads as
//    contiguous runs, instead of three gathered dots per pair whose loads no two lanes shared;
//  * row sums stay in registers for the whole tile, and the partner sums of a step meet in 7
//    exchanges per 256 pairs, where one pair per lane needed 15-20 shuffles a pair;
//  * 4 independent pairs per lane without a branch between them cover the latency of the FP64
//    pipe; pairs within the width of the charges (erf, exp) are redone in one loop after them.
// Measured on a B200 with events, both kernels one after the other against one pair per lane and
// partner tiles in shared memory: 20,480 atoms 2.42 -> 1.36 ms (largest tiles), 1000 waters 142 -> 72 us,
// 512 conformers 285 -> 165 us, 194 atoms 70 -> 27 us (smallest tiles).  Under the profiler, which
// starts every kernel cold, on 20,480 atoms: Coulomb (128 x 64) 0.57 ms, the FP64 pipe 49 % busy (25 of 55
// instructions a pair; 0.29 ms of FP64 issue); D4 (32 x 64) 0.89 ms, latency of the operand loads and
// the dependent chain (FP64 pipe 26 %).  One kernel for both terms was slower (1.38-2.0 ms, events):
// the D4 part takes the registers of the Coulomb part, and far tiles cannot leave early.
#pragma once

namespace {

// warps per SM the pair kernels are built for: 168 registers a thread, without spills but for the
// exact-gradient form of Coulomb (FAR, 40-44 bytes); 16 warps at 128 registers spilled in every form and
// measured 3 % slower on the 20,480-atom cluster
constexpr int kPairWarps = 12;

// c += A B, A 16 x 4 (lane: rows g and g + 8, column t), B 4 x 8 (lane: row t, column g),
// c 16 x 8 (lane: rows g, g, g + 8, g + 8, columns 2t, 2t + 1, 2t, 2t + 1)
__device__ __forceinline__ void mma_16x8x4(double (&c)[4], double a0, double a1, double b)
{
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

// Coulomb pairs inside the reach of the charges' width (erf(x) < 1 in FP64), of the four pairs of
// rows ra, rb with partners ja, jb: energy and dE/dr / r of those set in `near`, one pair of
// every lane per turn.  One copy of erf and exp (unrolled over the pairs their code overran the
// instruction cache: 2.8 of 7.9 stall cycles per instruction on the conformer batch).
__device__ __forceinline__ void coulomb_near_pairs(const View& V, unsigned near, int ra, int rb, int ja, int jb,
                                                   const double (&d2)[4], const double (&qq)[4], double (&e)[4],
                                                   double (&f)[4])
{
    const double tsp = 2.0 / 1.772453850905516;
#pragma unroll 1
    do {
        const int k = __ffs(near) - 1;
        near &= near - 1;
        const double x = k < 2 ? (k == 0 ? d2[0] : d2[1]) : (k == 2 ? d2[2] : d2[3]);
        const double q = k < 2 ? (k == 0 ? qq[0] : qq[1]) : (k == 2 ? qq[2] : qq[3]);
        const double s = V.alpeeq[k < 2 ? ra : rb] + V.alpeeq[k & 1 ? jb : ja];
        if (x < 1e-20) {   // coincident atoms: no pair
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m == k) e[m] = f[m] = 0.0;
        } else if (x < 36.0 * s) {
            const double r = sqrt(x), g = 1.0 / sqrt(s), gr = g * r, ef = erf(gr);
            const double ek = q * ef / r;
            const double fk = q * ((g * exp(-gr * gr) * tsp) / r - ef / x) / r;
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m == k) {
                    e[m] = ek;
                    f[m] = fk;
                }
        }
    } while (near);
}

constexpr int kPairCoul = 1, kPairD4 = 2;
// largest coordinate change since the set-up (bohr) under which a pair within 50 bohr is
// certainly on the D4 list (set-up distance <= 60): 50 + 2 sqrt(3) 2.8 < 60
constexpr double kPairFreeMove = 2.8;

// Sums of the step over the warp's 32 rows: reduce-scatter over g, partner by bit 2 of g, component
// by its low bits.  v: 4 components of partner 2t, then of 2t + 1; returns component g % 4 of
// partner 2t + g / 4.
__device__ __forceinline__ double partner_sums(double (&v)[8], int g)
{
    constexpr unsigned full = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const bool up = (g & 4) != 0;
        const double send = up ? v[k] : v[k + 4], keep = up ? v[k + 4] : v[k];
        v[k] = keep + __shfl_xor_sync(full, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool up = (g & 2) != 0;
        const double send = up ? v[k] : v[k + 2], keep = up ? v[k + 2] : v[k];
        v[k] = keep + __shfl_xor_sync(full, send, 8);
    }
    const bool up = (g & 1) != 0;
    return (up ? v[1] : v[0]) + __shfl_xor_sync(full, up ? v[0] : v[1], 4);
}

// The same over t for the row sums: lane (g, t) ends with row g + 8 a, a = 2 (t & 1) + (t >> 1), its
// four components in r[0].
__device__ __forceinline__ void row_sums(double (&r)[4][4], int t)
{
    constexpr unsigned full = 0xffffffffu;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool up = (t & 1) != 0;
            const double send = up ? r[a][k] : r[a + 2][k], keep = up ? r[a + 2][k] : r[a][k];
            r[a][k] = keep + __shfl_xor_sync(full, send, 1);
        }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const bool up = (t & 2) != 0;
        const double send = up ? r[0][k] : r[1][k], keep = up ? r[1][k] : r[0][k];
        r[0][k] = keep + __shfl_xor_sync(full, send, 2);
    }
}

// true when no atom of rows [r0, r1) (32 at most) is within sqrt(cut2) of one of [j0, j1): the gap
// of their boxes in 1/16 bohr, rounded towards each other
__device__ __forceinline__ bool tile_far(const View& V, int r0, int r1, int j0, int j1, float cut2)
{
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double4 p = V.pos[min(r0 + lane, r1 - 1)];
    const double px[3] = {p.x, p.y, p.z};
    int clo[3], chi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        clo[d] = 0x7fffffff;
        chi[d] = -0x7fffffff;
    }
    for (int j = j0 + lane; j < j1; j += 32) {
        const double4 q = V.pos[j];
        const double qx[3] = {q.x, q.y, q.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            clo[d] = min(clo[d], __double2int_rd(16.0 * qx[d]));
            chi[d] = max(chi[d], __double2int_ru(16.0 * qx[d]));
        }
    }
    float gap2 = 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long long rl = __reduce_min_sync(full, __double2int_rd(16.0 * px[d]));
        const long long rh = __reduce_max_sync(full, __double2int_ru(16.0 * px[d]));
        const long long cl = __reduce_min_sync(full, clo[d]), ch = __reduce_max_sync(full, chi[d]);
        // integers up to the difference: a coordinate of 1e8 bohr in FP32 is 8 bohr off
        const float gap = (float)max(0ll, max(cl - rh, rl - ch));
        gap2 += gap * gap;
    }
    return gap2 > cut2 * 256.f * 1.0001f;
}

// Both kernels: tiles {first row, end of rows, first partner, end of partners}, rows at most 32 WR
// (a warp per 32), partners at most COLS, all of one molecule; pairs with j > i only.
//
// Adds the partner sums of the block's warps (colacc) and a warp's row sums; FAR: the fourth
// component is the potential of the cut pairs, otherwise dE/dCN.
template <int WR, int COLS, int NC, bool FAR>
__device__ __forceinline__ void add_partners(const View& V, const double (*colacc)[NC][COLS], int j0, int jend)
{
    for (int k = threadIdx.x; k < NC * COLS; k += 32 * WR) {
        const int comp = k / COLS, c = k % COLS, j = j0 + c;
        if (j >= jend) continue;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < WR; ++w) s += colacc[w][comp][c];
        if (s != 0.0) atomicAdd(comp < 3 ? V.grad + 3 * j + comp : (FAR ? V.cfar : V.dEdcn) + j, s);
    }
}

// ---- Coulomb (r <= 100 bohr) ----
// FAR (exact-gradient mode): also the potential of the pairs beyond, whose EEQ element is 1/r.
template <int WR, int COLS, bool CELL, bool FAR>
__global__ void __launch_bounds__(32 * WR, kPairWarps / WR) k_pairs_coul(View V, const int4* __restrict__ tiles)
{
    constexpr unsigned full = 0xffffffffu;
    constexpr int NC = FAR ? 4 : 3;
    __shared__ double colacc[WR][NC][COLS];
    __shared__ double esum[WR];
    // the warp's rows {x, y, z, q}: read again for every 16 rows of a step, which leaves the
    // registers to the pairs
    __shared__ double srow[WR][4][32];
    const int4 tl = tiles[blockIdx.x];
    const int iend = tl.y, j0 = tl.z, jend = tl.w;
    const int warp = WR > 1 ? threadIdx.x >> 5 : 0, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = tl.x + 32 * warp;
    double ec = 0.0;
    if (r0 < iend) {
        {
            const int i = min(r0 + lane, iend - 1);
            const double4 p = V.pos[i];
            srow[warp][0][lane] = p.x;
            srow[warp][1][lane] = p.y;
            srow[warp][2][lane] = p.z;
            srow[warp][3][lane] = V.q[i];
        }
        // the self terms of the rows, once: with the row block's first tile
        if (j0 == tl.x && r0 + lane < iend) ec = coulomb_self(V, r0 + lane);
        __syncwarp();
        double ga[4][4];   // row sums
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int k = 0; k < 4; ++k) ga[a][k] = 0.0;
        const int hmax_hi = __double2hiint(*V.hmax);
        for (int J = j0; J < jend; J += 8) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = 0.0;
            double s = 0.0;
            if (J + 7 > r0) {   // the step holds a pair with j > i (uniform in the warp)
                int jc[2], jid[2];
                double qx[2], qy[2], qz[2], qj[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int j = J + 2 * t + c;
                    jid[c] = j < jend ? j : -1;
                    jc[c] = min(j, jend - 1);
                    const double4 p = V.pos[jc[c]];
                    qx[c] = p.x; qy[c] = p.y; qz[c] = p.z;
                    qj[c] = V.q[jc[c]];
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {   // rows g + 16 h and g + 16 h + 8
                    const int l0 = g + 16 * h;
                    double dx[4], dy[4], dz[4], d2[4], qq[4], e[4], f[4];
                    int rid[2];
                    double px[2], py[2], pz[2], qi[2];
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const int i = r0 + l0 + 8 * a;
                        rid[a] = i < iend ? i : 0x7fffffff;
                        px[a] = srow[warp][0][l0 + 8 * a];
                        py[a] = srow[warp][1][l0 + 8 * a];
                        pz[a] = srow[warp][2][l0 + 8 * a];
                        qi[a] = srow[warp][3][l0 + 8 * a];
                    }
                    bool any = false;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {   // no branch: four independent chains
                        const int a = k >> 1, c = k & 1;
                        dx[k] = px[a] - qx[c];
                        dy[k] = py[a] - qy[c];
                        dz[k] = pz[a] - qz[c];
                        if (CELL) mic(V.cell, dx[k], dy[k], dz[k]);
                        d2[k] = dx[k] * dx[k] + dy[k] * dy[k] + dz[k] * dz[k];
                        qq[k] = qi[a] * qj[c];
                        // non-negative doubles order like their bit patterns (a NaN is above
                        // all), so the cut-offs are integer comparisons beside the FP64 pipe
                        const bool ok = jid[c] > rid[a];
                        const bool in = ok && __double_as_longlong(d2[k]) <= 0x40c3880000000000ll;   // d2 <= 1e4
                        const double y = rsqrt_pos(d2[k]);
                        const double ir = in ? y : 0.0;
                        e[k] = qq[k] * ir;
                        f[k] = -(e[k] * (ir * ir));
                        any |= in && __double2hiint(d2[k]) <= hmax_hi;
                        if (FAR && ok && d2[k] > 10000.0) {
                            const double irf = rsqrt(d2[k]);
                            ga[2 * h + a][3] += qj[c] * irf;
                            v[4 * c + 3] += qi[a] * irf;
                        }
                    }
                    if (any) {
                        unsigned near = 0;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (jid[k & 1] > rid[k >> 1] && __double2hiint(d2[k]) <= hmax_hi) near |= 1u << k;
                        const int ra = min(r0 + l0, iend - 1), rb = min(r0 + l0 + 8, iend - 1);
                        coulomb_near_pairs(V, near, ra, rb, jc[0], jc[1], d2, qq, e, f);
                    }
                    ec += (e[0] + e[1]) + (e[2] + e[3]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int a = 2 * h + (k >> 1), c = k & 1;
                        ga[a][0] += f[k] * dx[k];
                        ga[a][1] += f[k] * dy[k];
                        ga[a][2] += f[k] * dz[k];
                        v[4 * c] -= f[k] * dx[k];
                        v[4 * c + 1] -= f[k] * dy[k];
                        v[4 * c + 2] -= f[k] * dz[k];
                    }
                }
                s = partner_sums(v, g);
            }
            if (NC == 4 || (g & 3) < 3) colacc[warp][NC == 4 ? g & 3 : min(g & 3, 2)][J - j0 + 2 * t + (g >> 2)] = s;
        }
        row_sums(ga, t);
        const int i = r0 + g + 8 * (2 * (t & 1) + (t >> 1));
        if (i < iend) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (ga[0][k] != 0.0) atomicAdd(V.grad + 3 * i + k, ga[0][k]);
            if (FAR && ga[0][3] != 0.0) atomicAdd(V.cfar + i, ga[0][3]);
        }
    } else {
        for (int k = lane; k < NC * COLS; k += 32) colacc[warp][k / COLS][k % COLS] = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) ec += __shfl_xor_sync(full, ec, o);
    if (lane == 0) esum[warp] = ec;
    if (WR > 1) __syncthreads();
    else __syncwarp();
    add_partners<WR, COLS, NC, FAR>(V, colacc, j0, jend);
    if (threadIdx.x == 0) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < WR; ++w) s += esum[w];
        if (s != 0.0) atomicAdd(V.E + 16 * (V.nmol == 1 ? 0 : V.mol[tl.x]) + T_COUL, s);
    }
}

// ---- D4 (r <= 50 bohr, set-up distance <= 60) ----
// Tiles whose boxes are farther apart leave at once (no test in a cell, whose images move).
template <int WR, int COLS, bool CELL>
__global__ void __launch_bounds__(32 * WR, kPairWarps / WR) k_pairs_d4(View V, const int4* __restrict__ tiles)
{
    constexpr unsigned full = 0xffffffffu;
    __shared__ double colacc[WR][4][COLS];
    __shared__ double esum[WR];
    __shared__ double srow[WR][4][32];   // the warp's rows {x, y, z, c4}
    const int4 tl = tiles[blockIdx.x];
    const int iend = tl.y, j0 = tl.z, jend = tl.w;
    const int warp = WR > 1 ? threadIdx.x >> 5 : 0, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = tl.x + 32 * warp;
    double ed = 0.0;
    const bool act = r0 < iend && jend > r0 + 1 && (CELL || !tile_far(V, r0, min(r0 + 32, iend), j0, jend, 2500.f));
    if (WR > 1 ? !__syncthreads_or(act) : !act) return;
    if (act) {
        {
            const int i = min(r0 + lane, iend - 1);
            const double4 p = V.pos[i];
            srow[warp][0][lane] = p.x;
            srow[warp][1][lane] = p.y;
            srow[warp][2][lane] = p.z;
            srow[warp][3][lane] = V.c4[i];
        }
        __syncwarp();
        double ga[4][4];   // row sums
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int k = 0; k < 4; ++k) ga[a][k] = 0.0;
        const bool check0 = CELL || !(V.msd[2] <= kPairFreeMove);
        const bool want_dc = !V.exact;
        const int sh = V.pshift[V.nmol == 1 ? 0 : V.mol[tl.x]];
        const int gs = 8 * V.Rp;   // doubles of a group of 8 packed rows
        const int prow = ((r0 + sh) >> 3) * gs + lane;
        for (int J = j0; J < jend; J += 8) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = 0.0;
            double s = 0.0;
            if (J + 7 > r0) {
                int jc[2], jid[2];
                double qx[2], qy[2], qz[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int j = J + 2 * t + c;
                    jid[c] = j < jend ? j : -1;
                    jc[c] = min(j, jend - 1);
                    const double4 p = V.pos[jc[c]];
                    qx[c] = p.x; qy[c] = p.y; qz[c] = p.z;
                }
                bool hit = false;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int l0 = g + 16 * h;
                    double dx[4], dy[4], dz[4], d2[4];
                    bool in4[4];
                    int rid[2];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int a = k >> 1, c = k & 1;
                        const int i = r0 + l0 + 8 * a;
                        rid[a] = i < iend ? i : 0x7fffffff;
                        dx[k] = srow[warp][0][l0 + 8 * a] - qx[c];
                        dy[k] = srow[warp][1][l0 + 8 * a] - qy[c];
                        dz[k] = srow[warp][2][l0 + 8 * a] - qz[c];
                        if (CELL) mic(V.cell, dx[k], dy[k], dz[k]);
                        d2[k] = dx[k] * dx[k] + dy[k] * dy[k] + dz[k] * dz[k];
                        const long long b = __double_as_longlong(d2[k]);   // ordered as the doubles
                        in4[k] = jid[c] > rid[a] && b <= 0x40a3880000000000ll && b >= 0x3bc79ca10c924223ll;   // 1e-20 .. 2500
                    }
                    if (!__any_sync(full, in4[0] || in4[1] || in4[2] || in4[3])) continue;
                    hit = true;
                    double c6[4] = {0.0, 0.0, 0.0, 0.0}, di[4] = {0.0, 0.0, 0.0, 0.0}, dj[4] = {0.0, 0.0, 0.0, 0.0};
                    {
                        // operand runs of the rows' two groups of 8 atoms and of the partners'
                        const int oa = prow + 2 * h * gs, ob = oa + gs, oj = ((J + sh) >> 3) * gs + lane;
                        if (want_dc) {
#pragma unroll 2
                            for (int k = 0; k < gs; k += 32) {
                                const double a0 = V.g0p[oa + k], a1 = V.g0p[ob + k], b0 = V.w0p[oj + k];
                                const double a2 = V.hdgp[oa + k], a3 = V.hdgp[ob + k], b1 = V.wp[oj + k];
                                const double a4 = V.wp[oa + k], a5 = V.wp[ob + k], b2 = V.hdgp[oj + k];
                                mma_16x8x4(c6, a0, a1, b0);
                                mma_16x8x4(di, a2, a3, b1);
                                mma_16x8x4(dj, a4, a5, b2);
                            }
                        } else {
#pragma unroll 2
                            for (int k = 0; k < gs; k += 32) mma_16x8x4(c6, V.g0p[oa + k], V.g0p[ob + k], V.w0p[oj + k]);
                        }
                    }
                    const int ra = min(r0 + l0, iend - 1), rb = min(r0 + l0 + 8, iend - 1);
                    const double ci[2] = {srow[warp][3][l0], srow[warp][3][l0 + 8]};
                    const double cj[2] = {V.c4[jc[0]], V.c4[jc[1]]};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int a = k >> 1, c = k & 1;
                        bool in = in4[k];
                        if (check0 && in) in = d2_exact(V.pos0[a ? rb : ra], V.pos0[jc[c]]) <= 3600.0;
                        // sr = sqrt(r4r2 of the pair); zeta_i zeta_j is folded into c6, di, dj
                        const double sr = ci[a] * cj[c], q2 = in ? d2[k] : 1.0, q4 = q2 * q2;
                        const double b0 = fma(0.58, sr, 4.80), b02 = b0 * b0, b04 = b02 * b02;
                        const double r6 = q4 * q2;
                        const double a6 = fma(b04, b02, r6), a8 = fma(q4, q4, b04 * b04);
                        const double inv = in ? rcp_pos(a6 * a8) : 0.0;   // t6 = t8 = 0 off the list
                        const double t6 = a8 * inv, t8 = a6 * inv, s8 = 2.0 * (sr * sr) * t8;
                        const double sum = t6 + s8;
                        ed -= c6[k] * sum;
                        // dE/dr / r = c6 (6 r^4 t6^2 + 16 r4r2 r^6 t8^2)
                        const double f = c6[k] * (6.0 * q4 * (t6 * t6) + 8.0 * r6 * (s8 * t8));
                        ga[2 * h + a][0] += f * dx[k];
                        ga[2 * h + a][1] += f * dy[k];
                        ga[2 * h + a][2] += f * dz[k];
                        ga[2 * h + a][3] -= di[k] * sum;
                        v[4 * c] -= f * dx[k];
                        v[4 * c + 1] -= f * dy[k];
                        v[4 * c + 2] -= f * dz[k];
                        v[4 * c + 3] -= dj[k] * sum;
                    }
                }
                if (hit) s = partner_sums(v, g);
            }
            colacc[warp][g & 3][J - j0 + 2 * t + (g >> 2)] = s;
        }
        row_sums(ga, t);
        const int i = r0 + g + 8 * (2 * (t & 1) + (t >> 1));
        if (i < iend) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (ga[0][k] != 0.0) atomicAdd(V.grad + 3 * i + k, ga[0][k]);
            if (ga[0][3] != 0.0) atomicAdd(V.dEdcn + i, ga[0][3]);
        }
    } else {
        for (int k = lane; k < 4 * COLS; k += 32) colacc[warp][k / COLS][k % COLS] = 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) ed += __shfl_xor_sync(full, ed, o);
    if (lane == 0) esum[warp] = ed;
    if (WR > 1) __syncthreads();
    else __syncwarp();
    add_partners<WR, COLS, 4, false>(V, colacc, j0, jend);
    if (threadIdx.x == 0) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < WR; ++w) s += esum[w];
        if (s != 0.0) atomicAdd(V.E + 16 * (V.nmol == 1 ? 0 : V.mol[tl.x]) + T_DISP, s);
    }
}

}  // namespace
