// Non-bonded GFN-FF kernels: geometry in, coordination numbers, D4 weights, repulsion,
// all-pairs Coulomb + D4 dispersion, self energy, CN chain rule and the outputs.
// Included inside namespace gfnff by engine.cu (one translation unit).
//
// The kernels that go over all pairs by rows (k_pairs, the plain form of the Coulomb and D4 pairs, and
// k_resp_pairs) share one layout; the Coulomb and D4 pairs of the default path are in k_pairs.cuh, and CN,
// repulsion and the chain rule take a warp per atom.  A block owns kTile consecutive atoms i (one per
// thread) and walks the partners j of its molecule range in tiles of kTile staged through
// shared memory, so every partner record is read from L2 once per block and broadcast to
// all threads.  grid.y splits the partner range of an i-block (nsplit slices) so that small
// systems still fill the 148 SMs; per-atom partial sums then meet in FP64 atomics.  Atoms
// are Morton-sorted at upload, so the lanes of a warp are spatial neighbours and the
// short-range branches (erf, exp) stay coherent.
#pragma once

namespace {

constexpr int kTile = 128;

// partner range [jb, je) of this block's slice
__device__ __forceinline__ void tile_range(const View& V, int i0, int nsplit, int& jb, int& je)
{
    const int last = min(V.n, i0 + kTile) - 1;
    const int lo = V.jr[i0].x, hi = V.jr[last].y;
    const int ntiles = (hi - lo + kTile - 1) / kTile;
    const int per = (ntiles + nsplit - 1) / nsplit;
    jb = lo + (int)blockIdx.y * per * kTile;
    je = min(hi, jb + per * kTile);
}

// ------------------------------------------------------------------------------------
// geometry in (caller order -> internal order) and the HB refresh metric
// (gfnff_method.cpp:2228-2259)
// ------------------------------------------------------------------------------------
// (nl_ref, nl_bad): reference geometry of the CN neighbour list; an atom more than
// sqrt(nl_lim2) away from it marks the list stale (kept until the host rebuilds it).
// msd[1] receives the topology refresh metric, the largest |coordinate change| since the
// geometry topo_ref of the last topology (gfnff_method.cpp:1021-1031), as the bits of a
// non-negative double (which order like the integers); msd[2] the largest |coordinate change|
// since the set-up geometry pos0 (all atoms of a batch)
// Also clears what the evaluation adds into (Z): a memset node each cost more than the writes.
struct StepZero {
    double *grad, *dEdcn, *cfar, *E;   // 3n, n, n (or null), nE
    int nE;
    int* bad;                          // nmol
    int nmol;
    int* words[4];                     // single counters (or null)
};
__global__ void k_positions(int n, const int* __restrict__ perm, const double* __restrict__ xyz, double scale,
                            double4* pos, const double4* __restrict__ ref, double* msd,
                            const double4* __restrict__ nl_ref, double nl_lim2, int* nl_bad,
                            const double4* __restrict__ topo_ref, const double4* __restrict__ pos0, StepZero Z)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0, dmax = 0.0, d0max = 0.0;
    for (int k = i; k < Z.nE; k += gridDim.x * blockDim.x) Z.E[k] = 0.0;
    for (int k = i; k < Z.nmol; k += gridDim.x * blockDim.x) Z.bad[k] = 0;
    if (i < 4 && Z.words[i]) *Z.words[i] = 0;
    if (i < n) {
        Z.grad[3 * i] = Z.grad[3 * i + 1] = Z.grad[3 * i + 2] = 0.0;
        Z.dEdcn[i] = 0.0;
        if (Z.cfar) Z.cfar[i] = 0.0;
        const int o = perm[i];
        const double x = xyz[3 * o] * scale, y = xyz[3 * o + 1] * scale, z = xyz[3 * o + 2] * scale;
        pos[i] = make_double4(x, y, z, 0.0);
        const double4 p0 = pos0[i];
        d0max = fmax(fabs(x - p0.x), fmax(fabs(y - p0.y), fabs(z - p0.z)));
        const double4 r = ref[i];
        s = (x - r.x) * (x - r.x) + (y - r.y) * (y - r.y) + (z - r.z) * (z - r.z);
        const double4 t = topo_ref[i];
        dmax = fmax(fabs(x - t.x), fmax(fabs(y - t.y), fabs(z - t.z)));
        if (nl_ref) {
            const double4 q = nl_ref[i];
            const double d2 = (x - q.x) * (x - q.x) + (y - q.y) * (y - q.y) + (z - q.z) * (z - q.z);
            if (d2 > nl_lim2) atomicOr(nl_bad, 1);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        d0max = fmax(d0max, __shfl_xor_sync(0xffffffffu, d0max, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (dmax > 0.0)
            atomicMax(reinterpret_cast<unsigned long long*>(msd + 1), (unsigned long long)__double_as_longlong(dmax));
        if (d0max > 0.0)
            atomicMax(reinterpret_cast<unsigned long long*>(msd + 2), (unsigned long long)__double_as_longlong(d0max));
    }
    block_add(s, msd);
}

// One counting term 0.5 (1 + erf(kn (r - rc) / rc)), kn = -7.5, of the GFN-FF CN
// (cn_calculator.cpp:367-428); d2 = r^2, rc = the pair's covalent radius sum (bohr).  FP64:
// as written.  FP32 (mixed form): the argument in FP64, then the identity 0.5 (1 + erf(z)) =
// 0.5 erfc(-z) with only the small tail erfc(|z|) in FP32, subtracted from an exact 1 for
// z >= 0 and accumulated in FP64: 1 + erf(z) in FP32 cancels to a few significant bits for
// the distant pairs, whose rounding then adds up over ~100 partners per atom.
template <class R>
__device__ __forceinline__ double cn_count(double d2, double rc)
{
    const double r = sqrt(d2);
    const double z = -7.5 * ((r - rc) / rc);
    if constexpr (std::is_same<R, double>::value) {
        return 0.5 * (1.0 + erf(z));
    } else {
        const double t = (double)erfcf((float)fabs(z));
        return z >= 0.0 ? 1.0 - 0.5 * t : 0.5 * t;
    }
}

// ------------------------------------------------------------------------------------
// Coordination numbers (erf counting over partners closer than 6 bohr, cn_calculator.cpp:367-428),
// their log-squash (cnmax = 4.4) and its derivative, D4 Gaussian weights (wf = 4) and the half
// contraction of their derivative with the reference C6 (d4param_generator.cpp:1079-1290,
// :1692-1740): one warp per atom, one launch (CN by list, CN by all pairs when the list is stale,
// and the weights were three).
//
// The partners come from a Verlet list (pairs within 6 + 1 bohr at the list's reference geometry,
// same molecule, CSR by atom, both directions), valid while no atom moved more than half the
// 1-bohr skin (*nl_bad, checked in k_positions at every evaluation).  Without a valid list the
// warp scans its molecule, 32 atoms a step: 2 x 3 us on 194 atoms where a block per 128 atoms and
// partner tiles in shared memory took 41 (CN) and 48 us (chain rule).
//
// The weights: lane r of every eight holds reference r (7 at most), so the exponentials of an atom
// run side by side, and the lanes then share the packed references.
// ------------------------------------------------------------------------------------
template <bool CELL, class F>
__device__ __forceinline__ void cn_partners(const View& V, int i, const double4& pi, const int* off, const int* nbr,
                                            const int* nl_bad, F f)
{
    const int lane = threadIdx.x & 31;
    if (off && *nl_bad == 0) {
        for (int p = off[i] + lane; p < off[i + 1]; p += 32) {
            const int j = nbr[p];
            const double4 pj = V.pos[j];
            const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (d2 < 36.0) f(j, dx, dy, dz, d2);
        }
    } else {
        const int2 rg = V.jr[i];
        for (int j = rg.x + lane; j < rg.y; j += 32) {
            const double4 pj = V.pos[j];
            double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
            if (CELL) mic(V.cell, dx, dy, dz);
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (d2 < 36.0 && j != i) f(j, dx, dy, dz, d2);
        }
    }
}

// NA: atoms per warp, one after the other for the CN and side by side (eight lanes each) for the
// weights, whose logarithms and exponentials are the larger part of a large system's time; one where
// there are warps to spare.  Four against one, us: 3000 atoms 15.3 / 12.3, 5400 14.6 / 14.4, 8100 15.2 / 17.4,
// 18,000 18.4 / 27.6; batches of 7700 atoms 17.3 / 17.2, 16,400 19.6 / 25.4, 52,600 36.6 / 61.9.
template <class R, bool CELL, int NA>
__global__ void __launch_bounds__(kBlock) k_cn_d4(View V, const int* __restrict__ off, const int* __restrict__ nbr,
                                                 const int* nl_bad)
{
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = NA == 1 ? 0 : lane >> 3;
    const int i0 = (blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * NA;
    if (i0 >= V.n) return;
    double s = 0.0;
#pragma unroll 1
    for (int a = 0; a < NA; ++a) {
        const int ia = min(i0 + a, V.n - 1);
        const double4 pi = V.pos[ia];
        const double ri = V.rcov_cn[ia];
        double t = 0.0;
        cn_partners<CELL>(V, ia, pi, off, nbr, nl_bad, [&](int j, double, double, double, double d2) {
            t += cn_count<R>(d2, ri + V.rcov_cn[j]);
        });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(full, t, o);
        if (sub == a) s = t;
    }
    const int i = min(i0 + sub, V.n - 1);
    const bool act = i0 + sub < V.n;
    const double cnmax = 4.4;
    const double cn = log(1.0 + exp(cnmax)) - log(1.0 + exp(cnmax - s));
    const int nr = V.nref[i], r = lane & 7;
    double ex = 0.0, dex = 0.0;
    if (r < nr) {
        const double d = cn - V.refcn[i * 7 + r];
        ex = exp(-4.0 * d * d);
        dex = (-2.0 * 4.0) * d * ex;
    }
    double norm = ex, dnorm = dex;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        norm += __shfl_xor_sync(full, norm, o);
        dnorm += __shfl_xor_sync(full, dnorm, o);
    }
    double w = 0.0, dw = 0.0;
    if (r < nr) {
        if (norm > 1e-10) {
            const double inv = 1.0 / norm, inv2 = 1.0 / (norm * norm);
            w = ex * inv;
            dw = (dex * norm - ex * dnorm) * inv2;
        } else {
            w = r == 0 ? 1.0 : 0.0;
        }
    }
    const double z = V.zeta[i];
    const int row = i + V.pshift[V.nmol == 1 ? 0 : V.mol[i]];
    const int l = NA == 1 ? lane : r;   // lane among those of the atom
    if (act && l == 0) {
        V.cn[i] = cn;
        V.dlog[i] = exp(cnmax) / (exp(cnmax) + exp(s));
        V.dxdcn[i] = V.cnf[i] / (2.0 * sqrt(fmax(cn, 0.0)) + 1e-16);
    }
    if (act && l < nr) V.wp[pk(V.Rp, row, V.kof[i] + l)] = z * w;
    const double* C = V.c6p + (size_t)V.slot[i] * 7 * V.Rp;
    double dwa[7];
#pragma unroll
    for (int a = 0; a < 7; ++a) dwa[a] = __shfl_sync(full, dw, (lane & 24) + a);
    for (int k = l; k < V.Rp; k += NA == 1 ? 32 : 8) {
        double dg = 0.0;
#pragma unroll
        for (int a = 0; a < 7; ++a)
            if (a < nr) dg += dwa[a] * C[a * V.Rp + k];
        if (act) V.hdgp[pk(V.Rp, row, k)] = z * dg;
    }
}

// ------------------------------------------------------------------------------------
// repulsion over per-atom CSR lists holding both pair directions
// (ff_workspace_gfnff.cpp:774-848); kind 0 = bonded, 1 = non-bonded.  One warp per atom.
// ------------------------------------------------------------------------------------
template <class R>
__global__ void __launch_bounds__(kBlock) k_repulsion(View V, const int* off, const int* nbj, const double* alpha,
                                                     const double* repab, const unsigned char* kind)
{
    const int i = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    double eb = 0.0, enb = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    if (i < V.n) {
        const double4 pi = V.pos[i];
        for (int p = off[i] + lane; p < off[i + 1]; p += 32) {
            const double4 pj = V.pos[nbj[p]];
            double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            if (V.cell.on) mic(V.cell, dx, dy, dz);
            const double d2 = dx * dx + dy * dy + dz * dz;
            const R r = sqrt((R)d2);
            if (r > R(20) || r < R(1e-8)) continue;
            const R sr = sqrt(r), al = (R)alpha[p];
            const R e = (R)repab[p] * exp(-al * (r * sr)) / r;
            if (kind[p]) enb += 0.5 * (double)e; else eb += 0.5 * (double)e;
            const R dEdr = -e / r - R(1.5) * al * sr * e;
            const double f = (double)(dEdr / r);
            gx += f * dx; gy += f * dy; gz += f * dz;
        }
        for (int o = 16; o > 0; o >>= 1) {
            gx += __shfl_down_sync(0xffffffffu, gx, o);
            gy += __shfl_down_sync(0xffffffffu, gy, o);
            gz += __shfl_down_sync(0xffffffffu, gz, o);
        }
        // atomics: the kernel runs beside others that add to the same gradient entries
        if (lane == 0) {
            if (gx != 0.0) atomicAdd(V.grad + 3 * i, gx);
            if (gy != 0.0) atomicAdd(V.grad + 3 * i + 1, gy);
            if (gz != 0.0) atomicAdd(V.grad + 3 * i + 2, gz);
        }
    }
    const int m = i < V.n ? V.mol[i] : -1;
    eadd(V, eb, m, T_BREP);
    eadd(V, enb, m, T_NBREP);
}

// ------------------------------------------------------------------------------------
// all-pairs Coulomb (r <= 100 bohr; ff_workspace_gfnff.cpp:850-900) and D4 dispersion
// over the setup pair list (setup distance <= 60 bohr, evaluated for r <= 50;
// :715-772, d4param_generator.cpp:1959-2092) with the frozen setup C6 and the per-step
// dC6/dCN chain term.  Both directions of a pair are evaluated (row i collects its own
// gradient and dE/dCN_i); energies are halved.
//
// Coulomb fast path: erf(x) rounds to exactly 1 in double for x >= 6 (erfc(6) = 2.2e-17
// is below half an ulp of 1), i.e. for r^2 >= 36 (a_i + a_j); the pair is then q q / r and
// its exp(-x^2) gradient term is below 2e-15 relative, so both are dropped there.
// This kernel (each block a run of atoms against all partners, both directions of a pair) is the
// plain form of the terms; k_pairs_coul and k_pairs_d4 (k_pairs.cuh) evaluate the same pairs once.  It is one of
// the set-up tuner's variants ("rows").
// ------------------------------------------------------------------------------------
// Coulomb self term of atom i (ff_workspace.cpp:415-536)
__device__ __forceinline__ double coulomb_self(const View& V, int i)
{
    const int2 rg = V.jr[i];
    if (rg.y - rg.x < 2 || !(V.alpeeq[i] > 0.0)) return 0.0;
    const double q = V.q[i], chi = V.chi_base[i] + V.cnf[i] * sqrt(fmax(V.cn[i], 0.0));
    return -q * chi + 0.5 * q * q * V.adiag[i];
}

// one D4 pair: energy e, dE/dr / r in dedr, dE/dCN_i in dc (zeta folded into the operands)
__device__ __forceinline__ void d4_pair(const View& V, double d2, int rowi, int kj, const double (*sw0)[kTile],
                                        const double (*sw)[kTile], int jj, int nr, double szi, double szj,
                                        double& e, double& dedr, double& dc)
{
    double c6 = 0.0, dc6 = 0.0;
    for (int b = 0; b < nr; ++b) {
        c6 += V.g0p[pk(V.Rp, rowi, kj + b)] * sw0[b][jj];
        dc6 += V.hdgp[pk(V.Rp, rowi, kj + b)] * sw[b][jj];
    }
    const double q2 = d2;
    const double r4r2 = 3.0 * szi * szj;
    const double t = 0.58 * sqrt(r4r2) + 4.80;
    const double r0sq = t * t;
    const double r6 = q2 * q2 * q2, r06 = r0sq * r0sq * r0sq;
    const double t6 = 1.0 / (r6 + r06);
    const double t8 = 1.0 / (r6 * q2 + r06 * r0sq);
    const double sum = t6 + 2.0 * r4r2 * t8;
    e = -(c6 * sum);
    const double d6 = -6.0 * q2 * q2 * t6 * t6, d8 = -8.0 * r6 * t8 * t8;
    dedr = -(c6 * (d6 + 2.0 * r4r2 * d8));
    dc = -(dc6 * sum);
}

__global__ void __launch_bounds__(kTile) k_pairs(View V, int nsplit)
{
    __shared__ double sx[kTile], sy[kTile], sz[kTile], s0x[kTile], s0y[kTile], s0z[kTile];
    __shared__ double sq[kTile], sa[kTile], ssz[kTile];
    __shared__ double sw0[7][kTile], sw[7][kTile];
    __shared__ int sko[kTile], snr[kTile];
    const int i0 = blockIdx.x * kTile, i = i0 + threadIdx.x;
    int jb, je;
    tile_range(V, i0, nsplit, jb, je);
    const bool act = i < V.n;
    const int ic = act ? i : i0;
    const double4 pi = V.pos[ic], p0i = V.pos0[ic];
    const double ai = V.alpeeq[ic], qi = V.q[ic], szi = V.szr[ic];
    const int2 rg = act ? V.jr[i] : make_int2(0, 0);
    const int rowi = ic + V.pshift[V.mol[ic]];
    const double tsp = 2.0 / 1.772453850905516;
    double ec = 0.0, ed = 0.0, gx = 0.0, gy = 0.0, gz = 0.0, dcn = 0.0, cfar = 0.0;
    for (int t0 = jb; t0 < je; t0 += kTile) {
        __syncthreads();
        const int jl = t0 + threadIdx.x;
        if (jl < je) {
            const int u = threadIdx.x;
            const double4 p = V.pos[jl], p0 = V.pos0[jl];
            sx[u] = p.x; sy[u] = p.y; sz[u] = p.z;
            s0x[u] = p0.x; s0y[u] = p0.y; s0z[u] = p0.z;
            sq[u] = V.q[jl]; sa[u] = V.alpeeq[jl]; ssz[u] = V.szr[jl];
            sko[u] = V.kof[jl]; snr[u] = V.nref[jl];
            const int row = jl + V.pshift[V.mol[jl]];
            for (int b = 0; b < snr[u]; ++b) {
                sw0[b][u] = V.w0p[pk(V.Rp, row, sko[u] + b)];
                sw[b][u] = V.wp[pk(V.Rp, row, sko[u] + b)];
            }
        }
        __syncthreads();
        const int cnt = min(kTile, je - t0);
        if (!act) continue;
        for (int jj = 0; jj < cnt; ++jj) {
            const int j = t0 + jj;
            if (j == i || j < rg.x || j >= rg.y) continue;
            double dx = pi.x - sx[jj], dy = pi.y - sy[jj], dz = pi.z - sz[jj];
            if (V.cell.on) mic(V.cell, dx, dy, dz);
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (d2 < 1e-20) continue;
            double f = 0.0;   // dE/dr / r
            if (d2 <= 10000.0) {
                const double s = ai + sa[jj];
                const double qq = qi * sq[jj];
                if (d2 >= 36.0 * s) {
                    const double ir = rsqrt(d2);
                    const double e = qq * ir;
                    ec += e;
                    f -= e * ir * ir;
                } else {
                    const double r = sqrt(d2);
                    const double g = 1.0 / sqrt(s);
                    const double gr = g * r;
                    const double ef = erf(gr);
                    ec += qq * ef / r;
                    f += qq * ((g * exp(-gr * gr) * tsp) / r - ef / d2) / r;
                }
            } else if (V.cfar) {
                cfar += sq[jj] * rsqrt(d2);   // cut pair: its EEQ element is 1/r
            }
            if (d2 <= 2500.0 &&
                d2_exact(p0i, make_double4(s0x[jj], s0y[jj], s0z[jj], 0.0)) <= 3600.0) {
                double e, dedr, dc;
                d4_pair(V, d2, rowi, sko[jj], sw0, sw, jj, snr[jj], szi, ssz[jj], e, dedr, dc);
                ed += e;
                f += dedr;
                if (!V.exact) dcn += dc;
            }
            gx += f * dx; gy += f * dy; gz += f * dz;
        }
    }
    if (act) {
        if (gx != 0.0) atomicAdd(V.grad + 3 * i, gx);
        if (gy != 0.0) atomicAdd(V.grad + 3 * i + 1, gy);
        if (gz != 0.0) atomicAdd(V.grad + 3 * i + 2, gz);
        if (dcn != 0.0) atomicAdd(V.dEdcn + i, dcn);
        if (cfar != 0.0) atomicAdd(V.cfar + i, cfar);
    }
    const int m = act ? V.mol[i] : -1;
    eadd(V, 0.5 * ec + (act && blockIdx.y == 0 ? coulomb_self(V, i) : 0.0), m, T_COUL);
    eadd(V, 0.5 * ed, m, T_DISP);
}

// ------------------------------------------------------------------------------------
// EEQ charge response (exact-gradient mode): with u = B M^-1 B^T w and w = dE/dq of the
// Coulomb pairs cut at 100 bohr, the gradient gains -sum_ij u_i q_j dA_ij/dr over all
// pairs (A is the uncut EEQ matrix) and u_i dx_i/dCN_i through the CN chain (k_tail).
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kTile) k_resp_pairs(View V, int nsplit)
{
    __shared__ double sx[kTile], sy[kTile], sz[kTile], sq[kTile], su[kTile], sa[kTile];
    const int i0 = blockIdx.x * kTile, i = i0 + threadIdx.x;
    int jb, je;
    tile_range(V, i0, nsplit, jb, je);
    const bool act = i < V.n;
    const int ic = act ? i : i0;
    const double4 pi = V.pos[ic];
    const double qi = V.q[ic], ui = V.u[ic], ai = V.alpeeq[ic];
    const int2 rg = act ? V.jr[i] : make_int2(0, 0);
    const double tsp = 2.0 / 1.772453850905516;
    double gx = 0.0, gy = 0.0, gz = 0.0;
    for (int t0 = jb; t0 < je; t0 += kTile) {
        __syncthreads();
        const int jl = t0 + threadIdx.x;
        if (jl < je) {
            const double4 p = V.pos[jl];
            sx[threadIdx.x] = p.x; sy[threadIdx.x] = p.y; sz[threadIdx.x] = p.z;
            sq[threadIdx.x] = V.q[jl]; su[threadIdx.x] = V.u[jl]; sa[threadIdx.x] = V.alpeeq[jl];
        }
        __syncthreads();
        const int cnt = min(kTile, je - t0);
        if (!act) continue;
        for (int jj = 0; jj < cnt; ++jj) {
            const int j = t0 + jj;
            if (j == i || j < rg.x || j >= rg.y) continue;
            const double dx = pi.x - sx[jj], dy = pi.y - sy[jj], dz = pi.z - sz[jj];
            const double d2 = dx * dx + dy * dy + dz * dz;
            const double s = ai + sa[jj];
            double dadr_r;   // dA/dr / r
            if (d2 >= 36.0 * s) {
                const double ir = rsqrt(d2);
                dadr_r = -ir * ir * ir;
            } else {
                const double r = sqrt(d2), g = 1.0 / sqrt(s), gr = g * r;
                dadr_r = ((g * exp(-gr * gr) * tsp) / r - erf(gr) / d2) / r;
            }
            const double f = -(ui * sq[jj] + su[jj] * qi) * dadr_r;
            gx += f * dx; gy += f * dy; gz += f * dz;
        }
    }
    if (act) {
        if (gx != 0.0) atomicAdd(V.grad + 3 * i, gx);
        if (gy != 0.0) atomicAdd(V.grad + 3 * i + 1, gy);
        if (gz != 0.0) atomicAdd(V.grad + 3 * i + 2, gz);
    }
}

// ------------------------------------------------------------------------------------
// The end of an evaluation, a warp per atom: the CN chain rule
// grad_i += sum_j dS_ij/dr (v_i + v_j) (x_i - x_j)/r over the 6 bohr neighbours
// (gfnff_method.cpp:5837-6260, forcefieldthread.h:80-109) with the chain weight
// v = dlogCN (dE/dCN - q cnf/(2 sqrt CN)) (ff_workspace.cpp:415-536) formed where it is read, the
// outputs in the caller's atom order, finiteness flags per molecule; the last block to finish
// sums the totals and statuses of the molecules.  One launch for what were five (weights, chain
// by list, chain by all pairs, outputs, totals); partners as in k_cn_d4.
// ------------------------------------------------------------------------------------
struct TailArgs {
    const int *off, *nbr, *nl_bad;
    double *gout, *qout, *cnout;
    int* bad;
    const int* eeq_info;
    const double* e0;
    double* etot;
    unsigned* done;   // blocks finished; back to 0 at the end
};

__device__ __forceinline__ double chain_weight(const View& V, int i)
{
    const double q = V.q[i];
    // the EEQ charge response u adds u dx/dCN (exact-gradient mode)
    const double qe = V.u ? q - V.u[i] : q;
    return V.dlog[i] * (V.dEdcn[i] - qe * V.dxdcn[i]);
}

template <bool CELL>
__global__ void __launch_bounds__(kBlock) k_tail(View V, TailArgs T)
{
    __shared__ bool last;
    const int i = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i < V.n) {
        const double4 pi = V.pos[i];
        const double ri = V.rcov_cn[i], vi = chain_weight(V, i);
        const double kn = -7.5, sqrtpi = 1.77245385091;
        double gx = 0.0, gy = 0.0, gz = 0.0;
        cn_partners<CELL>(V, i, pi, T.off, T.nbr, T.nl_bad, [&](int j, double dx, double dy, double dz, double d2) {
            const double r = sqrt(d2);
            const double rs = ri + V.rcov_cn[j];
            const double dr = (r - rs) / rs;
            const double de = (kn / sqrtpi) * exp(-kn * kn * dr * dr) / rs;
            const double f = -(de / r) * (vi + chain_weight(V, j));
            gx += f * dx; gy += f * dy; gz += f * dz;
        });
        for (int o = 16; o > 0; o >>= 1) {
            gx += __shfl_down_sync(0xffffffffu, gx, o);
            gy += __shfl_down_sync(0xffffffffu, gy, o);
            gz += __shfl_down_sync(0xffffffffu, gz, o);
        }
        if (lane == 0) {
            const int o = V.perm[i];
            gx += V.grad[3 * i];
            gy += V.grad[3 * i + 1];
            gz += V.grad[3 * i + 2];
            T.gout[3 * o] = gx;
            T.gout[3 * o + 1] = gy;
            T.gout[3 * o + 2] = gz;
            T.qout[o] = V.q[i];
            T.cnout[o] = V.cn[i];
            if (!isfinite(gx) || !isfinite(gy) || !isfinite(gz)) atomicOr(T.bad + V.mol[i], 1);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(T.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // per molecule: total energy, status (NOT_SPD from the EEQ factorisation, NONFINITE)
    for (int m = threadIdx.x; m < V.nmol; m += blockDim.x) {
        double tot = T.e0[m];
        for (int t = 0; t < T_TOTAL; ++t) tot += V.E[16 * m + t];
        V.E[16 * m + T_TOTAL] = tot;
        T.etot[m] = tot;
        int st = 0;
        if (T.eeq_info && T.eeq_info[m] == 2) st = GFNFF_CUDA_ERROR;
        else if (T.eeq_info && T.eeq_info[m] == 3) st = GFNFF_REFINE_NOT_CONVERGED;
        else if (T.eeq_info && T.eeq_info[m] != 0) st = GFNFF_NOT_SPD;
        else if (!isfinite(tot) || __ldcg(T.bad + m)) st = GFNFF_NONFINITE;
        V.status[m] = st;
    }
    if (threadIdx.x == 0) *T.done = 0u;
}

// device enumeration of the D4 pair list at the setup geometry (topology check)
__global__ void k_disp_count(int n, const double4* pos0, const int2* jr, unsigned long long* cnt, int2* out,
                             unsigned long long cap)
{
    const int i = blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j <= i || j >= n || j >= jr[i].y) return;
    if (d2_exact(pos0[i], pos0[j]) <= 3600.0) {
        const unsigned long long s = atomicAdd(cnt, 1ull);
        if (out && s < cap) out[s] = make_int2(i, j);
    }
}

// ------------------------------------------------------------------------------------
// The terms with a thread per term (angles, torsions, inversions, three-body and halogen-bond
// terms) in one launch: the blocks of the term lists follow one another (end[k]: first block past
// list k).  As launches of their own (up to seven, 6-9 us each whatever their length) they were the
// longest chain beside the charges on small molecules: 43 us with the repulsion for 26 atoms.
// ------------------------------------------------------------------------------------
struct TermArgs {
    TripSoA BM, AT;
    TorsSoA T, S;
    AngleSoA A;
    InvSoA I;
    XBSoA X;
    int end[7];
};
__global__ void __launch_bounds__(kBlock) k_terms(View V, TermArgs P)
{
    const int b = blockIdx.x;
    if (b < P.end[0]) batm_term(V, b, P.BM);
    else if (b < P.end[1]) torsion_term(V, b - P.end[0], P.T, 0);
    else if (b < P.end[2]) angle_term(V, b - P.end[1], P.A);
    else if (b < P.end[3]) inversion_term(V, b - P.end[2], P.I);
    else if (b < P.end[4]) torsion_term(V, b - P.end[3], P.S, 1);
    else if (b < P.end[5]) atm_term(V, b - P.end[4], P.AT);
    else xbond_term(V, b - P.end[5], P.X);
}

}  // namespace
