// Batched EEQ by conjugate gradients, one thread-block cluster per molecule (batches, and single
// molecules of at most kStageAtoms atoms).  Included inside namespace gfnff by engine.cu.
//
// The reduced matrix M of a molecule changes little between geometries, so its inverse at the
// set-up geometry (FP32, k_eeq_inv, once per set-up) is a preconditioner that needs 4 products there,
// 11-14 at 0.02 Angstrom of noise per coordinate, 14-19 at 0.06 and 16-27 at 0.12 (FP64 form, 26 to 302
// atoms; 20 for a C8 chain bent by 2 rad), where a factorisation has nr dependent steps: k_eeq_batch's
// Cholesky takes 230 us for 193 unknowns, latency all of it, and 27 products 108 us.  Here the cluster's CTAs hold equal row slices of M (FP64, built
// from the atoms) and of the inverse (FP32, one bulk copy while M is built) in shared memory for
// the whole solve; the vectors are replicated in every CTA, and a product's slice is stored into
// all of them (DSMEM), so an iteration is two products from shared memory and two cluster
// barriers.  Every CTA does the same arithmetic on the same vectors, so all take the same branches.
//
// Accuracy: the recurrence runs to a residual of 1e-15 max|b| (FP64 form; the rounding level of a
// direct solve) or 1e-4 of the absolute bar (mixed form: a refined solve's last correction also lands
// that far below the bar; ending at the bar itself, 3 to 4 products earlier and 9 to 14 us on 193
// unknowns, left errors of 1.6e-10 in the charges of conformers instead of 2e-14, where the
// tensor-core path has 2e-11), and the result is accepted on the true FP64
// residual b - M x: at most 1e-12 max|b|, or the bar.  A search direction with p M p <= 0 (M not
// positive definite) or too many iterations (M nearly singular, or far from the set-up geometry)
// leaves the molecule to a direct elimination in the same kernel (cg_direct), which always ends
// with a solution or a pivot that is not positive: every entry (single evaluations, device loops,
// MD, batches) gets the status that a factorisation gives.
//
// Definiteness: CG meets a negative direction only if its residual has a part along it (then it
// cannot converge past it: with positive Ritz values only, the residual polynomial grows on the
// negative axis), and symmetric molecules have right-hand sides without one (H2: b = 0).  So the
// solve starts from a pseudo-random vector u (cg_start), scaled so that M u is an eighth of b: every
// direction is in the first residual, whatever b is.  M u comes out of the build of M (with it and
// the larger first residual, 193 unknowns at 14 products: 65 -> 69 us, 25 unknowns the same; the counts
// do not change).
#pragma once

namespace {

struct CgArgs {
    const int* mols;        // molecules of this launch
    const int* roff;        // reduced-index offsets
    const int* red2atom;
    const int* anchor;
    const int* qlist;
    int nq;
    const double* q0;
    const float* pinv;      // inverses at the set-up geometry, rows of cg_ld(nr) floats
    const long long* poff;
    double* y;
    int* info;              // 0, or 1: not positive definite
    int* iters;             // largest number of products of the launch
    double tol_abs;         // > 0: the mixed form's bar
};

__host__ __device__ constexpr int cg_ld(int nr) { return (nr + 3) & ~3; }
// doubles of the vectors and the staged atoms: x r b p s w, two z, va, r in FP32; per atom x y z alpha diagonal Born
__host__ __device__ constexpr size_t cg_vec(int nr, int na) { return 10 * (size_t)nr + 6 * (size_t)na; }
__host__ __device__ constexpr size_t cg_smem(int nr, int na, int cs)
{
    const size_t rows = (nr + cs - 1) / cs;
    return 4 * rows * cg_ld(nr) + 8 * (rows * nr + cg_vec(nr, na)) + 4 * 2 * (size_t)nr + 32;
}

// atoms of one molecule in shared memory and the elements of its reduced matrix
struct CgMol {
    double *x, *y, *z, *al, *ad, *br, *va;
    int *red, *anc;
    bool single, born;
    double keps;
    __device__ double a(int i, int j) const
    {
        if (i == j) return ad[i];
        const double dx = x[i] - x[j], dy = y[i] - y[j], dz = z[i] - z[j];
        const double d2 = dx * dx + dy * dy + dz * dz, s = al[i] + al[j];
        // the square overflows above 1e154 bohr: 1/r = 0 (one comparison; a call to an out-of-line form, as in
        // k_eeq_M_tiles, took 93 registers instead of 76, which the side streams' kernels miss)
        const bool inf = __double2hiint(d2) == 0x7ff00000;
        const double ir = inf ? 0.0 : rsqrt_pos(d2), r = inf ? d2 : d2 * ir;
        double v = ir;
        if (d2 < 36.0 * s) v = erf(r * rsqrt_pos(s)) * ir;
        if (born) v += born_p16(keps, r, br[i], br[j]);
        return v;
    }
    __device__ double m(int r, int c) const
    {
        const int k = red[r], l = red[c];
        if (single) return ((a(k, l) - va[r]) - va[c]) + ad[anc[r]];
        const int ak = anc[r], al_ = anc[c];
        return a(k, l) - a(k, al_) - a(ak, l) + a(ak, al_);
    }
};

// stages the atoms of the molecule of reduced rows [r0, r0 + nr); the whole block calls it
__device__ void cg_stage(const View& V, const int* red2atom, const int* anchor, int r0, int nr, CgMol& S)
{
    const int2 rg = V.jr[red2atom[r0]];
    for (int i = threadIdx.x; i < rg.y - rg.x; i += blockDim.x) {
        const double4 p = V.pos[rg.x + i];
        S.x[i] = p.x; S.y[i] = p.y; S.z[i] = p.z;
        S.al[i] = V.alpeeq[rg.x + i];
        S.ad[i] = V.adiag[rg.x + i] + (V.brad ? V.bdiag[rg.x + i] : 0.0);
        S.br[i] = V.brad ? V.brad[rg.x + i] : 0.0;
    }
    for (int r = threadIdx.x; r < nr; r += blockDim.x) {
        const int k = red2atom[r0 + r];
        S.red[r] = k - rg.x;
        S.anc[r] = anchor[k] - rg.x;
    }
    S.single = anchor[red2atom[r0]] == anchor[red2atom[r0 + nr - 1]];
    S.born = V.brad != nullptr;
    S.keps = V.keps;
    __syncthreads();
    if (S.single)
        for (int r = threadIdx.x; r < nr; r += blockDim.x) S.va[r] = S.a(S.red[r], S.anc[r]);
    __syncthreads();
}

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
template <int CS>
__device__ __forceinline__ void cluster_barrier()
{
    if (CS == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
}
// stores v at the address p of this CTA's shared memory, in the CTA `rank` of the cluster
__device__ __forceinline__ void cluster_store(double* p, int rank, double v)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ void cluster_store_f(float* p, int rank, float v)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// out[row0 + q] = A v for the `rows` rows of this CTA's slice, stored into every CTA of the cluster:
// a warp takes four rows at a time, whose sums meet in 6 exchanges (reduce-scatter: lane l ends
// with row l / 8 of the four).  In the storage type of A: FP64 for M, FP32 for the inverse, whose
// products need no more (converting its elements took longer than the products).
template <int CS, class T>
__device__ __forceinline__ void cg_product(const T* A, int ld, int rows, int row0, int n, const T* v, double* out)
{
    constexpr unsigned full = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int q = 4 * warp; q < rows; q += 4 * nw) {
        T s[4] = {T(0), T(0), T(0), T(0)};
        const T* a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = A + (size_t)min(q + i, rows - 1) * ld;
#pragma unroll 4
        for (int c = lane; c < n; c += 32) {
            const T vc = v[c];
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] = fma(a[i][c], vc, s[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const bool up = (lane & 16) != 0;
            const T send = up ? s[i] : s[i + 2], keep = up ? s[i + 2] : s[i];
            s[i] = keep + __shfl_xor_sync(full, send, 16);
        }
        const bool up = (lane & 8) != 0;
        T t = (up ? s[1] : s[0]) + __shfl_xor_sync(full, up ? s[0] : s[1], 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(full, t, o);
        const int i = lane >> 3, dst = lane & 7;   // every lane of the row's eight stores to one CTA
        if (dst < CS && q + i < rows) {
            double* p = out + row0 + q + i;
            if (CS == 1) *p = (double)t;
            else cluster_store(p, dst, (double)t);
        }
    }
}

// |v| rounded up to FP32, as bits, which order as the values with NaN above all: a maximum over them
// keeps a NaN (fmaxf drops it), so that no bound on it holds
__device__ __forceinline__ unsigned abs_bits(double v) { return __float_as_uint(__double2float_ru(fabs(v))); }

// r.z, z.w and max |r|, the same in every warp
__device__ __forceinline__ void cg_dots(const double* r, const double* z, const double* w, int n, double& rz,
                                        double& zw, float& rmax)
{
    constexpr unsigned full = 0xffffffffu;
    double a = 0.0, b = 0.0;
    unsigned m = 0;
#pragma unroll 2
    for (int c = threadIdx.x & 31; c < n; c += 32) {
        const double rc = r[c], zc = z[c];
        a = fma(rc, zc, a);
        b = fma(zc, w[c], b);
        m = max(m, abs_bits(rc));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(full, a, o);
        b += __shfl_xor_sync(full, b, o);
    }
    rz = a;
    zw = b;
    rmax = __uint_as_float(__reduce_max_sync(full, m));
}

// max |v| and max |w|, the same in every warp
__device__ __forceinline__ void cg_max(const double* v, const double* w, int n, float& vmax, float& wmax)
{
    unsigned a = 0, b = 0;
    for (int c = threadIdx.x & 31; c < n; c += 32) {
        a = max(a, abs_bits(v[c]));
        b = max(b, abs_bits(w[c]));
    }
    vmax = __uint_as_float(__reduce_max_sync(0xffffffffu, a));
    wmax = __uint_as_float(__reduce_max_sync(0xffffffffu, b));
}

// positive, and far from the ends of the range (2^-1007 .. 2^1007): a scalar that rcp_pos takes
__device__ __forceinline__ bool cg_scalar(double v)
{
    return (unsigned)__double2hiint(v) - 0x01000000u < 0x7ee00000u - 0x01000000u;
}

// entry c of the start vector, in [-1, 1): the bits of c mixed by multiplications and shifts
__device__ __forceinline__ double cg_start(int c)
{
    unsigned h = (unsigned)(c + 1) * 2654435761u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    return (double)(int)h * 0x1p-31;
}

// Gauss-Jordan elimination of M x = b on the cluster's row slices, without pivoting (M symmetric: a
// pivot that is not positive means that it is not positive definite).  The owner of row k stores it
// into every CTA, two buffers in turn: the one of step k + 2 is written after the barrier of step
// k + 1, which every CTA reaches with its reads of step k done.  M and the slice of b are used up;
// x goes to y.  True if every pivot was positive, the same in every CTA.  A barrier a row: 38 us for
// 25 unknowns, 140 for 91, 350 for 193, 650 for 301 (CG at 0.03 Angstrom noise 30, 51, 69, 79).
template <int CS>
__device__ __noinline__ bool cg_direct(double* M, int rows, int row0, int nr, double* b, double* rowbuf, double* bk2,
                                       double* y)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    cluster_barrier<CS>();   // every CTA is done with its vectors
    for (int k = 0; k < nr; ++k) {
        double* row = rowbuf + (k & 1) * nr;
        double* bk = bk2 + (k & 1);
        if (k >= row0 && k < row0 + rows) {   // the owner
            const double* Mk = M + (size_t)(k - row0) * nr;
            for (int c = threadIdx.x; c < (nr - k) * CS; c += blockDim.x) {
                const int dst = CS == 1 ? 0 : c / (nr - k), j = k + (CS == 1 ? c : c % (nr - k));
                if (CS == 1) row[j] = Mk[j];
                else cluster_store(row + j, dst, Mk[j]);
            }
            if (threadIdx.x < CS) {
                if (CS == 1) *bk = b[k];
                else cluster_store(bk, threadIdx.x, b[k]);
            }
        }
        cluster_barrier<CS>();
        const double piv = row[k];
        if (!(piv > 0.0)) return false;
        const double inv = 1.0 / piv, bv = *bk;
        for (int q = warp; q < rows; q += nw) {
            if (row0 + q == k) continue;
            double* Mi = M + (size_t)q * nr;
            const double f = Mi[k] * inv;
            for (int j = k + 1 + lane; j < nr; j += 32) Mi[j] -= f * row[j];
            if (lane == 0) b[row0 + q] -= f * bv;
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < rows; q += blockDim.x) y[row0 + q] = b[row0 + q] / M[(size_t)q * nr + row0 + q];
    return true;
}

// products after which the elimination is the cheaper end (1.6-5.3 us a product against the times of
// cg_direct): a solve costs at most about twice the elimination
__device__ __forceinline__ int cg_max_iter(int nr) { return 20 + 2 * nr / 5; }

constexpr int kCgThreads = 512;   // at most: a warp per four rows of the slice (cg_threads)
inline int cg_threads(int nr, int cs) { return 64 * std::min(kCgThreads / 64, std::max(2, ((nr + cs - 1) / cs + 7) / 8)); }

template <int CS>
__global__ void __launch_bounds__(kCgThreads) k_eeq_cg(View V, CgArgs A)
{
    extern __shared__ __align__(16) unsigned char cg_raw[];
    __shared__ __align__(8) unsigned long long bar;
    const int mol = A.mols[blockIdx.x / CS];
    const int rank = CS == 1 ? 0 : (int)cluster_rank();
    const int r0 = A.roff[mol], nr = A.roff[mol + 1] - r0;
    if (nr == 0) {   // one atom per fragment: nothing to solve (uniform over the cluster)
        if (threadIdx.x == 0 && rank == 0) A.info[mol] = 0;
        return;
    }
    const int rows_max = (nr + CS - 1) / CS, row0 = min(nr, rank * rows_max), rows = min(nr, row0 + rows_max) - row0;
    const int ld = cg_ld(nr);
    const int2 rg = V.jr[A.red2atom[r0]];
    const int na = rg.y - rg.x;
    const float* Pm = reinterpret_cast<const float*>(cg_raw);
    double* M = reinterpret_cast<double*>(cg_raw + 4 * (size_t)rows_max * ld);   // ld is a multiple of 4
    double* x = M + (size_t)rows_max * nr;
    double *r = x + nr, *b = r + nr, *p = b + nr, *s = p + nr, *w = s + nr, *z2 = w + nr;
    float* rf = reinterpret_cast<float*>(z2 + 2 * nr);   // nr floats in nr doubles
    CgMol S;
    S.va = z2 + 3 * nr;
    S.x = S.va + nr; S.y = S.x + na; S.z = S.y + na; S.al = S.z + na; S.ad = S.al + na; S.br = S.ad + na;
    S.red = reinterpret_cast<int*>(S.br + na);
    S.anc = S.red + nr;
    if (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if (rows > 0) {
            const unsigned bytes = 4u * (unsigned)(rows * ld);
            mbar_expect_tx(&bar, bytes);
            bulk_copy(cg_raw, A.pinv + A.poff[mol] + (size_t)row0 * ld, bytes, &bar);
        }
    }
    for (int q = threadIdx.x; q < nr; q += blockDim.x) x[q] = cg_start(q);
    cg_stage(V, A.red2atom, A.anchor, r0, nr, S);
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        // M u of the slice is stored into every CTA once all of them run
        if (CS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        if (CS == 1) {   // each element once, into both triangles
            for (int q = warp; q < rows; q += nw)
                for (int c = lane; c <= q; c += 32) M[(size_t)q * nr + c] = M[(size_t)c * nr + q] = S.m(q, c);
        } else {
            for (int q = warp; q < rows; q += nw) {
                double g = 0.0;
                for (int c = lane; c < nr; c += 32) {
                    const double v = S.m(row0 + q, c);
                    M[(size_t)q * nr + c] = v;
                    g = fma(v, x[c], g);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
                if (lane < CS) cluster_store(w + row0 + q, lane, g);
            }
        }
    }
    for (int q = threadIdx.x; q < nr; q += blockDim.x) {
        const int k = A.red2atom[r0 + q];
        b[q] = eeq_rhs_atom(V, k, A.qlist, A.nq, A.q0) - eeq_rhs_atom(V, A.anchor[k], A.qlist, A.nq, A.q0);
    }
    if (rows > 0) mbar_wait(&bar, 0);   // bounded; without the inverse the solve fails its checks
    cluster_barrier<CS>();
    if (CS == 1) {
        cg_product<CS, double>(M, nr, rows, row0, nr, x, w);
        __syncthreads();
    }
    float bmax, umax;
    cg_max(b, w, nr, bmax, umax);
    {
        // (mixed form: at least 1e-4 where b is smaller than that, far above the residual to reach)
        const float size = A.tol_abs > 0.0 ? fmaxf(bmax, 1e7f * (float)A.tol_abs) : bmax;
        const double t = size > 0.f ? (double)(0.125f * size / umax) : 1.0;
        for (int q = threadIdx.x; q < nr; q += blockDim.x) {
            x[q] *= t;
            r[q] = b[q] - t * w[q];
            rf[q] = (float)r[q];
        }
        __syncthreads();
    }
    // Single-reduction CG (A. T. Chronopoulos, C. W. Gear, J. Comput. Appl. Math. 25 (1989)
    // 153-168): the products P r and M z follow one another, and all scalars of an iteration come
    // from one pass over r, z and w = M z; M p is carried along as s.  A CTA stores its slice of the
    // next z while another may still read the last one, so z alternates between two buffers; w is
    // stored only after the barrier that follows z, which every CTA reaches with its reads done.
    double rz, zw, irz_old = 0.0, ialpha = 0.0, dummy;   // 1 / the last r.z and alpha
    float rmax;
    const float scale = bmax > 0.f ? bmax : umax;
    const float stop = A.tol_abs > 0.0 ? 1e-4f * (float)A.tol_abs : 1e-15f * scale;
    const float accept = A.tol_abs > 0.0 ? (float)A.tol_abs : 1e-12f * scale;
    const int max_iter = cg_max_iter(nr);
    int it = 0, state = -1;   // -1: running, 0: solved, else left to the elimination
    bool start = true;
    while (state < 0) {
        double* z = z2 + (it & 1) * nr;
        cg_product<CS, float>(Pm, ld, rows, row0, nr, rf, z);
        cluster_barrier<CS>();
        cg_product<CS, double>(M, nr, rows, row0, nr, z, w);
        cluster_barrier<CS>();
        ++it;
        cg_dots(r, z, w, nr, rz, zw, rmax);
        if (!start && (rmax <= stop || it >= max_iter)) {   // the true residual decides
            cluster_barrier<CS>();   // every CTA has read w
            cg_product<CS, double>(M, nr, rows, row0, nr, x, w);
            cluster_barrier<CS>();
            for (int q = threadIdx.x; q < nr; q += blockDim.x) {
                r[q] = b[q] - w[q];
                rf[q] = (float)r[q];
            }
            __syncthreads();
            cg_dots(r, r, r, nr, dummy, zw, rmax);
            if (rmax <= accept) state = 0;
            else if (it >= max_iter) state = 3;
            start = true;
            continue;
        }
        const double beta = start ? 0.0 : rz * irz_old;
        const double pmp = start ? zw : zw - beta * rz * ialpha;
        if (!(cg_scalar(pmp) && cg_scalar(rz))) {   // not positive definite, or not a number
            state = 1;
            break;
        }
        const double alpha = rz * rcp_pos(pmp);   // a division is 0.25 us of dependent operations in every iteration
        irz_old = rcp_pos(rz);
        ialpha = pmp * irz_old;
        __syncthreads();   // every warp has read r, z and w
        for (int q = threadIdx.x; q < nr; q += blockDim.x) {
            const double pq = start ? z[q] : z[q] + beta * p[q], sq = start ? w[q] : w[q] + beta * s[q];
            p[q] = pq;
            s[q] = sq;
            x[q] += alpha * pq;
            r[q] -= alpha * sq;
            rf[q] = (float)r[q];
        }
        start = false;
        __syncthreads();
    }
    if (state != 0) {
        const bool ok = cg_direct<CS>(M, rows, row0, nr, b, z2, w, A.y + r0);
        state = ok ? 0 : 1;
    } else if (rank == 0) {
        __syncthreads();
        for (int q = threadIdx.x; q < nr; q += blockDim.x) A.y[r0 + q] = bmax == 0.f ? 0.0 : x[q];
    }
    if (rank == 0 && threadIdx.x == 0) {
        A.info[mol] = state;
        atomicMax(A.iters, it);
    }
    cluster_barrier<CS>();   // no CTA leaves while another may store into it
}

// FP32 inverse of the reduced matrix at the current geometry, one cluster per molecule as in k_eeq_cg
// (Gauss-Jordan in place on row slices in shared memory, no pivoting: M is positive definite).  The
// owner of row k stores it into every CTA (two buffers in turn, so that one barrier a step is
// enough).  A pivot that is not positive leaves the inverse diagonal instead.
constexpr size_t inv_smem(int nr, int na, int cs)
{
    return 4 * ((size_t)(nr + cs - 1) / cs + 2) * cg_ld(nr) + 8 * ((size_t)nr + 6 * (size_t)na) + 8 * (size_t)nr + 32;
}
template <int CS>
__global__ void __launch_bounds__(512) k_eeq_inv(View V, CgArgs A, float* pinv)
{
    extern __shared__ __align__(16) unsigned char inv_raw[];
    __shared__ float diag[kStageAtoms];
    const int m = A.mols[blockIdx.x / CS];
    const int rank = CS == 1 ? 0 : (int)cluster_rank();
    const int r0 = A.roff[m], nr = A.roff[m + 1] - r0;
    if (nr == 0) return;   // uniform over the cluster
    const int rows_max = (nr + CS - 1) / CS, row0 = min(nr, rank * rows_max), rows = min(nr, row0 + rows_max) - row0;
    const int ld = cg_ld(nr);
    const int2 rg = V.jr[A.red2atom[r0]];
    const int na = rg.y - rg.x;
    float* M = reinterpret_cast<float*>(inv_raw);
    float* rowbuf = M + (size_t)rows_max * ld;
    double* st = reinterpret_cast<double*>(rowbuf + 2 * ld);
    CgMol S;
    S.va = st;
    S.x = S.va + nr; S.y = S.x + na; S.z = S.y + na; S.al = S.z + na; S.ad = S.al + na; S.br = S.ad + na;
    S.red = reinterpret_cast<int*>(S.br + na);
    S.anc = S.red + nr;
    cg_stage(V, A.red2atom, A.anchor, r0, nr, S);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int q = warp; q < rows; q += nw)
        for (int c = lane; c < nr; c += 32) {
            const float v = (float)S.m(row0 + q, c);
            M[(size_t)q * ld + c] = v;
            if (c == row0 + q) diag[q] = v;
        }
    cluster_barrier<CS>();
    bool bad = false;
    for (int k = 0; k < nr; ++k) {
        float* row = rowbuf + (k & 1) * ld;
        if (k >= row0 && k < row0 + rows)   // the owner
            for (int c = threadIdx.x; c < nr * CS; c += blockDim.x) {
                const int dst = CS == 1 ? 0 : c / nr, j = CS == 1 ? c : c % nr;
                const float v = M[(size_t)(k - row0) * ld + j];
                if (CS == 1) row[j] = v;
                else cluster_store_f(row + j, dst, v);
            }
        cluster_barrier<CS>();
        if (!(row[k] > 0.f)) {   // the same row in every CTA
            bad = true;
            break;
        }
        const float ip = 1.f / row[k];
        for (int q = warp; q < rows; q += nw) {
            float* Mi = M + (size_t)q * ld;
            const float f = Mi[k] * ip;
            const bool own = row0 + q == k;
            __syncwarp();
            for (int j = lane; j < nr; j += 32)
                Mi[j] = own ? (j == k ? ip : row[j] * ip) : (j == k ? -f : Mi[j] - f * row[j]);
        }
        __syncthreads();
    }
    float* out = pinv + A.poff[m] + (size_t)row0 * ld;
    __syncthreads();
    for (int q = warp; q < rows; q += nw)
        for (int c = lane; c < ld; c += 32) {
            float v = c < nr ? M[(size_t)q * ld + c] : 0.f;
            if (bad) v = c == row0 + q ? (diag[q] > 0.f ? 1.f / diag[q] : 1.f) : 0.f;
            out[(size_t)q * ld + c] = v;
        }
    cluster_barrier<CS>();
}

}  // namespace
