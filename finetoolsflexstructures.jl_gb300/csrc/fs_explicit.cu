// Explicit central-difference time stepping
// (examples/shells/dynamics/homogeneous/explicit/plate_expl_examples.jl:61-94,
// _cd_loop!, with mass-proportional damping C and the external force of the
// example's force!: F(t) = g(t) Fmag, a fixed load vector times a scalar time
// function, given as its values at the step times):
//
//   U += dt V + dt^2/2 A;  F = g(t) Fmag;  E = K U;  F -= E + C (V + dt/2 A);
//   V += dt/2 A;  A = invMC F;  V += dt/2 A
//
// The product K U, the force, acceleration and velocity of a row and the next
// step's displacement are one kernel (k_cd_step) on the 6x6 node blocks of
// K (block rows = the neighbour lists of the pattern, filled from the CSR matrix
// once at set-up) against a node-padded copy of U; two kernels, the displacement
// update and a row-parallel product on the CSR arrays, when no pattern of the
// current mesh is at hand.  The displacement
// and velocity sums carry Kahan compensation terms so
// that a long run in double does not drift.  With FS_FP64 the restoring force
// K U is formed in double.  With FS_MIXED it is formed in float: the
// displacement kernel also writes a float copy of U and the product runs on
// float values (a double product would spend one double conversion and one
// double FMA per stored value, the scarcest pipe on GB300); the force,
// acceleration and velocity updates stay in double.  With FS_MIXED_COMP each
// value is kept as its float rounding plus the rounding's residual in bf16
// (K to about 33 bits, 6 bytes a value), the displacement copy is a float
// pair (hi, lo: U to about 48 bits), and K U is summed in compensated float
// sums (Dot2 on the float value times hi; the products with lo and with the
// residual added to the error term).  A row of K U is a small remainder of
// its terms for a smooth displacement field, so the float copy of U, the
// float sum and the float rounding of K each leave errors far above their
// own 6e-8 in it (measured in that order of size).  The step loop is
// captured once into a CUDA graph and replayed.
#include <cuda_bf16.h>

#include <algorithm>
#include <vector>

#include "fs_elem_common.cuh"

namespace fs {

static const int CD_TPB = 256;
static const int CD_LANES = 8;  // lanes per CSR row
static const int CD_GRAPH_STEPS = 64;   // even: a graph ends on the displacement copy it began with
// block step: threads of a block, the most in one block an SM, and the threads
// an SM up to which a mesh is small (launch_block_step)
static const int CD_BLOCK_TPB = 64, CD_ONE_BLOCK_TPB = 512;
constexpr int cd_small_tpb(int precision) { return precision == FS_MIXED ? 512 : 128; }

// one entry of a displacement copy: double, float, or the float pair (hi, lo)
// with hi = U rounded and lo = the rest rounded
__device__ __forceinline__ void store_disp(double *p, double t) { *p = t; }
__device__ __forceinline__ void store_disp(float *p, double t) { *p = (float)t; }
__device__ __forceinline__ void store_disp(float2 *p, double t)
{
    const float h = (float)t;
    *p = make_float2(h, (float)(t - (double)h));
}

__device__ __forceinline__ void kahan_sum(double &s, double &c, double y)  // y: increment - c
{
    const double t = s + y;
    c = (t - s) - y;
    s = t;
}
// the displacement update of a dof; the new displacement
__device__ __forceinline__ double disp_sum(double &u, double &cu, double v, double a, double dt, double dt2_2)
{
    kahan_sum(u, cu, fma(dt, v, fma(dt2_2, a, -cu)));
    return u;
}

__global__ void k_cd_disp(int64_t n, double dt, double dt2_2, double *U, double *cU, const double *V,
                          const double *A, float *U32)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double y = (dt * V[i] + dt2_2 * A[i]) - cU[i];
    double u = U[i];
    double t = u + y;
    cU[i] = (t - u) - y;
    U[i] = t;
    if (U32) U32[i] = (float)t;
}

// the CSR path's displacement update writing the float-pair copy
__global__ void k_cd_disp_pair(int64_t n, double dt, double dt2_2, double *U, double *cU, const double *V,
                               const double *A, float2 *U2)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double y = (dt * V[i] + dt2_2 * A[i]) - cU[i];
    double u = U[i];
    double t = u + y;
    cU[i] = (t - u) - y;
    U[i] = t;
    store_disp(U2 + i, t);
}

// the displacement update of k_cd_step alone, writing the node-padded copy read
// by the block product (entries of excluded dofs stay zero)
template <class VT>
__global__ void k_cd_disp_pad(int64_t n, double dt, double dt2_2, double *U, double *cU, const double *V,
                              const double *A, const int32_t *pad_of_dof, VT *xp)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double u = U[i], cu = cU[i];
    const double t = disp_sum(u, cu, V[i], A[i], dt, dt2_2);
    cU[i] = cu;
    U[i] = t;
    const int32_t q = pad_of_dof[i];
    if (q >= 0) store_disp(xp + q, t);
}

// six contiguous values (8-byte aligned floats, 16-byte aligned doubles)
__device__ __forceinline__ void load6(const float *p, float v[6])
{
    const float2 *q = reinterpret_cast<const float2 *>(p);
    const float2 a = q[0], b = q[1], c = q[2];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}
__device__ __forceinline__ void load6(const double *p, double v[6])
{
    const double2 *q = reinterpret_cast<const double2 *>(p);
    const double2 a = q[0], b = q[1], c = q[2];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}

__device__ __forceinline__ void load6(const float2 *p, float2 v[6])
{
    const float4 *q = reinterpret_cast<const float4 *>(p);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 a = q[k];
        v[2 * k] = make_float2(a.x, a.y);
        v[2 * k + 1] = make_float2(a.z, a.w);
    }
}

// External load of step j of the current batch: the state's step index plus
// j + 1 selects g (zero past the table); null Fmag: no load.
struct CdLoad {
    const double *Fmag;
    const double *mul;
    int64_t nmul;
    const int64_t *step;
    int j;
    __device__ __forceinline__ double at(int64_t row) const
    {
        if (!Fmag) return 0.0;
        const int64_t s = *step + j + 1;
        const double g = s < nmul ? mul[s] : 0.0;
        return g * Fmag[row];
    }
};

__global__ void k_step_advance(int64_t *step, int64_t nsteps) { *step += nsteps; }

__device__ __forceinline__ void kahan_add(double &s, double &c, double incr)
{
    double y = incr - c;
    double t = s + y;
    c = (t - s) - y;
    s = t;
}

// VT: value type of K and of the displacement copy the product reads
template <class VT>
__global__ void __launch_bounds__(CD_TPB) k_cd_rows(int64_t n, const int64_t *rowptr, const int32_t *colidx,
                                                  const VT *vals, const VT *Uk, double *V, double *cV,
                                                  double *A, const double *C, const double *invMC, double dt_2,
                                                  CdLoad ld)
{
    int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / CD_LANES;
    const int sub = threadIdx.x & (CD_LANES - 1);
    const unsigned mask = 0xffffffffu;
    VT sv = 0;
    if (row < n) {
        for (int64_t k = rowptr[row] + sub; k < rowptr[row + 1]; k += CD_LANES) sv += vals[k] * Uk[colidx[k]];
    }
#pragma unroll
    for (int o = CD_LANES / 2; o > 0; o >>= 1) sv += __shfl_xor_sync(mask, sv, o);
    double s = (double)sv;
    if (row < n && sub == 0) {
        double a = A[row], v = V[row], cv = cV[row];
        double f = ld.at(row);
        f -= s + C[row] * (v + dt_2 * a);
        kahan_add(v, cv, dt_2 * a);
        a = invMC[row] * f;
        kahan_add(v, cv, dt_2 * a);
        A[row] = a;
        V[row] = v;
        cV[row] = cv;
    }
}

// compensated accumulation of (kv + kr) * (xh + xl) into (s, c): Dot2 on
// kv * xh, the small products kv * xl and kr * xh added to the error term
// (kr * xl is below the error of the result)
__device__ __forceinline__ void acc_pair(float &s, float &c, float kv, float kr, float2 x)
{
    dot2_step(s, c, kv, x.x);
    c = __fmaf_rn(kv, x.y, c);
    c = __fmaf_rn(kr, x.x, c);
}
// (s1, c1) += (s2, c2) without losing the rounding of s1 + s2 (TwoSum)
__device__ __forceinline__ void add_pair(float &s, float &c, float s2, float c2)
{
    const float t = __fadd_rn(s, s2);
    const float z = __fsub_rn(t, s);
    const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(s2, z));
    c = __fadd_rn(__fadd_rn(c, c2), e);
    s = t;
}

// The CSR product of k_cd_rows with the float-pair displacement copy and the
// compensated float sum (FS_MIXED_COMP).
__global__ void __launch_bounds__(CD_TPB) k_cd_rows_comp(int64_t n, const int64_t *rowptr, const int32_t *colidx,
                                                       const float *vals, const __nv_bfloat16 *res,
                                                       const float2 *Uk, double *V, double *cV, double *A,
                                                       const double *C, const double *invMC, double dt_2, CdLoad ld)
{
    int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / CD_LANES;
    const int sub = threadIdx.x & (CD_LANES - 1);
    const unsigned mask = 0xffffffffu;
    float s = 0.f, c = 0.f;
    if (row < n) {
        for (int64_t k = rowptr[row] + sub; k < rowptr[row + 1]; k += CD_LANES) acc_pair(s, c, vals[k], __bfloat162float(res[k]), Uk[colidx[k]]);
    }
#pragma unroll
    for (int o = CD_LANES / 2; o > 0; o >>= 1) {
        const float s2 = __shfl_xor_sync(mask, s, o), c2 = __shfl_xor_sync(mask, c, o);
        add_pair(s, c, s2, c2);
    }
    if (row < n && sub == 0) {
        const double sv = (double)s + (double)c;
        double a = A[row], v = V[row], cv = cV[row];
        double f = ld.at(row);
        f -= sv + C[row] * (v + dt_2 * a);
        kahan_add(v, cv, dt_2 * a);
        a = invMC[row] * f;
        kahan_add(v, cv, dt_2 * a);
        A[row] = a;
        V[row] = v;
        cV[row] = cv;
    }
}

// float values and their bf16 residuals: hi = float(v), res = v - hi
__device__ __forceinline__ void split_value(double v, float &hi, __nv_bfloat16 &res)
{
    hi = (float)v;
    res = __float2bfloat16_rn((float)(v - (double)hi));
}

__global__ void k_split_values(int64_t n, const double *src, float *hi, __nv_bfloat16 *res)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) split_value(src[i], hi[i], res[i]);
}

// ---------------------------------------------------------------------------
// the step on the 6x6 node blocks
// ---------------------------------------------------------------------------
// One thread owns two dofs of a node (three threads a node) and does their whole
// step: the two rows of K U, the force, acceleration and velocity, and, but for
// the last step before the state is looked at, the displacement of the next step,
// written to the other of two displacement copies.  A row's products are added
// in the order of the neighbours and, within a block, of the columns.
//
// K is symmetric, so each off-diagonal block is stored once, with the lower
// node's dofs as rows; CdItem names a row's blocks.  The second reader finds a
// block in L2 as long as the nodes between the two (the band of the numbering)
// fit there, which leaves half of the reads from memory.  A block lies in 2x2
// tiles (of 16 bytes in float, 32 in double; the bf16 residuals likewise, 8
// bytes), three tiles a thread: a tile row for a block read as stored, a tile
// column with the tiles transposed for the other reading, so that both take
// the same wide loads.
//
// What bounds it: with FS_FP64 the double pipe (2 operations per clock and SM),
// 6 operations per block of a row and about 14 a dof (conversions between float
// and double are done on the bits, the two velocity increments in one
// compensated sum); otherwise the load pipe (a warp's loads touch 11 blocks,
// 1.6 lines each) and memory.  A step on quads, 512 x 512: 128 us with
// FS_MIXED_COMP (470 MB, 3.7 TB/s, load pipe 63 %), 187 FS_FP64, 84 FS_MIXED; in
// two kernels that read every block as it is, 168, 218 and 108.
struct CdItem {
    int32_t node;   // the neighbour
    uint32_t pos;   // 2 * its block + (1: read it transposed)
};

// two neighbouring entries (16, 8 or 4 bytes) of a block and of its residual
template <int PREC> struct CdTypes {
    using V = float;       // block values
    using X = float;       // displacement copy
};
template <> struct CdTypes<FS_FP64> {
    using V = double;
    using X = double;
};
template <> struct CdTypes<FS_MIXED_COMP> {
    using V = float;
    using X = float2;
};

// position of entry (i, j) of a block
__host__ __device__ __forceinline__ int tile_entry(int i, int j) { return ((i >> 1) * 3 + (j >> 1)) * 4 + (i & 1) * 2 + (j & 1); }

// rows 2p and 2p + 1 of a block: tile q holds columns 2q, 2q + 1
template <int PREC> struct CdRows {
    float4 t[3];
    uint2 r[PREC == FS_MIXED_COMP ? 3 : 1];
    __device__ __forceinline__ void load(const float *blk, const __nv_bfloat16 *res, uint32_t pos, int p)
    {
        const int64_t at = (int64_t)(pos >> 1) * 9 + ((pos & 1) ? p : 3 * p);
        const int step = (pos & 1) ? 3 : 1;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            t[q] = __ldg(reinterpret_cast<const float4 *>(blk) + at + q * step);
            if constexpr (PREC == FS_MIXED_COMP) r[q] = __ldg(reinterpret_cast<const uint2 *>(res) + at + q * step);
        }
    }
    __device__ __forceinline__ void get(bool tr, int q, float a[4]) const
    {
        a[0] = t[q].x;
        a[1] = tr ? t[q].z : t[q].y;
        a[2] = tr ? t[q].y : t[q].z;
        a[3] = t[q].w;
    }
    __device__ __forceinline__ void get_residual(bool tr, int q, float a[4]) const
    {
        const unsigned b = __byte_perm(r[q].x, r[q].y, tr ? 0x5410 : 0x3210);  // first row's two
        const unsigned d = __byte_perm(r[q].x, r[q].y, tr ? 0x7632 : 0x7654);
        a[0] = __uint_as_float(b << 16);
        a[1] = __uint_as_float(b & 0xffff0000u);
        a[2] = __uint_as_float(d << 16);
        a[3] = __uint_as_float(d & 0xffff0000u);
    }
};
template <> struct CdRows<FS_FP64> {
    double2 t[3][2];
    __device__ __forceinline__ void load(const double *blk, const __nv_bfloat16 *, uint32_t pos, int p)
    {
        const int64_t at = (int64_t)(pos >> 1) * 9 + ((pos & 1) ? p : 3 * p);
        const int step = (pos & 1) ? 3 : 1;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const double2 *s = reinterpret_cast<const double2 *>(blk) + 2 * (at + q * step);
            t[q][0] = __ldg(s);
            t[q][1] = __ldg(s + 1);
        }
    }
    __device__ __forceinline__ void get(bool tr, int q, double a[4]) const
    {
        a[0] = t[q][0].x;
        a[1] = tr ? t[q][1].x : t[q][0].y;
        a[2] = tr ? t[q][0].y : t[q][1].x;
        a[3] = t[q][1].y;
    }
};

// the double nearest a float, on the bits (a conversion instruction takes the double pipe)
__device__ __forceinline__ double widen(float f)
{
    const unsigned b = __float_as_uint(f), e = (b >> 23) & 0xff;
    if (e == 0 || e == 0xff) return (double)f;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
}
// t as the float pair of store_disp: hi = t rounded to nearest even, lo = the
// rest, rounded; on the bits where hi and the scale of lo are normal floats
__device__ __forceinline__ float2 split_disp(double t)
{
    const unsigned h = (unsigned)__double2hiint(t), l = (unsigned)__double2loint(t), e = (h >> 20) & 0x7ff;
    if (e - 952u >= 190u) {
        float2 v;
        store_disp(&v, t);
        return v;
    }
    const unsigned keep = (((h & 0x7fffffffu) - (896u << 20)) << 3) | (l >> 29);   // hi, truncated
    const unsigned rest = l & 0x1fffffffu;                                       // below its last place
    const unsigned up = (rest + 0x0fffffffu + (keep & 1)) >> 29;
    const unsigned sign = h & 0x80000000u;
    const float scale = __uint_as_float(sign | (e - 1075u + 127u) << 23);        // of t's last place
    return make_float2(__uint_as_float(sign | (keep + up)), (float)((int)rest - (int)(up << 29)) * scale);
}
__device__ __forceinline__ void put_disp(double *p, double t) { *p = t; }
__device__ __forceinline__ void put_disp(float *p, double t) { *p = (float)t; }
__device__ __forceinline__ void put_disp(float2 *p, double t) { *p = split_disp(t); }

struct CdStep {
    int64_t nnodes, n;
    const int32_t *dof;
    const int64_t *off;    // a node's items
    const CdItem *item;
    const void *blk;
    const __nv_bfloat16 *res;
    double *U, *cU, *V, *cV, *A;
    const double *C, *invMC;
    double dt, dt2_2, dt_2;
};

// NEXT: also the displacement of the next step, copied to `xn`; UN blocks at a
// time, their loads and those of the next ones' items in flight together.  The
// kernel may start while the step before still writes `xp`: no restrict, which
// would let the compiler take it for read-only, and only plain loads of it
template <int PREC, bool NEXT, int UN>
__global__ void __launch_bounds__(UN == 1 ? CD_ONE_BLOCK_TPB : cd_small_tpb(PREC)) k_cd_step(CdStep s, const typename CdTypes<PREC>::X *xp,
                                                          typename CdTypes<PREC>::X *xn, CdLoad ld)
{
    using V = typename CdTypes<PREC>::V;
    const int64_t th = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, r = th / 3;
    const int p = (int)(th - 3 * r);
    if (r >= s.nnodes) return;
    int64_t b = s.off[r];
    const int64_t b1 = s.off[r + 1];
    CdItem it[UN];
    CdRows<PREC> k[UN];
#pragma unroll
    for (int u = 0; u < UN; u++)
        if (b + u < b1) it[u] = s.item[b + u];
#pragma unroll
    for (int u = 0; u < UN; u++)
        if (b + u < b1) k[u].load((const V *)s.blk, s.res, it[u].pos, p);
    const int32_t d[2] = {s.dof[(int64_t)(2 * p) * s.nnodes + r], s.dof[(int64_t)(2 * p + 1) * s.nnodes + r]};
    // what the step before wrote is read from here on
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();  // (here: one step ahead, no more)
    V sum[2] = {0, 0}, err[2] = {0, 0};
    while (b < b1) {
        CdItem nx[UN];
#pragma unroll
        for (int u = 0; u < UN; u++)
            if (b + UN + u < b1) nx[u] = s.item[b + UN + u];
        typename CdTypes<PREC>::X x[UN][6];
#pragma unroll
        for (int u = 0; u < UN; u++)
            if (b + u < b1) load6(xp + (int64_t)it[u].node * 6, x[u]);
#pragma unroll
        for (int u = 0; u < UN; u++)
            if (b + u < b1) {
                const bool tr = it[u].pos & 1;
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    V a[4];
                    k[u].get(tr, q, a);
                    if constexpr (PREC == FS_MIXED_COMP) {
                        float e[4];
                        k[u].get_residual(tr, q, e);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            acc_pair(sum[i], err[i], a[2 * i], e[2 * i], x[u][2 * q]);
                            acc_pair(sum[i], err[i], a[2 * i + 1], e[2 * i + 1], x[u][2 * q + 1]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            sum[i] += a[2 * i] * x[u][2 * q];
                            sum[i] += a[2 * i + 1] * x[u][2 * q + 1];
                        }
                    }
                }
            }
        b += UN;
#pragma unroll
        for (int u = 0; u < UN; u++)
            if (b + u < b1) {
                it[u] = nx[u];
                k[u].load((const V *)s.blk, s.res, it[u].pos, p);
            }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (d[i] > s.n) continue;
        const int64_t row = d[i] - 1;
        double kx;
        if constexpr (PREC == FS_FP64) kx = sum[i];
        else if constexpr (PREC == FS_MIXED_COMP) kx = widen(sum[i]) + widen(err[i]);
        else kx = widen(sum[i]);
        const double a0 = s.A[row];
        double v = s.V[row], cv = s.cV[row];
        const double e = kx + s.C[row] * (v + s.dt_2 * a0);
        const double a = s.invMC[row] * (ld.Fmag ? ld.at(row) - e : -e);
        kahan_sum(v, cv, fma(s.dt_2, a0 + a, -cv));
        s.A[row] = a;
        s.V[row] = v;
        s.cV[row] = cv;
        if constexpr (NEXT) {
            double u = s.U[row], cu = s.cU[row];
            put_disp(xn + r * 6 + 2 * p + i, disp_sum(u, cu, v, a, s.dt, s.dt2_2));
            s.U[row] = u;
            s.cU[row] = cu;
        }
    }
}

// block `pos` of node r and its neighbour in slot s, entry (i, j) = K[dof(r,
// i), dof(nbr, j)] (zero where either dof is excluded or the matrix has no
// entry), and the items of the node's slots; one warp a node.  first_upper:
// only the blocks of the node itself and its higher neighbours are stored, from
// first_upper[r] on, and status tells of values that differ from their mirror.
__device__ __forceinline__ double find_entry(const int64_t *rowptr, const int32_t *colidx, const double *vals, int32_t d, int32_t e)
{
    int64_t lo = rowptr[d - 1], hi = rowptr[d] - 1;
    while (lo <= hi) {
        const int64_t mid = (lo + hi) >> 1;
        const int32_t cc = colidx[mid];
        if (cc == e - 1) return vals[mid];
        if (cc < e - 1) lo = mid + 1; else hi = mid - 1;
    }
    return 0.0;
}
__device__ __forceinline__ int slot_of(const int32_t *nbr, int n, int32_t node)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (nbr[mid] < node) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__global__ void k_cd_fill(int64_t nnodes, int64_t n, int precision, const int32_t *dof, const int64_t *rowptr,
                          const int32_t *colidx, const double *vals, const int64_t *nbr_off, const int32_t *nbr,
                          const int64_t *first_upper, CdItem *item, void *blk, __nv_bfloat16 *res, int *status)
{
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= nnodes) return;
    const int64_t off = nbr_off[r];
    const int ns = (int)(nbr_off[r + 1] - off);
    const int s0 = first_upper ? slot_of(nbr + off, ns, (int32_t)r) : 0;
    const int64_t b0 = first_upper ? first_upper[r] : off;
    for (int s = lane; s < ns; s += 32) {
        const int32_t o = nbr[off + s];
        int64_t b = b0 + (s - s0);
        if (s < s0) {
            const int64_t oo = nbr_off[o];
            const int on = (int)(nbr_off[o + 1] - oo);
            b = first_upper[o] + slot_of(nbr + oo, on, (int32_t)r) - slot_of(nbr + oo, on, o);
        }
        item[off + s] = CdItem{o, (uint32_t)b << 1 | (s < s0 ? 1u : 0u)};
    }
    for (int idx = lane; idx < (ns - s0) * 36; idx += 32) {
        const int s = s0 + idx / 36, ij = idx % 36, i = ij / 6, j = ij - 6 * i;
        const int32_t d = dof[(int64_t)i * nnodes + r];
        const int32_t e = dof[(int64_t)j * nnodes + nbr[off + s]];
        double v = 0.0;
        if (d <= n && e <= n) {
            v = find_entry(rowptr, colidx, vals, d, e);
            if (first_upper &&
                __double_as_longlong(v) != __double_as_longlong(find_entry(rowptr, colidx, vals, e, d)))
                atomicOr(status, DEV_UNSYMMETRIC);
        }
        const int64_t at = (b0 + s - s0) * 36 + tile_entry(i, j);
        if (precision == FS_FP64)
            ((double *)blk)[at] = v;
        else if (precision == FS_MIXED_COMP)
            split_value(v, ((float *)blk)[at], res[at]);
        else
            ((float *)blk)[at] = (float)v;
    }
}

// dofs that no node has
__global__ void k_cd_unowned(int64_t n, const int32_t *pad_of_dof, int *status)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && pad_of_dof[i] < 0) atomicOr(status, DEV_UNOWNED);
}

__global__ void k_pad_map(int64_t nnodes, int64_t n, const int32_t *dof, int32_t *pad_of_dof)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 6 * nnodes) return;
    const int64_t r = q / 6;
    const int k = (int)(q - 6 * r);
    const int32_t d = dof[(int64_t)k * nnodes + r];
    if (d <= n) pad_of_dof[d - 1] = (int32_t)q;
}

static CdStep cd_step(fs_ctx *c)
{
    auto &x = c->ex;
    return CdStep{x.nnodes, x.n, c->mesh.dof, c->pat.nbr_off, (const CdItem *)x.item, x.blk, (const __nv_bfloat16 *)x.res,
                  x.U, x.cU, x.V, x.cV, x.A, x.C, x.invMC, x.dt, x.dt * x.dt / 2, x.dt / 2};
}

// One step on the blocks, reading displacement copy `from`.  In a small mesh
// the loads of a thread, one after the other, make the time, so it has four
// blocks in flight (triangles, 60 x 60, FP64: 8.1 us a step, 9.6 with one; two
// kernels took 9.2); in a larger one other warps fill that time and registers
// limit them (250 x 250: 69 and 44 us).  The line lies at 128 threads an SM,
// with float values at 512 (FS_MIXED: 160 x 160 9.0 and 10.2 us, 250 x 250 23.8
// and 23.2).  A mesh of no more than one block of threads an SM starts each
// step's blocks, which read what no step changes, while the step before ends
// (100 x 100, FP64: 10.9 us, 12.2 without); with more blocks the early ones
// crowd some SMs (160 x 160 in blocks of 64: 17 to 29 us).
template <int PREC, int UN> static int launch_block_step(fs_ctx *c, bool next, int from, const CdLoad &ld, int tpb, bool early)
{
    using X = typename CdTypes<PREC>::X;
    auto &x = c->ex;
    X *xp[2] = {(X *)x.xp, (X *)x.xp + 6 * x.nnodes};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((3 * x.nnodes + tpb - 1) / tpb));
    cfg.blockDim = dim3((unsigned)tpb);
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    const X *in = xp[from];
    return cuda_check(c, cudaLaunchKernelEx(&cfg, next ? k_cd_step<PREC, true, UN> : k_cd_step<PREC, false, UN>,
                                            cd_step(c), in, xp[1 - from], ld),
                      "explicit step launch");
}
template <int PREC> static int launch_block_step(fs_ctx *c, bool next, int from, const CdLoad &ld)
{
    const int64_t per_sm = (3 * c->ex.nnodes + c->ex.sms - 1) / c->ex.sms;
    if (per_sm > CD_ONE_BLOCK_TPB) return launch_block_step<PREC, 1>(c, next, from, ld, CD_BLOCK_TPB, false);
    const int tpb = (int)(per_sm + 31) / 32 * 32;
    if (per_sm > cd_small_tpb(PREC)) return launch_block_step<PREC, 1>(c, next, from, ld, tpb, true);
    return launch_block_step<PREC, 4>(c, next, from, ld, tpb, true);
}
static int launch_block_step(fs_ctx *c, bool next, int from, const CdLoad &ld)
{
    if (c->ex.precision == FS_FP64) return launch_block_step<FS_FP64>(c, next, from, ld);
    if (c->ex.precision == FS_MIXED) return launch_block_step<FS_MIXED>(c, next, from, ld);
    return launch_block_step<FS_MIXED_COMP>(c, next, from, ld);
}

// the displacement update alone, of a step on the blocks
static int launch_disp(fs_ctx *c)
{
    auto &x = c->ex;
    const unsigned g = (unsigned)((x.n + CD_TPB - 1) / CD_TPB);
    const double dt = x.dt, h = dt * dt / 2;
    if (x.n == 0) return FS_OK;
    if (x.precision == FS_FP64)
        k_cd_disp_pad<<<g, CD_TPB, 0, c->stream>>>(x.n, dt, h, x.U, x.cU, x.V, x.A, x.pad_of_dof, (double *)x.xp);
    else if (x.precision == FS_MIXED)
        k_cd_disp_pad<<<g, CD_TPB, 0, c->stream>>>(x.n, dt, h, x.U, x.cU, x.V, x.A, x.pad_of_dof, (float *)x.xp);
    else
        k_cd_disp_pad<<<g, CD_TPB, 0, c->stream>>>(x.n, dt, h, x.U, x.cU, x.V, x.A, x.pad_of_dof, (float2 *)x.xp);
    return cuda_check(c, cudaGetLastError(), "displacement update launch");
}

// nsteps steps; on the blocks (one_pass) each step but the last of a run also
// does the next one's displacement update, so the first finds it done, and
// reads the copy that the one before wrote, from copy 0 on
static int enqueue_steps(fs_ctx *c, int64_t nsteps, bool last)
{
    auto &x = c->ex;
    int64_t n = x.n;
    double dt = x.dt;
    CdLoad ld{x.load ? x.Fmag : nullptr, x.mul, x.nmul, x.step, 0};
    unsigned g1 = (unsigned)((n + CD_TPB - 1) / CD_TPB);
    unsigned g2 = (unsigned)((n * CD_LANES + CD_TPB - 1) / CD_TPB);
    for (int64_t s = 0; s < nsteps; s++) {
        ld.j = (int)s;
        if (x.bsr) {
            if (!x.one_pass) FS_TRY(launch_disp(c));
            FS_TRY(launch_block_step(c, x.one_pass && !(last && s + 1 == nsteps), x.one_pass ? (int)(s & 1) : 0, ld));
            continue;
        }
        if (x.precision == FS_MIXED_COMP) {
            k_cd_disp_pair<<<g1, CD_TPB, 0, c->stream>>>(n, dt, dt * dt / 2, x.U, x.cU, x.V, x.A, (float2 *)x.U32);
            k_cd_rows_comp<<<g2, CD_TPB, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, x.vals32,
                                                          (const __nv_bfloat16 *)x.res, (const float2 *)x.U32, x.V,
                                                          x.cV, x.A, x.C, x.invMC, dt / 2, ld);
            continue;
        }
        bool single = x.precision != FS_FP64;
        k_cd_disp<<<g1, CD_TPB, 0, c->stream>>>(n, dt, dt * dt / 2, x.U, x.cU, x.V, x.A, single ? x.U32 : nullptr);
        if (!single)
            k_cd_rows<double><<<g2, CD_TPB, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, c->vals, x.U, x.V,
                                                            x.cV, x.A, x.C, x.invMC, dt / 2, ld);
        else
            k_cd_rows<float><<<g2, CD_TPB, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, x.vals32, x.U32, x.V,
                                                           x.cV, x.A, x.C, x.invMC, dt / 2, ld);
    }
    if (x.load && nsteps > 0) k_step_advance<<<1, 1, 0, c->stream>>>(x.step, nsteps);
    return cuda_check(c, cudaGetLastError(), "explicit step launch");
}

int explicit_launch_steps(fs_ctx *c, int64_t nsteps)
{
    auto &x = c->ex;
    if (nsteps <= 0) return FS_OK;
    if (!x.exec) {
        FS_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        int st = enqueue_steps(c, CD_GRAPH_STEPS, false);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(c->stream, &g);
        if (st != FS_OK) return st;
        FS_CUDA(c, e);
        x.graph = g;
        FS_CUDA(c, cudaGraphInstantiate(&x.exec, g, 0));
        x.graph_steps = CD_GRAPH_STEPS;
    }
    if (x.bsr && x.one_pass) FS_TRY(launch_disp(c));
    // the last step of all is not in the graph
    const int64_t full = (nsteps - 1) / x.graph_steps, rest = nsteps - full * x.graph_steps;
    for (int64_t k = 0; k < full; k++) FS_CUDA(c, cudaGraphLaunch(x.exec, c->stream));
    return enqueue_steps(c, rest, true);
}

__global__ void k_to_float(int64_t n, const double *src, float *dst)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = (float)src[i];
}

// ---------------------------------------------------------------------------
// power iteration for the largest generalized eigenvalue of (K, M), M
// diagonal: the reference's `pwr` (clamp_cyl_expl_examples.jl:131-142),
// w = K v / |K v|, v = M^-1 w / |M^-1 w|, omega = sqrt(v'Kv / v'Mv).
// Reductions are two-pass with a fixed order: bitwise reproducible.
// ---------------------------------------------------------------------------
static const int PI_TPB = 256;
static const int PI_BLOCKS = 1024;

// y = alpha K x, CD_LANES lanes per row
__global__ void k_spmv(int64_t n, const int64_t *rowptr, const int32_t *colidx, const double *vals,
                       const double *x, double *y, double alpha = 1.0)
{
    int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / CD_LANES;
    const int sub = threadIdx.x & (CD_LANES - 1);
    double s = 0.0;
    if (row < n)
        for (int64_t k = rowptr[row] + sub; k < rowptr[row + 1]; k += CD_LANES) s += vals[k] * x[colidx[k]];
#pragma unroll
    for (int o = CD_LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (row < n && sub == 0) y[row] = alpha * s;
}

// partial[b] = sum over this block's strided range of a[i] * b[i] (b may be a weight)
__global__ void k_dot_partial(int64_t n, const double *a, const double *b, double *partial)
{
    __shared__ double sh[PI_TPB];
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * PI_TPB + threadIdx.x; i < n; i += (int64_t)PI_BLOCKS * PI_TPB)
        s += a[i] * b[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = PI_TPB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void k_dot_final(const double *partial, double *out)
{
    __shared__ double sh[PI_TPB];
    double s = 0.0;
    for (int i = threadIdx.x; i < PI_BLOCKS; i += PI_TPB) s += partial[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = PI_TPB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

// y = x * (1/sqrt(*nrm2)) * (w ? w[i] : 1)
__global__ void k_scale(int64_t n, const double *x, const double *nrm2, const double *w, double *y)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double f = 1.0 / sqrt(*nrm2);
    y[i] = x[i] * f * (w ? w[i] : 1.0);
}

// deterministic start vector in [0, 1) from a 64-bit mix of (seed, i)
__global__ void k_start(int64_t n, uint64_t seed, double *v)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t z = seed + 0x9e3779b97f4a7c15ull * (uint64_t)(i + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z = z ^ (z >> 31);
    v[i] = (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

void end_explicit(fs_ctx *c)
{
    auto &x = c->ex;
    if (x.exec) cudaGraphExecDestroy(x.exec);
    if (x.graph) cudaGraphDestroy(x.graph);
    x.exec = nullptr;
    x.graph = nullptr;
    x.ready = false;
}

}  // namespace fs

using namespace fs;

extern "C" {

int fs_power_iteration(fs_ctx *c, const double *mdiag, int64_t iters, uint64_t seed, double *omega_max)
{
    if (!c || !mdiag || !omega_max || iters < 1) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    FS_TRY(check_last_stiffness(c));
    int64_t n = c->mat_n;
    if (n == 0) return set_err(c, FS_ERR_BAD_INPUT, "empty matrix");
    size_t need = sizeof(double) * (size_t)(4 * n + PI_BLOCKS + 4);
    FS_TRY(ensure_scratch(c, need));
    double *v = (double *)c->scratch, *w = v + n, *minv = w + n, *md = minv + n;
    double *partial = md + n, *red = partial + PI_BLOCKS;
    FS_CUDA(c, cudaMemcpyAsync(md, mdiag, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    unsigned g = (unsigned)((n + 255) / 256), gs = (unsigned)((n * CD_LANES + 255) / 256);
    std::vector<double> h((size_t)n);
    for (int64_t i = 0; i < n; i++) h[i] = 1.0 / mdiag[i];
    FS_CUDA(c, cudaMemcpyAsync(minv, h.data(), sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    k_start<<<g, 256, 0, c->stream>>>(n, seed, v);
    for (int64_t it = 0; it < iters; it++) {
        k_spmv<<<gs, 256, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, c->vals, v, w);
        k_dot_partial<<<PI_BLOCKS, PI_TPB, 0, c->stream>>>(n, w, w, partial);
        k_dot_final<<<1, PI_TPB, 0, c->stream>>>(partial, red);
        k_scale<<<g, 256, 0, c->stream>>>(n, w, red, minv, v);       // v = M^-1 w / |w|
        k_dot_partial<<<PI_BLOCKS, PI_TPB, 0, c->stream>>>(n, v, v, partial);
        k_dot_final<<<1, PI_TPB, 0, c->stream>>>(partial, red);
        k_scale<<<g, 256, 0, c->stream>>>(n, v, red, nullptr, v);    // v = v / |v|
    }
    // Rayleigh quotient v'Kv / v'Mv
    double one = 1.0;
    FS_CUDA(c, cudaMemcpyAsync(red + 3, &one, sizeof(double), cudaMemcpyHostToDevice, c->stream));
    k_spmv<<<gs, 256, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, c->vals, v, w);
    k_dot_partial<<<PI_BLOCKS, PI_TPB, 0, c->stream>>>(n, v, w, partial);
    k_dot_final<<<1, PI_TPB, 0, c->stream>>>(partial, red + 1);
    k_scale<<<g, 256, 0, c->stream>>>(n, v, red + 3, md, w);  // w = m .* v
    k_dot_partial<<<PI_BLOCKS, PI_TPB, 0, c->stream>>>(n, v, w, partial);
    k_dot_final<<<1, PI_TPB, 0, c->stream>>>(partial, red + 2);
    FS_CUDA(c, cudaGetLastError());
    double hr[2];
    FS_CUDA(c, cudaMemcpyAsync(hr, red + 1, sizeof(double) * 2, cudaMemcpyDeviceToHost, c->stream));
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    *omega_max = sqrt(hr[0] / hr[1]);
    return FS_OK;
}

int fs_explicit_setup(fs_ctx *c, int precision, const double *invMC, const double *C, double dt)
{
    if (!c || !invMC || !C) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    FS_TRY(check_last_stiffness(c));
    if (precision != FS_FP64 && precision != FS_MIXED && precision != FS_MIXED_COMP)
        return set_err(c, FS_ERR_BAD_INPUT, "unknown precision");
    if (!(dt > 0.0)) return set_err(c, FS_ERR_BAD_INPUT, "time step must be positive");
    auto &x = c->ex;
    end_explicit(c);  // no state until all buffers are there: an allocation may fail
    x.load = false;
    int64_t n = c->mat_n;
    x.n = n;
    x.dt = dt;
    x.precision = precision;
    FS_TRY(dalloc(c, &x.U, (size_t)n)); FS_TRY(dalloc(c, &x.V, (size_t)n)); FS_TRY(dalloc(c, &x.A, (size_t)n));
    FS_TRY(dalloc(c, &x.cU, (size_t)n)); FS_TRY(dalloc(c, &x.cV, (size_t)n));
    FS_TRY(dalloc(c, &x.invMC, (size_t)n)); FS_TRY(dalloc(c, &x.C, (size_t)n));
    size_t bn = sizeof(double) * (size_t)std::max<int64_t>(n, 1);
    FS_CUDA(c, cudaMemsetAsync(x.U, 0, bn, c->stream));
    FS_CUDA(c, cudaMemsetAsync(x.V, 0, bn, c->stream));
    FS_CUDA(c, cudaMemsetAsync(x.A, 0, bn, c->stream));
    FS_CUDA(c, cudaMemsetAsync(x.cU, 0, bn, c->stream));
    FS_CUDA(c, cudaMemsetAsync(x.cV, 0, bn, c->stream));
    FS_CUDA(c, cudaMemcpyAsync(x.invMC, invMC, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    FS_CUDA(c, cudaMemcpyAsync(x.C, C, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    // 6x6 node-block form when the pattern of the current mesh is there (its
    // neighbour lists are the block rows); otherwise the CSR product
    x.bsr = c->pat.n >= 0 && c->pat.nbr_off && c->mesh.nnodes > 0;
    if (x.bsr) {
        const MeshDev &m = c->mesh;
        const int64_t nn = m.nnodes;
        int64_t nbr_total = 0;
        FS_CUDA(c, cudaMemcpyAsync(&nbr_total, c->pat.nbr_off + nn, sizeof(int64_t), cudaMemcpyDeviceToHost, c->stream));
        FS_CUDA(c, cudaStreamSynchronize(c->stream));
        // block values: double or float; displacement copy: double, float,
        // or float pairs (FS_MIXED_COMP)
        const size_t es = precision == FS_FP64 ? 8 : 4, xs = precision == FS_MIXED ? 4 : 8;
        dfree(&x.xp);
        dfree(&x.item);
        FS_CUDA(c, cudaMalloc(&x.xp, 2 * xs * 6 * (size_t)nn));
        FS_CUDA(c, cudaMemsetAsync(x.xp, 0, 2 * xs * 6 * (size_t)nn, c->stream));
        FS_TRY(dalloc(c, &x.pad_of_dof, (size_t)n));
        FS_CUDA(c, cudaMemsetAsync(x.pad_of_dof, 0xff, sizeof(int32_t) * (size_t)std::max<int64_t>(n, 1), c->stream));
        k_pad_map<<<(unsigned)((6 * nn + 255) / 256), 256, 0, c->stream>>>(nn, n, m.dof, x.pad_of_dof);
        if (n) k_cd_unowned<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(n, x.pad_of_dof, c->d_status);
        const unsigned gw = (unsigned)((nn * 32 + 255) / 256);
        FS_CUDA(c, cudaMalloc(&x.item, sizeof(CdItem) * (size_t)std::max<int64_t>(nbr_total, 1)));
        // each off-diagonal block once, or all where K is not symmetric to the last bit
        int bits = DEV_UNSYMMETRIC;
        for (int once = 1; once >= 0 && (bits & DEV_UNSYMMETRIC); once--) {
            const size_t nblocks = (size_t)std::max<int64_t>(once ? c->pat.nitems : nbr_total, 1);
            dfree(&x.blk);
            dfree(&x.res);
            FS_CUDA(c, cudaMalloc(&x.blk, es * 36 * nblocks));
            if (precision == FS_MIXED_COMP) FS_CUDA(c, cudaMalloc(&x.res, 2 * 36 * nblocks));
            k_cd_fill<<<gw, 256, 0, c->stream>>>(nn, n, precision, m.dof, c->mat_rowptr, c->mat_colidx, c->vals,
                                                 c->pat.nbr_off, c->pat.nbr, once ? c->pat.item_off : nullptr,
                                                 (CdItem *)x.item, x.blk, (__nv_bfloat16 *)x.res, c->d_status);
            FS_CUDA(c, cudaGetLastError());
            const int before = once ? 0 : bits & ~DEV_UNSYMMETRIC;
            FS_TRY(read_status(c, &bits));
            bits |= before;
        }
        x.one_pass = !(bits & DEV_UNOWNED);
        FS_CUDA(c, cudaDeviceGetAttribute(&x.sms, cudaDevAttrMultiProcessorCount, c->device));
        x.nnodes = nn;
    } else if (precision != FS_FP64) {
        // float copy of U, or float pairs (two floats a dof) for FS_MIXED_COMP
        FS_TRY(dalloc(c, &x.U32, (size_t)n * (precision == FS_MIXED_COMP ? 2 : 1)));
        FS_TRY(dalloc(c, &x.vals32, (size_t)c->mat_nnz));
        dfree(&x.res);
        if (precision == FS_MIXED_COMP) {
            FS_CUDA(c, cudaMalloc(&x.res, 2 * (size_t)std::max<int64_t>(c->mat_nnz, 1)));
            if (c->mat_nnz)
                k_split_values<<<(unsigned)((c->mat_nnz + 255) / 256), 256, 0, c->stream>>>(
                    c->mat_nnz, c->vals, x.vals32, (__nv_bfloat16 *)x.res);
        } else if (c->mat_nnz)
            k_to_float<<<(unsigned)((c->mat_nnz + 255) / 256), 256, 0, c->stream>>>(c->mat_nnz, c->vals, x.vals32);
        FS_CUDA(c, cudaGetLastError());
    }
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    x.ready = true;
    return FS_OK;
}

int fs_explicit_set_state(fs_ctx *c, const double *U, const double *V, const double *A)
{
    if (!c) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    auto &x = c->ex;
    if (!x.ready) return set_err(c, FS_ERR_STATE, "call fs_explicit_setup first");
    size_t bn = sizeof(double) * (size_t)x.n;
    if (U) FS_CUDA(c, cudaMemcpyAsync(x.U, U, bn, cudaMemcpyHostToDevice, c->stream));
    if (V) FS_CUDA(c, cudaMemcpyAsync(x.V, V, bn, cudaMemcpyHostToDevice, c->stream));
    if (A) FS_CUDA(c, cudaMemcpyAsync(x.A, A, bn, cudaMemcpyHostToDevice, c->stream));
    if (bn) {
        FS_CUDA(c, cudaMemsetAsync(x.cU, 0, bn, c->stream));
        FS_CUDA(c, cudaMemsetAsync(x.cV, 0, bn, c->stream));
    }
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    return FS_OK;
}

int fs_explicit_set_load(fs_ctx *c, const double *Fmag, const double *mul, int64_t nmul, int64_t step0)
{
    if (!c || nmul < 0 || step0 < 0) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    auto &x = c->ex;
    if (!x.ready) return set_err(c, FS_ERR_STATE, "call fs_explicit_setup first");
    if (Fmag && nmul > 0 && !mul) return set_err(c, FS_ERR_BAD_INPUT, "missing time function values");
    // the captured steps hold the load pointers: capture again on the next run
    if (x.exec) cudaGraphExecDestroy(x.exec);
    if (x.graph) cudaGraphDestroy(x.graph);
    x.exec = nullptr;
    x.graph = nullptr;
    x.load = Fmag != nullptr;
    if (!x.load) return FS_OK;
    FS_TRY(grow(c, &x.Fmag, &x.cap_Fmag, (size_t)std::max<int64_t>(x.n, 1)));
    FS_TRY(grow(c, &x.mul, &x.cap_mul, (size_t)std::max<int64_t>(nmul, 1)));
    if (!x.step) FS_TRY(dalloc(c, &x.step, 1));
    x.nmul = nmul;
    FS_CUDA(c, cudaMemcpyAsync(x.Fmag, Fmag, sizeof(double) * (size_t)x.n, cudaMemcpyHostToDevice, c->stream));
    if (nmul) FS_CUDA(c, cudaMemcpyAsync(x.mul, mul, sizeof(double) * (size_t)nmul, cudaMemcpyHostToDevice, c->stream));
    FS_CUDA(c, cudaMemcpyAsync(x.step, &step0, sizeof(int64_t), cudaMemcpyHostToDevice, c->stream));
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    return FS_OK;
}

int fs_explicit_run(fs_ctx *c, int64_t nsteps)
{
    if (!c || nsteps < 0) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    if (!c->ex.ready) return set_err(c, FS_ERR_STATE, "call fs_explicit_setup first");
    FS_TRY(explicit_launch_steps(c, nsteps));
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    return FS_OK;
}

int fs_explicit_get_state(fs_ctx *c, double *U, double *V, double *A)
{
    if (!c) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    auto &x = c->ex;
    if (!x.ready) return set_err(c, FS_ERR_STATE, "call fs_explicit_setup first");
    size_t bn = sizeof(double) * (size_t)x.n;
    if (U) FS_TRY(copy_out(c, U, x.U, bn));
    if (V) FS_TRY(copy_out(c, V, x.V, bn));
    if (A) FS_TRY(copy_out(c, A, x.A, bn));
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    return FS_OK;
}

// Restoring force of the shells: -K U with the last assembled matrix.
int fs_restoring_force(fs_ctx *c, const double *U, double *F)
{
    if (!c) return FS_ERR_BAD_INPUT;
    FS_CUDA(c, cudaSetDevice(c->device));
    FS_TRY(check_last_stiffness(c));
    const int64_t n = c->mat_n;
    if (n && (!U || !F)) return set_err(c, FS_ERR_BAD_INPUT, "missing vector");
    if (n == 0) return FS_OK;
    FS_TRY(ensure_scratch(c, sizeof(double) * 2 * (size_t)n));
    double *u = (double *)c->scratch, *f = u + n;
    FS_CUDA(c, cudaMemcpyAsync(u, U, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    const unsigned gs = (unsigned)((n * CD_LANES + 255) / 256);
    k_spmv<<<gs, 256, 0, c->stream>>>(n, c->mat_rowptr, c->mat_colidx, c->vals, u, f, -1.0);
    FS_CUDA(c, cudaGetLastError());
    FS_CUDA(c, cudaMemcpyAsync(F, f, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
    FS_CUDA(c, cudaStreamSynchronize(c->stream));
    return FS_OK;
}

}  // extern "C"
