// CSR value gather: element node blocks -> CSR values.
//
// The unit of work is a node-block pair (r, s), r <= s, of the assembled
// matrix: its 6x6 block is the sum of the element blocks that touch both
// nodes (two for an edge of a triangulated plate, six for a node's own
// block).  The symbolic phase lists these blocks with their contributions, in
// ascending assembly rank, as positions of stored element blocks (GatherRound).
// The element kernels store every block with the lower node's dofs as its
// rows, so a contribution is read as it lies.
//
// Six threads own one block, thread i its row i: 24 or 48 contiguous bytes of
// every contribution, added in order.  The sums of thread i are six
// contiguous values (through the symmetry of the matrix, of column i) of the
// rows of node s: the six threads store them in 48-byte runs; the rows of node
// r get them through a transpose in shared memory (a node's own block is
// symmetric: its rows are its columns).  No atomics; every stored value is the
// left-to-right sum of its element contributions in assembly order, as
// Julia's sparse(I, J, V) combines duplicates.
//
// Bound by the latency of three dependent rounds of loads (a block's
// description; its first contributions, the positions of the next ones and the
// places of its rows and columns; the next contributions) and then by DRAM
// traffic.  What hides it is many resident warps: a warp sums five blocks and
// ends (51, 64 and 54 registers for float, float-pair and double entries).  A
// warp that went on to the next five with their descriptions loaded ahead, or
// copied rounds of contributions ahead through shared memory (cp.async), had
// more loads in flight but too few warps: 1.26 and 1.56 ms against 0.98 ms for
// the float pairs of the 1024 x 1024 triangulated plate.  In the list, groups
// of GATHER_GROUP nodes have first the nodes' own blocks, then the off-diagonal
// ones, so that the five blocks of a warp have equally many contributions.
// 1024 x 1024 triangulated plate, float, float-pair and double entries:
// 0.75, 0.98 and 0.97 ms; a warp per node that staged the node's element
// blocks in shared memory took 1.25, 1.96 and 2.09 ms.
#include "fs_elem_common.cuh"

namespace fs {

// exact float -> double from the bit pattern for zeros and normal numbers
__device__ __forceinline__ double f2d_normal(float f)
{
    const uint32_t u = __float_as_uint(f);
    uint32_t h = (uint32_t)((int32_t)u >> 3) & 0x8fffffffu;
    if (f != 0.f) h += 0x38000000u;
    return __hiloint2double((int)h, (int)(u << 29));
}
// neither subnormal nor infinite nor NaN
__device__ __forceinline__ bool plain_float(float f)
{
    return f == 0.f || ((__float_as_uint(f) & 0x7fffffffu) - 0x00800000u < 0x7f000000u);
}

// The sums of one thread's six entries.  set() takes the first contribution,
// add() the next ones (rows of six entries in shared memory), values() the
// sums rounded to double.  Double entries: double addition.  Float entries
// (FS_MIXED): an unevaluated float pair, the high sum's error added to the low
// part (TwoSum), the low part's rounding left (below 2^-46 of the largest
// contribution); one double add per stored value instead of a conversion and
// an add per contribution, a double add costing as much as 64 float operations
// on GB300.  Float-pair entries (FS_MIXED_COMP; two entries stored as hi, hi,
// lo, lo): an unevaluated float triple, the stored high half added to the
// high part and the stored low half and the high sum's error to the low part
// by TwoSum, the low part's errors going to the tail, so that what is lost is
// the tail's rounding (at most 8 n^2 (n + 1) 2^-72 of the n contributions'
// magnitudes); entries 2q and 2q + 1 in one packed register pair.
template <class R> struct RowSum;
template <> struct RowSum<double> {
    double v[6];
    struct Load {
        double2 x[3];
    };
    static __device__ __forceinline__ Load load(const double *blk, int i)
    {
        const double2 *q = reinterpret_cast<const double2 *>(blk + 6 * i);
        return {{q[0], q[1], q[2]}};
    }
    static __device__ __forceinline__ Load strided(const double *blk, int i)
    {
        const double *p = blk + i;
        return {{make_double2(p[0], p[6]), make_double2(p[12], p[18]), make_double2(p[24], p[30])}};
    }
    __device__ __forceinline__ void set(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            v[2 * q] = l.x[q].x;
            v[2 * q + 1] = l.x[q].y;
        }
    }
    __device__ __forceinline__ void add(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            v[2 * q] += l.x[q].x;
            v[2 * q + 1] += l.x[q].y;
        }
    }
    __device__ __forceinline__ void values(double (&o)[6]) const
    {
#pragma unroll
        for (int k = 0; k < 6; k++) o[k] = v[k];
    }
};
__device__ __forceinline__ float two_sum_err(float &s, float v)
{
    const float t = s + v;
    const float bp = t - s;
    const float e = (s - (t - bp)) + (v - bp);
    s = t;
    return e;
}
template <> struct RowSum<float> {
    float hi[6], lo[6];
    struct Load {
        float2 x[3];
    };
    static __device__ __forceinline__ Load load(const float *blk, int i)
    {
        const float2 *q = reinterpret_cast<const float2 *>(blk + 6 * i);
        return {{q[0], q[1], q[2]}};
    }
    static __device__ __forceinline__ Load strided(const float *blk, int i)
    {
        const float *p = blk + i;
        return {{make_float2(p[0], p[6]), make_float2(p[12], p[18]), make_float2(p[24], p[30])}};
    }
    __device__ __forceinline__ void set(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            hi[2 * q] = l.x[q].x;
            hi[2 * q + 1] = l.x[q].y;
            lo[2 * q] = lo[2 * q + 1] = 0.f;
        }
    }
    __device__ __forceinline__ void add(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            lo[2 * q] += two_sum_err(hi[2 * q], l.x[q].x);
            lo[2 * q + 1] += two_sum_err(hi[2 * q + 1], l.x[q].y);
        }
    }
    // hi + lo: exact in double unless their exponents are more than 29
    // apart, then rounded once
    __device__ __forceinline__ void values(double (&o)[6]) const
    {
        bool plain = true;
#pragma unroll
        for (int k = 0; k < 6; k++) plain = plain && plain_float(hi[k]) && plain_float(lo[k]);
        if (plain) {
#pragma unroll
            for (int k = 0; k < 6; k++) o[k] = f2d_normal(hi[k]) + f2d_normal(lo[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 6; k++) o[k] = f2d_exact(hi[k]) + f2d_exact(lo[k]);
        }
    }
};
template <> struct RowSum<float2> {
    f32x2 hi[3], lo[3], tl[3];
    struct Load {
        ulonglong2 x[3];  // entries 2q, 2q + 1: their high halves, their low halves
    };
    static __device__ __forceinline__ Load load(const float2 *blk, int i)
    {
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(blk + 6 * i);
        return {{q[0], q[1], q[2]}};
    }
    static __device__ __forceinline__ Load strided(const float2 *blk, int i)
    {
        const float *p = reinterpret_cast<const float *>(blk) + 4 * (i / 2) + (i & 1);
        Load l;
#pragma unroll
        for (int q = 0; q < 3; q++)
            l.x[q] = make_ulonglong2(x2_pack(p[24 * q], p[24 * q + 12]), x2_pack(p[24 * q + 2], p[24 * q + 14]));
        return l;
    }
    // a stored float pair is normalised (|lo| <= ulp(hi)/2): taken as is
    __device__ __forceinline__ void set(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            hi[q] = l.x[q].x;
            lo[q] = l.x[q].y;
            tl[q] = 0ull;
        }
    }
    __device__ __forceinline__ void add(const Load &l)
    {
#pragma unroll
        for (int q = 0; q < 3; q++) x2_triple_add(hi[q], lo[q], tl[q], l.x[q].x, l.x[q].y);
    }
    // hi + (lo + tl): lo + tl exact in double, then one rounding of the
    // whole to double (2^-53 of the value).  Ending in a float rounding of
    // the low parts instead (one double add, 2^-48 of the value) raised the
    // 20-eigenvalue error of the 256 x 256 layered plate from 1.1e-7 to
    // 2.8e-7: the soft modes amplify per-entry errors about 1e8-fold.
    __device__ __forceinline__ void values(double (&o)[6]) const
    {
        float h[6], l[6], t[6];
        bool plain = true;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            x2_unpack(hi[q], h[2 * q], h[2 * q + 1]);
            x2_unpack(lo[q], l[2 * q], l[2 * q + 1]);
            x2_unpack(tl[q], t[2 * q], t[2 * q + 1]);
        }
#pragma unroll
        for (int k = 0; k < 6; k++) plain = plain && plain_float(h[k]) && plain_float(l[k]) && plain_float(t[k]);
        if (plain) {
#pragma unroll
            for (int k = 0; k < 6; k++) o[k] = f2d_normal(h[k]) + (f2d_normal(l[k]) + f2d_normal(t[k]));
        } else {
#pragma unroll
            for (int k = 0; k < 6; k++) o[k] = f2d_exact(h[k]) + (f2d_exact(l[k]) + f2d_exact(t[k]));
        }
    }
};

static const int G_PER_WARP = 5;  // blocks of a warp (30 threads)

// sides: bit 0 writes the rows of node r, bit 1 those of node s
template <class R, int W>
__global__ void __launch_bounds__(32 * W)
    k_gather(int64_t nitems, const GatherItem *__restrict__ items, const uint32_t *__restrict__ src,
             const int64_t *__restrict__ rowstart, const int16_t *__restrict__ colpos, const R *__restrict__ ke,
             double *__restrict__ vals, int sides)
{
    __shared__ __align__(16) double gather_smem[W][G_PER_WARP * 36];
    const int lane = threadIdx.x & 31, g = lane / 6, i = lane - 6 * g;
    const int base = lane < 30 ? 6 * g : 0;  // the block's first lane
    const int64_t it = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G_PER_WARP + g;
    const uint4 *dsc = reinterpret_cast<const uint4 *>(items + it);
    uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
    if (g < G_PER_WARP && it < nitems) {
        w0 = dsc[0];
        w1 = dsc[1];
    }
    const uint32_t r = w0.x, s = w0.y, cnt = w1.x;
    const bool own = r == s;
    auto at = [&](uint32_t e) {
        const R *p = ke + (int64_t)(e & 0x7fffffffu) * 36;
        return (e >> 31) ? RowSum<R>::strided(p, i) : RowSum<R>::load(p, i);
    };
    // where this thread's row of either node starts and the position of its
    // column in the other's rows (-1: a dof outside the matrix)
    int64_t row_r = -1, row_s = -1;
    int col_r = -1, col_s = -1;
    double v[6] = {0, 0, 0, 0, 0, 0};
    if (cnt) {
        const typename RowSum<R>::Load x0 = at(w1.y), x1 = at(w1.z);
        const uint32_t *more = src + w1.w;
        uint32_t e[4] = {0, 0, 0, 0};
        if (cnt > 2) {
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) e[u] = more[min(2 + u, cnt - 1)];
        }
        if (own || (sides & 2)) {
            row_s = rowstart[6 * (int64_t)s + i];
            col_r = colpos[6 * (int64_t)w0.w + i];
        }
        if (!own && (sides & 1)) {
            row_r = rowstart[6 * (int64_t)r + i];
            col_s = colpos[6 * (int64_t)w0.z + i];
        }
        RowSum<R> sum;
        sum.set(x0);
        if (cnt > 1) sum.add(x1);
        if (cnt > 2) {
#pragma unroll
            for (uint32_t u = 0; u < 4; u += 2) {
                if (2 + u < cnt) {
                    const typename RowSum<R>::Load y0 = at(e[u]), y1 = at(e[u + 1]);
                    sum.add(y0);
                    if (3 + u < cnt) sum.add(y1);
                }
            }
            for (uint32_t q = 6; q < cnt; q++) sum.add(at(more[q]));
        }
        sum.values(v);
    }
    // the rows of node s at column i of node r
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const int64_t q = __shfl_sync(0xffffffffu, row_s, base + j);
        if (q >= 0 && col_r >= 0) vals[q + col_r] = v[j];
    }
    // the rows of node r at column i of node s: entry (j, i) of the block
    double *tr = gather_smem[threadIdx.x >> 5] + 6 * base;
    if (lane < 30) {
        double2 *t = reinterpret_cast<double2 *>(tr + 6 * i);
#pragma unroll
        for (int q = 0; q < 3; q++) t[q] = make_double2(v[2 * q], v[2 * q + 1]);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const int64_t q = __shfl_sync(0xffffffffu, row_r, base + j);
        if (q >= 0 && col_s >= 0) vals[q + col_s] = tr[6 * j + i];
    }
}

// blocks of `w` warps
template <class R>
static int run_gather(fs_ctx *c, const R *ke, double *vals)
{
    const PatternDev &P = c->pat;
    if (P.nitems == 0) return FS_OK;
    if (!P.items) return set_err(c, FS_ERR_UNSUPPORTED, "mesh too large for the value gather");
    const int w = c->tune.gather_warps == 8 || c->tune.gather_warps == 16 ? c->tune.gather_warps : 4;
    const int64_t per = (int64_t)w * G_PER_WARP;
    const unsigned grid = (unsigned)((P.nitems + per - 1) / per);
    auto launch = [&](auto kern, int side) {
        kern<<<grid, 32 * w, 0, c->stream>>>(P.nitems, P.items, P.src, P.rowstart, P.colpos, ke, vals, side);
    };
    // each pair summed once for both nodes' rows, or (mode 3) by both nodes, one
    // launch for the rows of either: the same contributions in the same order
    const bool both = c->tune.gather_once == 0;
    for (int side = both ? 1 : 3; side <= (both ? 2 : 3); side++)
        launch(w == 4 ? k_gather<R, 4> : w == 8 ? k_gather<R, 8> : k_gather<R, 16>, side);
    FS_CUDA(c, cudaGetLastError());
    return FS_OK;
}

int launch_gather(fs_ctx *c, int precision, double *vals) { return launch_gather_from(c, precision, c->ke, vals); }

// CSR values from element matrices held in `ke`; allocates nothing.
int launch_gather_from(fs_ctx *c, int precision, const void *ke, double *vals)
{
    if (precision == FS_FP64) return run_gather<double>(c, (const double *)ke, vals);
    if (precision == FS_MIXED_COMP) return run_gather<float2>(c, (const float2 *)ke, vals);
    return run_gather<float>(c, (const float *)ke, vals);
}

}  // namespace fs
