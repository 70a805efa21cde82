// FS_FP64 element matrices of the homogeneous shells (T3FF with average B,
// Q4RS), except for an assembly that drops exact zeros: which entries come out
// as zeros is a matter of rounding, so that one keeps the kernels in double
// (fs_elem_t3.cu, fs_elem_q4.cu).  Here: two kernels over chunks of elements (the math is
// csrc/fs_elem_fixed.cuh).
//
// The rows kernel forms the strain coefficients in double and expands them to
// rows in fixed point, one thread an element (T3) or Gauss point (Q4); about 440
// and 870 double instructions a thread (2,400 and 4,100 when rows and Gram
// product were double too) keep the double pipe, 2 operations per clock and SM on
// GB300, 55 to 60 % busy.  Three blocks of 128 threads per SM (168 registers):
// 4 to 6 % faster than two without spills.  The Gram kernel, bound by 32-bit
// integer multiply-adds (64 per clock and SM, 40 to 60 % busy), forms the node
// blocks of 32 elements in a block of 3 (T3) or 4 (Q4) warps, a thread an
// element, a warp its share of the node blocks, so that all lanes of a warp run
// the same code on neighbouring memory; its sums over a point's rows are
// unrolled, since the compiler copies every 64-bit sum of a rolled loop.  In one
// kernel the two need the first one's registers and shared memory for the rows,
// 1 KB a T3 element, which leaves 5 warps an SM: 4.4 ms against 3.5 ms (T3,
// 1024 x 1024) and 4.2 against 3.3 ms (Q4, 512 x 512); all in double 8.0 and
// 7.5 ms.
//
// A chunk's rows pass through a buffer of at most 1 GiB.  Small chunks would
// stay in L2 but leave the SMs idle at the end of each (64 MB: 6.2 and 5.4 ms).
#include <algorithm>

#include "fs_elem_common.cuh"
#include "fs_elem_fixed.cuh"

namespace fs {

static const size_t FX_CHUNK_BYTES = (size_t)1 << 30;  // rows of a chunk

// slots of an element: its rows, then its exponents (node j: m, t, q, and at the
// first node whether it is done elsewhere; then em and r)
constexpr int T3_SLOTS = CompactRows<3, 2>::SIZE + 4;
constexpr int Q4_SLOTS = Q4Compact::SIZE + 5;

__device__ __forceinline__ FxSlots fx_slots(FxSlot *rows, int nslots, int64_t e)
{
    return FxSlots{rows + (e / FX_GROUP) * (FX_GROUP * nslots) + e % FX_GROUP};
}
template <int NN> __device__ __forceinline__ void put_exponents(FxSlots x, const FxExp &ex, bool redo)
{
    auto put = [](FxSlot &o, int a, int b, int c, int d) {
        o.x = fx{(int)((unsigned)(a & 0xffff) | (unsigned)b << 16), (int)((unsigned)(c & 0xffff) | (unsigned)d << 16)};
    };
#pragma unroll
    for (int j = 0; j < NN; j++) put(x[j], ex.m[j], ex.t[j], ex.q[j], j == 0 && redo);
    put(x[NN], ex.em[0], ex.em[1], ex.em[2], ex.r);
}
// the exponents of an element where they lie
template <int NN> struct StoredExp {
    FxSlots x;
    int em[3], r;
    __device__ __forceinline__ explicit StoredExp(FxSlots slots) : x(slots)
    {
        const FxSlot v = x[NN];
#pragma unroll
        for (int c = 0; c < 3; c++) em[c] = v.s[c];
        r = v.s[3];
    }
    __device__ __forceinline__ bool redo() const { return x[0].s[3] != 0; }
    __device__ __forceinline__ FxNode node(int j) const
    {
        const FxSlot v = x[j];
        return FxNode{v.s[0], v.s[1], v.s[2]};
    }
};

// elements e0 .. e0 + n of a chunk; an element whose coefficients do not suit
// the fixed point (not finite, or next to a double's limits: a degenerate
// one; a triangle longer than T3_LONGEST) is marked in `redo` for the double kernel
__global__ void __launch_bounds__(128, 3) k_t3_rows(const MeshDev m, const MatConst mc, int64_t e0, int64_t n, FxSlot *rows,
                                                 uint8_t *redo, int *status)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const FxSlots slot = fx_slots(rows, T3_SLOTS, e);
    ElemIn<3> in;
    load_elem<3>(m, e0 + e, in);
    FxGeom<3> geo;
    FxMax mx;
    const bool bad = t3_coefs<true>(in, mc, slot, geo, mx) || !mx.usable();
    if (bad) atomicOr(status, DEV_REDO);
    redo[e0 + e] = bad;
    FxExp ex = fx_exponents(mx, 0);
    put_exponents<3>(slot + CompactRows<3, 2>::SIZE, ex, bad);
    if (!bad) t3_expand(slot, geo, in.valid, ex);
}

__global__ void __launch_bounds__(96, 4) k_t3_gram(const MeshDev m, int64_t e0, int64_t n, FxSlot *rows, double *ke)
{
    typedef CompactRows<3, 2> L;
    extern __shared__ __align__(16) FxSlot fx_smem[];
    const int w = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * FX_GROUP + (threadIdx.x & 31), r = e0 + e;
    // the group's rows (contiguous) to shared memory, all loads in flight at once
    {
        const char *src = reinterpret_cast<const char *>(rows + (int64_t)blockIdx.x * (FX_GROUP * T3_SLOTS));
        const unsigned dst = (unsigned)__cvta_generic_to_shared(fx_smem);
#pragma unroll 4
        for (int k = 16 * threadIdx.x; k < FX_GROUP * T3_SLOTS * (int)sizeof(FxSlot); k += 16 * 96)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + k), "l"(src + k) : "memory");
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
    }
    if (e >= n) return;
    const FxSlots slot{fx_smem + (threadIdx.x & 31)};
    const StoredExp<3> ex(slot + L::SIZE);
    if (ex.redo()) return;
    double *out = ke + r * (6 * 36);
    // block (w, w)
    {
        double o[3][6], ob[3][6];
        fx_block_top<1, L::MS, L::BS, L::BSS, true>(slot, 0, w, w, ex, o);
        store_rows<double, 3>(out + ub(w, w, 3) * 36, o);
        fx_block_bottom<1, L::BS, L::BSS, true>(slot, 0, w, w, slot + (L::DR + 3 * w), ex, ob);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) ob[i][j] = o[j][3 + i];
        store_rows<double, 3>(out + ub(w, w, 3) * 36 + 18, ob);
    }
    // blocks (0,1) (0,2) (1,2), the lower node's dofs as rows
    const int a = w == 2 ? 1 : 0, b = w == 0 ? 1 : 2;
    const bool sw = m.conn[r * 3 + a] > m.conn[r * 3 + b];
    const int p = sw ? b : a, q = sw ? a : b;
    double o[3][6];
    fx_block_top<1, L::MS, L::BS, L::BSS, false>(slot, 0, p, q, ex, o);
    store_rows<double, 3>(out + ub(a, b, 3) * 36, o);
    fx_block_bottom<1, L::BS, L::BSS, false>(slot, 0, p, q, slot, ex, o);
    store_rows<double, 3>(out + ub(a, b, 3) * 36 + 18, o);
}

// per-element staging area of the Q4 rows kernel
struct Q4Rows {
    double X[4][3], Xr[4][3], nrm[4][3];
    double rn[4];  // 1 / |n| of the nodal normals (0 for a zero one)
    double t, ss;  // thickness, square root of the stabilisation factor
    bool valid[4];
};

__global__ void __launch_bounds__(128, 3) k_q4_rows(const MeshDev m, const MatConst mc, int64_t e0, int64_t n, FxSlot *rows,
                                                 uint8_t *redo, int *status)
{
    typedef Q4Compact L;
    __shared__ Q4Rows stage[32];
    const int el = threadIdx.x >> 2, qp = threadIdx.x & 3;
    Q4Rows &sg = stage[el];
    const int64_t e = (int64_t)blockIdx.x * (blockDim.x >> 2) + el, r = e0 + e;
    const unsigned mask = 0xfu << ((threadIdx.x & 31) & ~3);  // the element's lanes
    if (e >= n) return;
    // --- stage the element: lane qp loads node qp ---
    {
        const int node = m.conn[r * 4 + qp];
        double X[3], nv[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            X[c] = m.xyz[(int64_t)c * m.nnodes + node];
            nv[c] = m.normals[(int64_t)c * m.nnodes + node];
            sg.X[qp][c] = X[c];
            sg.nrm[qp][c] = nv[c];
        }
        sg.valid[qp] = m.valid[node] != 0;
        const double nn = dot3(nv, nv);
        sg.rn[qp] = nn > 0.0 ? rsqrt(nn) : 0.0;
        __syncwarp(mask);
        double mx = 0.0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double cen = (sg.X[0][c] + sg.X[1][c] + sg.X[2][c] + sg.X[3][c]) * 0.25;
            sg.Xr[qp][c] = X[c] - cen;
            const double d = X[c] - sg.X[0][c];
            mx += d * d;
        }
        // the largest distance from the first node
        const double o1 = __shfl_xor_sync(mask, mx, 1);
        mx = o1 > mx ? o1 : mx;
        const double o2 = __shfl_xor_sync(mask, mx, 2);
        mx = o2 > mx ? o2 : mx;
        if (qp == 0) {
            sg.t = m.thick ? m.thick[r] : 0.0;
            sg.ss = sg.t * rsqrt(sg.t * sg.t + mc.stab_c * mx);
        }
        __syncwarp(mask);
    }
    // --- coefficients of this lane's point, traces and maxima of the element ---
    const FxSlots es = fx_slots(rows, Q4_SLOTS, e), slot = es + qp * L::GP;
    FxGeom<4> geo;
    FxMax mx;
    double tr[4] = {0, 0, 0, 0};
    bool bad = q4_coefs(sg.Xr, sg.nrm, sg.valid, sg.rn, sg.t, sg.ss, qp, mc, slot, geo, mx, tr) != 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        tr[k] += __shfl_xor_sync(mask, tr[k], 1);
        tr[k] += __shfl_xor_sync(mask, tr[k], 2);
    }
    // drilling stiffness: the mean over the valid nonzero normals of
    // max(0, tr / 2), times the scale (src/FEMMShellQ4RSModule.jl:807-859)
    double sum = 0.0;
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (sg.valid[k] && sg.rn[k] != 0.0) {
            const double v = tr[k] * 0.5;
            sum += v > 0.0 ? v : 0.0;
            cnt++;
        }
    const double kavg = (cnt ? sum / cnt : 0.0) * mc.drill_scale;
    const double sk = kavg > 0.0 && sg.valid[qp] && sg.rn[qp] != 0.0 ? sqrt(kavg) : 0.0;
    double dr[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        dr[c] = sk * sg.nrm[qp][c];
        fx_max(mx.r, dr[c]);
    }
    // maxima over the points, two at a time by their exponent fields
    auto over_points = [&](uint32_t &a, uint32_t &b) {
        uint32_t v = __byte_perm(a >> 20, b >> 20, 0x5410);
        v = __vmaxu2(v, __shfl_xor_sync(mask, v, 1));
        v = __vmaxu2(v, __shfl_xor_sync(mask, v, 2));
        a = v << 20;
        b = (v >> 16) << 20;
    };
#pragma unroll
    for (int k = 0; k < 4; k++) {
        over_points(mx.m[k], mx.w[k]);
        over_points(mx.q[k], mx.g[k]);
    }
    over_points(mx.r, mx.u);
    over_points(mx.e[0], mx.e[1]);
    over_points(mx.e[2], mx.e[2]);
    bad = __any_sync(mask, bad || !mx.usable());
    const FxExp ex = fx_exponents(mx, 1);
    if (qp == 0) {
        if (bad) atomicOr(status, DEV_REDO);
        redo[r] = bad;
        put_exponents<4>(es + L::SIZE, ex, bad);
    }
    if (bad) return;
    fx t[4][3][3];
    expand_slots<4, L::MS, L::BS, L::BSS>(slot, geo, ex, t);
#pragma unroll
    for (int c = 0; c < 3; c++) es[L::DR + 3 * qp + c].x = fx_make(dr[c], ex.r);
}

__global__ void __launch_bounds__(128, 3) k_q4_gram(const MeshDev m, int64_t e0, int64_t n, FxSlot *rows, double *ke)
{
    typedef Q4Compact L;
    const int w = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * FX_GROUP + (threadIdx.x & 31), r = e0 + e;
    if (e >= n) return;
    const FxSlots slot = fx_slots(rows, Q4_SLOTS, e);
    const StoredExp<4> ex(slot + L::SIZE);
    if (ex.redo()) return;
    const unsigned swapped = swapped_blocks<4>(m.conn + r * 4);
    double *out = ke + r * (10 * 36);
    // every warp a diagonal block, then three of the twelve halves of the
    // off-diagonal ones (rows 0-2 of the six, then rows 3-5)
    {
        double o[3][6], ob[3][6];
        fx_block_top<4, L::MS, L::BS, L::BSS, true>(slot, L::GP, w, w, ex, o);
        store_rows<double, 3>(out + ub(w, w, 4) * 36, o);
        fx_block_bottom<4, L::BS, L::BSS, true>(slot, L::GP, w, w, slot + (L::DR + 3 * w), ex, ob);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) ob[i][j] = o[j][3 + i];
        store_rows<double, 3>(out + ub(w, w, 4) * 36 + 18, ob);
    }
#pragma unroll 1
    for (int t = 0; t < 3; t++) {
        const int u = w + 4 * t, ob = u < 6 ? u : u - 6;
        const int a = ob < 3 ? 0 : (ob < 5 ? 1 : 2), b = ob < 3 ? ob + 1 : (ob < 5 ? ob - 1 : 3);
        const bool sw = (swapped >> (4 * a + b)) & 1u;
        const int p = sw ? b : a, q = sw ? a : b;
        double o[3][6];
        if (u < 6)
            fx_block_top<4, L::MS, L::BS, L::BSS, false>(slot, L::GP, p, q, ex, o);
        else
            fx_block_bottom<4, L::BS, L::BSS, false>(slot, L::GP, p, q, slot, ex, o);
        store_rows<double, 3>(out + ub(a, b, 4) * 36 + (u < 6 ? 0 : 18), o);
    }
}

// elements of a chunk: equal chunks of at most FX_CHUNK_BYTES
static int64_t chunk_elements(const MeshDev &m)
{
    const int64_t per = (int64_t)(m.nen == 3 ? T3_SLOTS : Q4_SLOTS) * (int64_t)sizeof(FxSlot) * FX_GROUP;
    const int64_t groups = (m.nelem + FX_GROUP - 1) / FX_GROUP, most = (int64_t)FX_CHUNK_BYTES / per;
    const int64_t chunks = std::max<int64_t>((groups + most - 1) / most, 1);
    return std::max<int64_t>((groups + chunks - 1) / chunks, 1) * FX_GROUP;
}

// slots that the marks of the elements to do in double take, ahead of the rows
static size_t mark_slots(const MeshDev &m) { return ((size_t)m.nelem + 255) / 256 * (256 / sizeof(FxSlot)); }

// The buffer of the marks and of a chunk's rows, kept by the context.  With no
// memory for the smallest chunk, fx_rows stays null.
int ensure_fp64_rows(fs_ctx *c)
{
    const MeshDev &m = c->mesh;
    if (m.etype != FS_T3FF && m.etype != FS_Q4RS) return FS_OK;
    const size_t group = (size_t)FX_GROUP * (m.nen == 3 ? T3_SLOTS : Q4_SLOTS);
    return fx_reserve(c->fx_rows ? c->cap_fx_rows : 0, c->fx_asked, mark_slots(m), (size_t)chunk_elements(m) / FX_GROUP, group,
                      FS_OK, FS_ERR_OOM, [&](size_t slots) {
                          FxSlot *rows = (FxSlot *)c->fx_rows;
                          const int st = grow(c, &rows, &c->cap_fx_rows, slots);
                          c->fx_rows = rows;
                          return st;
                      });
}

int run_fp64(fs_ctx *c, double *ke)
{
    const MeshDev &m = c->mesh;
    const bool t3 = m.nen == 3;
    // (the allocation-free path has the buffer, or none, from its pattern on)
    if (ke != c->noalloc_scratch) FS_TRY(ensure_fp64_rows(c));
    const size_t marks = mark_slots(m), group = (size_t)FX_GROUP * (t3 ? T3_SLOTS : Q4_SLOTS);
    const int64_t held = c->fx_rows ? (int64_t)fx_groups_held(c->cap_fx_rows, marks, group) * FX_GROUP : 0;
    if (!held) return t3 ? redo_t3(c, ke, nullptr) : redo_q4(c, ke, nullptr);
    uint8_t *redo = (uint8_t *)c->fx_rows;
    FxSlot *rows = (FxSlot *)c->fx_rows + marks;
    const int64_t chunk = std::min(chunk_elements(m), held);
    int epb = c->tune.elem_epb;
    if (t3 && epb != 32 && epb != 64) epb = 128;
    if (!t3 && epb != 8 && epb != 16) epb = 32;
    c->fx_marks.made();
    for (int64_t e0 = 0; e0 < m.nelem; e0 += chunk) {
        const int64_t n = std::min(chunk, m.nelem - e0);
        const unsigned groups = (unsigned)((n + FX_GROUP - 1) / FX_GROUP);
        if (t3) {
            k_t3_rows<<<nblk2(n, epb), epb, 0, c->stream>>>(m, c->mc, e0, n, rows, redo, c->d_status);
            k_t3_gram<<<groups, 96, sizeof(FxSlot) * FX_GROUP * T3_SLOTS, c->stream>>>(m, e0, n, rows, ke);
        } else {
            k_q4_rows<<<nblk2(n, epb), 4 * epb, 0, c->stream>>>(m, c->mc, e0, n, rows, redo, c->d_status);
            k_q4_gram<<<groups, 128, 0, c->stream>>>(m, e0, n, rows, ke);
        }
    }
    FS_CUDA(c, cudaGetLastError());
    return FS_OK;
}

// The status bits after the element kernels (and the gather into `vals`, if not
// null) have run; elements marked for it are done in double first, and
// gathered again.
int read_element_status(fs_ctx *c, int precision, void *ke, double *vals, int *bits)
{
    FS_TRY(read_status(c, bits));
    const bool redo = c->fx_marks.redo(*bits & DEV_REDO);
    const int first = *bits &= ~DEV_REDO;
    if (!redo) return FS_OK;
    FS_TRY(c->mesh.nen == 3 ? redo_t3(c, (double *)ke, (const uint8_t *)c->fx_rows) : redo_q4(c, (double *)ke, (const uint8_t *)c->fx_rows));
    if (vals) FS_TRY(launch_gather_from(c, precision, ke, vals));
    FS_TRY(read_status(c, bits));
    *bits |= first;
    return FS_OK;
}

}  // namespace fs
