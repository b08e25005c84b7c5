// exg_p2g.cuh -- K2: P2G of mass, momentum, force and the thermal channels
// (deposit_onto_grid_momentum, mpm_particle_grid_ops.cpp:405-588, and the
// thermal deposit, :703-844).  Included by exg_kernels.cu inside its
// anonymous namespace.
//
// One warp walks one row of T cells (nearest-node bins for quadratic) along
// x; the row's particles are contiguous after the sort.  32 (FP64: 16) particles at a
// time, one lane per particle loads the particle and leaves a record in the
// warp's shared memory: its deposit terms and its W weights per axis.  Then
// the warp reads the records back with the lanes laid out over the stencil:
// a lane owns the (y, z) pair of one of the W x W node columns, holds the
// column's W x-nodes in registers, and groups of W x W lanes take different
// particles of the same cell (2 for cubic, 3 for quadratic, 8 for linear).
// With N = wx wy wz and grad N = (dwx wy wz, wx dwy wz, wx wy dwz), a lane
// forms the row terms of its (y, z) once per particle,
//   m wy wz,  m v_d wy wz,  A_d = b_d wy wz + s_d1 dwy wz + s_d2 wy dwz,
//   C_d = s_d0 wy wz          (s = -V sigma, b = m g + external force),
// and adds wx A + dwx C to its nodes: 10 multiply-adds per node, no weight
// or term computed more than once per particle.  When the warp moves from
// cell cx to the next, no later cell of the row reaches node column cx, so
// that column alone is summed over the groups and added to the item's
// fixed-point node block: a quarter (third, half) of a cell's nodes instead
// of all of them.  The registers of the columns are addressed by node index
// mod W, and the records hold the x weights in the same rotation, so nothing
// is moved when the window slides.
//
// Every node's register sum runs over the particles in storage order with a
// fixed split over the groups, and the fixed-point adds are exact, so the
// result depends neither on the number of warps nor on which block takes
// which row: all launch shapes, the split of a tile into items and the
// batched kernel give the same bits.
#pragma once

// Particles staged per round.
template <class R>
constexpr int kP2GChunk = sizeof(R) == 4 ? 32 : 16;

// Launch shapes: most threads per block (fewer where their records do not
// fit shared memory).  The kernel waits on fixed latencies, shared memory and
// its particle loads, so warps decide its speed until registers spill: FP32
// cubic 988 / 852 / 925 us at 12 / 16 / 20 warps (9 M spheres), quadratic
// 800 / 699 / 622 us (8 M dam break); FP64 cubic 315 / 430 us at 12 / 16
// (1.1 M spheres).
constexpr int kP2GVariants = 3;
static_assert(kP2GVariants == EXG_NUM_VARIANTS, "the launchers dispatch EXG_NUM_VARIANTS P2G variants");
// The shape with one node block instead of two (Params::nbuf).
constexpr int kP2GOneBuf = kP2GVariants;
template <class R, int ORD, int VAR>
struct P2GVar {
    static constexpr int NBUF = VAR == kP2GOneBuf ? 1 : 2, V = VAR == kP2GOneBuf ? 0 : VAR;
    static constexpr int TAB[3][3] = {{512, 640, 384}, {640, 512, 384}, {384, 512, 256}};
    static constexpr int THREADS = TAB[sizeof(R) == 8 ? 2 : (P2GStc<ORD>::W == 4 ? 0 : 1)][V];
};

// Fixed-point values of an item's node block, rounded up to a multiple of 4
// (16-byte accesses).
template <bool THERM>
__host__ __device__ inline int p2g_values(const Params &P) {
    return ((THERM ? CH_ALL : CH_MOM_END) * P.PS * P.Bz + 3) & ~3;
}

// A particle's record, in elements of R: the terms
//   m p0 p1 p2 | b0 b1 s1 s3 | s2 s4 s0 s1 | b2 s4 s5 s2   (pairs as the
// packed FP32 instructions take them), with temperature
//   m cp, m cp T, m k, V Q | V q0, V q1, V q2, -,
// then (wx, dwx)[W], (wy, dwy)[W], (wz, dwz)[W].  The stride keeps the
// 16-byte accesses of consecutive records on different banks.
template <class R, int W, bool THERM>
struct P2GRec {
    static constexpr int V16 = 16 / sizeof(R);
    // (YO starts on a 16-byte boundary: W = 3 leaves two elements unused)
    static constexpr int XO = 16 + (THERM ? 8 : 0), YO = XO + 2 * (W + W % 2), ZO = YO + 2 * W, N = ZO + 2 * W;
    static_assert(XO % V16 == 0 && YO % V16 == 0, "16-byte accesses");
    static constexpr int UNITS = (N + V16 - 1) / V16;
    static constexpr int STRIDE = (UNITS | 1) * V16;
};

// Register sums of one node.  FP32 keeps channel pairs in float2 for the
// packed FP32 multiply-add.
template <class R, bool THERM>
struct P2GAcc {
    R c[THERM ? CH_ALL : CH_MOM_END];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < (THERM ? CH_ALL : CH_MOM_END); ++i) c[i] = R(0);
    }
    __device__ __forceinline__ R get(int ch) const { return c[ch]; }
};
template <bool THERM>
struct P2GAcc<float, THERM> {
    float2 mp0, p12, f01, t01, t23;
    float f2;
    __device__ __forceinline__ void zero() {
        mp0 = p12 = f01 = t01 = t23 = make_float2(0.f, 0.f);
        f2 = 0.f;
    }
    __device__ __forceinline__ float get(int ch) const {
        switch (ch) {
            case CH_M: return mp0.x;
            case CH_P: return mp0.y;
            case CH_P + 1: return p12.x;
            case CH_P + 2: return p12.y;
            case CH_F: return f01.x;
            case CH_F + 1: return f01.y;
            case CH_F + 2: return f2;
            case CH_MC: return t01.x;
            case CH_MCT: return t01.y;
            case CH_MK: return t23.x;
            default: return t23.y;
        }
    }
};

// How a warp's lanes cover the W x W (y, z) pairs: groups, and the channels
// a lane adds to the node block after the sum over the groups.
template <int W>
struct P2GLanes {
    static constexpr int G = W == 4 ? 2 : (W == 3 ? 3 : 8);
    int yz, grp;
    __device__ __forceinline__ P2GLanes() {
        const int lane = threadIdx.x & 31;
        yz = W == 3 ? lane % 9 : lane % (W * W);
        grp = W == 3 ? lane / 9 : lane / (W * W);
    }
    __device__ __forceinline__ bool active() const { return W != 3 || grp < 3; }
    // channels owned by the lane: first() + i * STEP for i < own<NCH>()
    static constexpr int STEP = W == 3 ? 3 : 1;
    template <int NCH>
    __host__ __device__ static constexpr int own() {
        if (W == 3) return (NCH + 2) / 3;
        int n = NCH;
        for (int g = G; g > 1; g >>= 1) n = (n + 1) / 2;
        return n;
    }
    // first owned channel and one past the last one the lane may own
    template <int NCH>
    __device__ __forceinline__ void first(int &c0, int &c1) const {
        if (W == 3) {
            c0 = grp;
            c1 = active() ? NCH : 0;
            return;
        }
        int n = NCH, lo = 0, hi = NCH;
#pragma unroll
        for (int m = G >> 1; m >= 1; m >>= 1) {
            const int half = (n + 1) / 2;
            if (grp & m)
                lo += half;
            else
                hi = min(hi, lo + half);
            n = half;
        }
        c0 = lo;
        c1 = hi;
    }
    // Sums v[0..NCH) over the groups; the lane's owned channels end in
    // v[0..own).  A fixed order whatever the launch.
    template <class R, int NCH>
    __device__ __forceinline__ void reduce(R (&v)[NCH]) const {
        constexpr unsigned FULL = 0xffffffffu;
        if constexpr (W == 3) {
            const int s1 = yz + 9 * (grp >= 2 ? 0 : grp + 1), s2 = yz + 9 * (grp == 0 ? 2 : (grp == 1 ? 0 : 1));
#pragma unroll
            for (int i = 0; i < (NCH + 2) / 3; ++i) {
                const R a = v[3 * i], b = 3 * i + 1 < NCH ? v[3 * i + 1 < NCH ? 3 * i + 1 : 0] : R(0),
                        c = 3 * i + 2 < NCH ? v[3 * i + 2 < NCH ? 3 * i + 2 : 0] : R(0);
                // channel 3 i + (grp + j) % 3 for j = 0, 1, 2
                const R a0 = grp == 0 ? a : (grp == 1 ? b : c), a1 = grp == 0 ? b : (grp == 1 ? c : a),
                        a2 = grp == 0 ? c : (grp == 1 ? a : b);
                const R x = __shfl_sync(FULL, a2, s1), y = __shfl_sync(FULL, a1, s2);
                v[i] = a0 + (x + y);
            }
        } else {
            int n = NCH;
#pragma unroll
            for (int m = G >> 1; m >= 1; m >>= 1) {
                const int half = (n + 1) / 2;
                const bool up = grp & m;
#pragma unroll
                for (int i = 0; i < NCH; ++i) {
                    if (i >= half) continue;
                    const R a = v[i], b = i + half < n ? v[i + half < NCH ? i + half : 0] : R(0);
                    const R got = __shfl_xor_sync(FULL, up ? a : b, m * W * W);
                    v[i] = (up ? b : a) + got;
                }
                n = half;
            }
        }
    }
};

// Whether every node of a cell's (bin's) window along axis d has the interior
// shape type.
template <int ORD>
__device__ __forceinline__ bool p2g_interior(const Params &P, int d, int iv) {
    return ORD == 1 || (ORD != 0 && (P.periodic[d] || (iv >= 3 && iv <= P.nc[d] - (ORD == 2 ? 3 : 4))));
}

// What the particles of one row share: the cell (bin) along y and z, whether
// it is interior there, and its coordinate.
struct P2GRow {
    int iv[2];
    bool inter[2];
    double xo[2];
};

// Loads particle p and writes its record.  x0: the tile's first cell along x.
template <class R, int ORD, bool THERM>
__device__ __forceinline__ void p2g_record(const SplineTables &tab, const Params &P, const Parts<R> &A, int p, int x0,
                                           const P2GRow &row, const R *grav, R *rec) {
    constexpr int W = P2GStc<ORD>::W;
    using L = P2GRec<R, W, THERM>;
    const bool live = A.phase[p] == 0;
    double x[3] = {A.x[0][p], A.x[1][p], A.x[2][p]};
    R m = A.mass[p], vol = A.vol[p], v[3], s[6], b[3], th[8];
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = A.v[d][p];
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] = A.sig[c][p];
    if constexpr (THERM) {
        th[0] = A.cp[p];
        th[1] = (R)(A.T[p] - P.Tref);
        th[2] = A.kc[p];
        th[3] = A.Q[p];
#pragma unroll
        for (int d = 0; d < 3; ++d) th[4 + d] = A.q[d][p];
        th[7] = R(0);
    }
    if (__any_sync(__activemask(), !live) && !live) {  // deposits nothing, whatever it holds
        m = vol = R(0);
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = R(0);
#pragma unroll
        for (int c = 0; c < 6; ++c) s[c] = R(0);
        if constexpr (THERM) {
#pragma unroll
            for (int c = 0; c < 8; ++c) th[c] = R(0);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) b[d] = m * grav[d];
    if (P.external_loads && live && x[0] > P.slab_lo[0] && x[0] < P.slab_hi[0] && x[1] > P.slab_lo[1] &&
        x[1] < P.slab_hi[1] && x[2] > P.slab_lo[2] && x[2] < P.slab_hi[2]) {
#pragma unroll
        for (int d = 0; d < 3; ++d) b[d] = fma(m, grav[d], (R)P.extforce[d]);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] = -vol * s[c];
    const R val[16] = {m,    m * v[0], m * v[1], m * v[2], b[0], b[1], s[1], s[3],
                       s[2], s[4],     s[0],     s[1],     b[2], s[4], s[5], s[2]};
    auto put = [&](int at, const R *q, int n) {  // 16-byte stores
        if constexpr (sizeof(R) == 4) {
            for (int i = 0; i < n; i += 4)
                *reinterpret_cast<float4 *>(rec + at + i) = make_float4(q[i], q[i + 1], q[i + 2], q[i + 3]);
        } else {
            for (int i = 0; i < n; i += 2) *reinterpret_cast<double2 *>(rec + at + i) = make_double2(q[i], q[i + 1]);
        }
    };
    put(0, val, 16);
    if constexpr (THERM) {
        const R mcp = m * th[0];
        const R tv[8] = {mcp,         (R)(mcp * th[1]), m * th[2],   vol * th[3],
                         vol * th[4], vol * th[5],      vol * th[6], R(0)};
        put(16, tv, 8);
    }
    // the cell (bin) along x as the sort key has it
    const int ivx = ORD == 2 ? dual_bin(P, 0, x[0]) : (int)floor((x[0] - P.plo[0]) * P.dxi[0]);
    const int iv[3] = {ivx, row.iv[0], row.iv[1]};
    const bool inter[3] = {p2g_interior<ORD>(P, 0, ivx), row.inter[0], row.inter[1]};
    const double xo[3] = {P.plo[0] + ivx * P.dx[0], row.xo[0], row.xo[1]};
    AxisW<R, W> a[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double xw = ORD == 2 ? dual_x(P, d, x[d]) : x[d];
        if constexpr (ORD == 2 || ORD == 3)
            fact_axis_weights<R, ORD>(tab, P, d, xw, iv[d], inter[d], (R)((xw - xo[d]) * P.dxi[d]), a[d]);
        else
            p2g_axis_weights<R, ORD>(tab, P, d, xw, iv[d], inter[d], a[d]);
    }
    // x weights rotated: node (first node of the window + s) at its index mod W
    int at = max(ivx - x0, 0) % W;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        if constexpr (sizeof(R) == 4)
            *reinterpret_cast<float2 *>(rec + L::XO + 2 * at) = make_float2(a[0].w[i], a[0].dw[i]);
        else
            *reinterpret_cast<double2 *>(rec + L::XO + 2 * at) = make_double2(a[0].w[i], a[0].dw[i]);
        at = W == 3 ? (at == 2 ? 0 : at + 1) : (at + 1) & (W - 1);
    }
    R yz[4 * W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
        yz[2 * i] = a[1].w[i];
        yz[2 * i + 1] = a[1].dw[i];
        yz[2 * W + 2 * i] = a[2].w[i];
        yz[2 * W + 2 * i + 1] = a[2].dw[i];
    }
    put(L::YO, yz, 4 * W);
}

// One particle's record into the W nodes of a lane's column.
template <class R, int W, bool THERM>
__device__ __forceinline__ void p2g_add(const R *rec, int sy, int sz, P2GAcc<R, THERM> (&acc)[W]) {
    using L = P2GRec<R, W, THERM>;
    if constexpr (sizeof(R) == 4) {
        const float4 q0 = *reinterpret_cast<const float4 *>(rec), q1 = *reinterpret_cast<const float4 *>(rec + 4),
                     q2 = *reinterpret_cast<const float4 *>(rec + 8), q3 = *reinterpret_cast<const float4 *>(rec + 12);
        const float2 y = *reinterpret_cast<const float2 *>(rec + L::YO + 2 * sy);
        const float2 z = *reinterpret_cast<const float2 *>(rec + L::ZO + 2 * sz);
        float2 x[W];
#pragma unroll
        for (int i = 0; i < W; i += 2) {
            if (i + 1 < W) {
                const float4 u = *reinterpret_cast<const float4 *>(rec + L::XO + 2 * i);
                x[i] = make_float2(u.x, u.y);
                x[i + 1 < W ? i + 1 : i] = make_float2(u.z, u.w);
            } else {
                x[i] = *reinterpret_cast<const float2 *>(rec + L::XO + 2 * i);
            }
        }
        const float wyz = y.x * z.x, dyz = y.y * z.x, wdz = y.x * z.y;
        const float2 wyz2 = make_float2(wyz, wyz), dyz2 = make_float2(dyz, dyz), wdz2 = make_float2(wdz, wdz);
        const float2 mp0 = __fmul2_rn(wyz2, make_float2(q0.x, q0.y)), p12 = __fmul2_rn(wyz2, make_float2(q0.z, q0.w));
        const float2 a01 = __ffma2_rn(wdz2, make_float2(q2.x, q2.y),
                                      __ffma2_rn(dyz2, make_float2(q1.z, q1.w),
                                                 __fmul2_rn(wyz2, make_float2(q1.x, q1.y))));
        const float2 c01 = __fmul2_rn(wyz2, make_float2(q2.z, q2.w));
        const float a2 = fmaf(wdz, q3.z, fmaf(dyz, q3.y, wyz * q3.x)), c2 = wyz * q3.w;
        float2 t01 = make_float2(0.f, 0.f), t23 = t01;
        float tc = 0.f;
        if constexpr (THERM) {
            const float4 q4 = *reinterpret_cast<const float4 *>(rec + 16),
                         q5 = *reinterpret_cast<const float4 *>(rec + 20);
            t01 = __fmul2_rn(wyz2, make_float2(q4.x, q4.y));
            t23 = __fmul2_rn(wyz2, make_float2(q4.z, q4.w));
            t23.y = fmaf(wdz, q5.z, fmaf(dyz, q5.y, t23.y));
            tc = wyz * q5.x;
        }
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const float2 w2 = make_float2(x[i].x, x[i].x), d2 = make_float2(x[i].y, x[i].y);
            acc[i].mp0 = __ffma2_rn(w2, mp0, acc[i].mp0);
            acc[i].p12 = __ffma2_rn(w2, p12, acc[i].p12);
            acc[i].f01 = __ffma2_rn(w2, a01, acc[i].f01);
            acc[i].f01 = __ffma2_rn(d2, c01, acc[i].f01);
            acc[i].f2 = fmaf(x[i].x, a2, acc[i].f2);
            acc[i].f2 = fmaf(x[i].y, c2, acc[i].f2);
            if constexpr (THERM) {
                acc[i].t01 = __ffma2_rn(w2, t01, acc[i].t01);
                acc[i].t23 = __ffma2_rn(w2, t23, acc[i].t23);
                acc[i].t23.y = fmaf(x[i].y, tc, acc[i].t23.y);
            }
        }
    } else {
        double q[THERM ? 24 : 16];
#pragma unroll
        for (int i = 0; i < (THERM ? 24 : 16); i += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(rec + i);
            q[i] = t.x;
            q[i + 1] = t.y;
        }
        const double2 y = *reinterpret_cast<const double2 *>(rec + L::YO + 2 * sy);
        const double2 z = *reinterpret_cast<const double2 *>(rec + L::ZO + 2 * sz);
        const double wyz = y.x * z.x, dyz = y.y * z.x, wdz = y.x * z.y;
        constexpr int NCH = THERM ? CH_ALL : CH_MOM_END;
        double a[NCH], c[4];  // c: the dwx terms of the force and of the source
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = wyz * q[k];
        a[CH_F] = fma(wdz, q[8], fma(dyz, q[6], wyz * q[4]));
        a[CH_F + 1] = fma(wdz, q[9], fma(dyz, q[7], wyz * q[5]));
        a[CH_F + 2] = fma(wdz, q[14], fma(dyz, q[13], wyz * q[12]));
        c[0] = wyz * q[10];
        c[1] = wyz * q[11];
        c[2] = wyz * q[15];
        if constexpr (THERM) {
#pragma unroll
            for (int k = 0; k < 3; ++k) a[CH_MC + k] = wyz * q[16 + k];
            a[CH_SRC] = fma(wdz, q[22], fma(dyz, q[21], wyz * q[19]));
            c[3] = wyz * q[20];
        }
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const double2 x = *reinterpret_cast<const double2 *>(rec + L::XO + 2 * i);
            const double wx = x.x, dwx = x.y;
#pragma unroll
            for (int k = 0; k < NCH; ++k) acc[i].c[k] = fma(wx, a[k], acc[i].c[k]);
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[i].c[CH_F + d] = fma(dwx, c[d], acc[i].c[CH_F + d]);
            if constexpr (THERM) acc[i].c[CH_SRC] = fma(dwx, c[3], acc[i].c[CH_SRC]);
        }
    }
}

// A block's node blocks (two; one where the staging of split tiles is too
// much, see p2g_split) and what its warps know of the item in each.
// The block works through a sequence of items, item n in buffer n % NBUF.  Warps
// take rows of an item from `next`; a warp that finds none left leaves for
// the next item without waiting for the rest.  The last warp to leave writes
// the item's node block out and zeroes it.  The next item is taken by the
// warp that draws the present one's last row (or the first one to want it):
// late, so that the last items of a launch spread over the blocks, but ahead
// of its first use.  Every warp passes through every item, so none can take a
// row of an item it has not read the header of.
struct P2GBuf {
    int item;        // item, or -1: no more
    int scene;       // scene of a batch
    int next, left;  // next row to take, warps that have not left
    int tile;        // tile, its coordinates, first particle
    int tc[3], s0;
    int part;        // the item's z planes: part * SZ ...
    // items of this buffer: whose opening is under way or done, opened
    // (written last), written out
    int req, opened, freed;
};

// Shared memory of a P2G block: spline tables, the one or two fixed-point node
// blocks (nv values each, nv a multiple of 4), the warps' records.
__host__ __device__ constexpr size_t p2g_acc_off() { return (sizeof(SplineTables) + 15) & ~size_t(15); }
template <class R>
__host__ __device__ constexpr size_t p2g_buf_bytes(int nv) { return sizeof(unsigned) * (fx_lo_words<R>() + 1) * (size_t)nv; }
template <class R, int ORD, bool THERM>
__host__ __device__ constexpr size_t p2g_warp_bytes() {
    return sizeof(R) * P2GRec<R, P2GStc<ORD>::W, THERM>::STRIDE * kP2GChunk<R>;
}
// Bounded waits for an item to be opened or written out by another warp of
// the block, in polls of 64 ns or more: a minute at least.  One warp walks a row
// whatever it holds (four million FP64 cubic particles in one row take it over
// a second), and as many as fit the device's memory take it less than that.  A
// bound by the particles of the launch cost the quadratic P2G 1.6 % (0.9 M
// particles 106.5 -> 108.2 us), a constant one nothing.
constexpr int kP2GWaitLimit = 1 << 30;

// The block's share of a P2G launch.  Src gives the items and, per scene,
// the grid and the particles: take(scene) is called by one lane and returns
// the next item or -1.
template <class R, int ORD, bool THERM, int NBUF, class Src>
__device__ __forceinline__ void p2g_run(const Src &src, unsigned char *smraw, P2GBuf *bufs, int nv, int pshift) {
    constexpr int W = P2GStc<ORD>::W, NCH = THERM ? CH_ALL : CH_MOM_END;
    using Lay = P2GRec<R, W, THERM>;
    using Ln = P2GLanes<W>;
    constexpr int G = Ln::G, NO = Ln::template own<NCH>();
    constexpr unsigned FULL = 0xffffffffu;
    SplineTables *tab = reinterpret_cast<SplineTables *>(smraw);
    unsigned char *accs = smraw + p2g_acc_off();
    R *rec = reinterpret_cast<R *>(accs + NBUF * p2g_buf_bytes<R>(nv) + (threadIdx.x >> 5) * p2g_warp_bytes<R, ORD, THERM>());
    load_tables(tab);
    for (int i = threadIdx.x; i < (int)(NBUF * p2g_buf_bytes<R>(nv) / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(accs)[i] = make_uint4(0u, 0u, 0u, 0u);
    step_kernel_begin(src.early());
    const int lane = threadIdx.x & 31;
    const Ln ln;
    const int sy = ln.yz % W, sz = ln.yz / W;
    int ch0, ch1;
    ln.template first<NCH>(ch0, ch1);
    const bool last = ch0 + (NO - 1) * Ln::STEP < ch1;  // the lane owns its last channel slot
    // the whole warp; false: gave up
    auto wait = [&](const P2GBuf &q, const int *what, int least) {
        for (int it = 0; it < kP2GWaitLimit; ++it) {
            const int o = lane == 0 ? *reinterpret_cast<const volatile int *>(what) : 0;
            if (__shfl_sync(FULL, o, 0) >= least) {
                __threadfence_block();
                return true;
            }
            __nanosleep(64);
        }
        if (lane == 0) src.fail(q.scene, ST_TIMEOUT);
        return false;
    };
    // opens item s of buffer q if no other warp does (the whole warp)
    auto open = [&](P2GBuf &q, int s) {
        int won = 0;
        if (lane == 0) won = atomicCAS(&q.req, s, s + 1) == s;
        if (!__shfl_sync(FULL, won, 0)) return true;
        if (!wait(q, &q.freed, s)) return false;
        if (lane == 0) {
            int scene = 0;
            const int item = src.take(scene);
            q.item = item;
            if (item >= 0) {
                const int w = item >> pshift, t = src.active(scene)[w];
                q.scene = scene;
                q.tile = w;
                q.part = item & ((1 << pshift) - 1);
                tile_coords(src.params(scene), t, q.tc);
                q.s0 = src.start(scene)[t];
                q.next = 0;
                q.left = (int)(blockDim.x >> 5);
            }
            __threadfence_block();
            *reinterpret_cast<volatile int *>(&q.opened) = s + 1;
        }
        __syncwarp();
        return true;
    };
    if (threadIdx.x < 2)
        bufs[threadIdx.x].scene = bufs[threadIdx.x].req = bufs[threadIdx.x].opened = bufs[threadIdx.x].freed = 0;
    __syncthreads();
    P2GAcc<R, THERM> acc[W];
#pragma unroll
    for (int i = 0; i < W; ++i) acc[i].zero();
    R sc[NO], grav[3];
    int cur = -1;  // scene of sc and grav
    for (int n = 0;; ++n) {
        const int b = n & (NBUF - 1), s = n >> (NBUF - 1);
        P2GBuf &q = bufs[b];
        if (!open(q, s) || !wait(q, &q.opened, s + 1)) return;
        const int item = *reinterpret_cast<volatile int *>(&q.item);
        if (item < 0) break;
        const int scene = q.scene;
        const Params &P = src.params(scene);
        const Parts<R> &A = src.parts(scene);
        const int32_t *perm = src.perm(scene);
        if (scene != cur) {
            cur = scene;
            const Ctl *ctl = src.ctl(scene);
#pragma unroll
            for (int i = 0; i < NO; ++i)
                sc[i] = ch0 + i * Ln::STEP < ch1 ? (R)ctl->scale[ch0 + i * Ln::STEP] : R(0);
#pragma unroll
            for (int d = 0; d < 3; ++d) grav[d] = (R)P.gravity[d];
        }
        const int B = P.B, T = P.T, SZ = T >> pshift, nrow = T * SZ;
        const int tc[3] = {q.tc[0], q.tc[1], q.tc[2]}, s0 = q.s0, z0 = q.part * SZ;
        const int *cs = src.cell_start(scene) + (long long)q.tile * (T * T * T + 1);
        unsigned char *blk = accs + b * p2g_buf_bytes<R>(nv);
        const int B3 = P.PS * P.Bz, at0 = ch0 * B3 + sz * P.PS + sy * B;
        for (;;) {
            int row = 0;
            if (lane == 0) row = atomicAdd(&q.next, 1);
            row = __shfl_sync(FULL, row, 0);
            if (row >= nrow) break;
            if (NBUF == 2 && row == nrow - 1) {
                // ahead of the next item's first use, if its buffer is free
                P2GBuf &qn = bufs[b ^ 1];
                const int sn = (n + 1) >> 1, f = lane == 0 ? *reinterpret_cast<volatile int *>(&qn.freed) : 0;
                if (__shfl_sync(FULL, f, 0) >= sn && !open(qn, sn)) return;
            }
            const int ly = row & (T - 1), lz = (row >> P.tshift) + z0;
            // lane i holds the first particle of the row's cell i, lane T the row's end
            const int bound = lane <= T ? cs[(((lz << P.tshift) | ly) << P.tshift) + lane] : 0;
            const int r1 = __shfl_sync(FULL, bound, T);
            int k = __shfl_sync(FULL, bound, 0), cb = k, ce = k;  // next particle; the staged ones are cb .. ce - 1
            if (k >= r1) continue;
            P2GRow rw;
            rw.iv[0] = tc[1] * T + ly;
            rw.iv[1] = tc[2] * T + lz;
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                rw.inter[d] = p2g_interior<ORD>(P, d + 1, rw.iv[d]);
                rw.xo[d] = P.plo[d + 1] + rw.iv[d] * P.dx[d + 1];
            }
            int at = at0 + (lz - z0) * P.PS + ly * B;  // the lane's column, node 0, first owned channel
            int pend = 0;  // node columns from the present cell's on that hold something
            // the particles of cell c
            auto deposit = [&](int c) {
                const int kend = c < T ? __shfl_sync(FULL, bound, c + 1) : k;
                if (k >= kend) return;
                pend = W;
                do {
                    if (k >= ce) {
                        __syncwarp();
                        cb = k;
                        ce = min(k + kP2GChunk<R>, r1);
                        if (cb + lane < ce)
                            p2g_record<R, ORD, THERM>(*tab, P, A, perm[s0 + cb + lane], tc[0] * T, rw, grav,
                                                      rec + lane * Lay::STRIDE);
                        __syncwarp();
                    }
                    const int lim = min(kend, ce);
                    const R *q1 = rec + (lim - cb) * Lay::STRIDE;
                    for (const R *qr = ln.active() ? rec + (k - cb + ln.grp) * Lay::STRIDE : q1; qr < q1;
                         qr += G * Lay::STRIDE)
                        p2g_add<R, W, THERM>(qr, sy, sz, acc);
                    k = lim;
                } while (k < kend);
            };
            // node column c, held in registers c mod W: after cell c no later
            // particle of the row reaches it
            auto flush = [&](auto sl) {
                constexpr int j = decltype(sl)::value < W ? decltype(sl)::value : 0;
                if (pend > 0) {
                    R v[NCH];
#pragma unroll
                    for (int ch = 0; ch < NCH; ++ch) v[ch] = acc[j].get(ch);
                    acc[j].zero();
                    ln.template reduce<R, NCH>(v);
#pragma unroll
                    for (int i = 0; i < NO; ++i)
                        if (W == 2 ? ch0 + i < ch1 : ln.active() && (i < NO - 1 || last))
                            fx_add_r<R>(blk, nv, at + i * Ln::STEP * B3, v[i], sc[i]);
                    --pend;
                }
                ++at;
            };
            using I0 = std::integral_constant<int, 0>;
            using I1 = std::integral_constant<int, 1>;
            using I2 = std::integral_constant<int, 2>;
            using I3 = std::integral_constant<int, 3>;
            if constexpr (sizeof(R) == 4) {
                // W cells at a time: the registers of a column are known when
                // compiled (cubic 844 against 870 us with the switch below)
                for (int c = 0; c < T || pend > 0; c += W) {
                    deposit(c);
                    flush(I0{});
                    deposit(c + 1);
                    flush(I1{});
                    if constexpr (W > 2) {
                        deposit(c + 2);
                        flush(I2{});
                    }
                    if constexpr (W > 3) {
                        deposit(c + 3);
                        flush(I3{});
                    }
                }
            } else {
                // FP64: the unrolled code costs more registers than the
                // switch does instructions (320 against 345 us)
                int slot = 0;
                for (int c = 0; c < T || pend > 0; ++c) {
                    deposit(c);
                    switch (slot) {
                        case 0: flush(I0{}); break;
                        case 1: flush(I1{}); break;
                        case 2: flush(I2{}); break;
                        default: flush(I3{}); break;
                    }
                    slot = slot == W - 1 ? 0 : slot + 1;
                }
            }
        }
        // the warp's adds are done before it counts as having left
        __threadfence_block();
        __syncwarp();
        int left = 0;
        if (lane == 0) left = atomicSub(&q.left, 1);
        if (__shfl_sync(FULL, left, 0) == 1) {
            __threadfence_block();
            fx_store_zero<R>(blk, nv, src.staging(scene) + (long long)item * stg_stride<R>(nv));
            __threadfence_block();
            __syncwarp();
            if (lane == 0) *reinterpret_cast<volatile int *>(&q.freed) = s + 1;
        }
    }
}

// Items of one scene, taken in turn from a device counter.
template <class R>
struct P2GScene {
    const Params &P;
    const Parts<R> &A;
    const int *act, *st, *cst;
    const int32_t *pm;
    long long *stg;
    Ctl *c;
    int pshift;
    __device__ __forceinline__ int take(int &) const {
        const int i = atomicAdd(&c->next_p2g, 1);
        return i < c->n_active_tiles << pshift ? i : -1;
    }
    __device__ __forceinline__ bool early() const { return step_early(P); }
    __device__ __forceinline__ const Params &params(int) const { return P; }
    __device__ __forceinline__ const Parts<R> &parts(int) const { return A; }
    __device__ __forceinline__ const int *active(int) const { return act; }
    __device__ __forceinline__ const int *start(int) const { return st; }
    __device__ __forceinline__ const int *cell_start(int) const { return cst; }
    __device__ __forceinline__ const int32_t *perm(int) const { return pm; }
    __device__ __forceinline__ long long *staging(int) const { return stg; }
    __device__ __forceinline__ const Ctl *ctl(int) const { return c; }
    __device__ __forceinline__ void fail(int, unsigned st) const { atomicOr(&c->status, st); }
};

template <class R, int ORD, bool THERM, int V>
__global__ void __launch_bounds__(P2GVar<R, ORD, V>::THREADS, 1)
    k_p2g(const __grid_constant__ Params P, const __grid_constant__ Parts<R> A, const int *active, const int *start,
          const int *cell_start, const int32_t *perm, long long *staging, Ctl *ctl) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ P2GBuf bufs[2];
    const P2GScene<R> src{P, A, active, start, cell_start, perm, staging, ctl, P.pshift};
    p2g_run<R, ORD, THERM, P2GVar<R, ORD, V>::NBUF>(src, smraw, bufs, p2g_values<THERM>(P), P.pshift);
}
