// poisson_cluster.cuh -- the whole Poisson solve of one grid in one
// thread-block cluster (included by poisson.cu, inside its namespaces).
//
// A solve of a grid that fits in the shared memory of 16 SMs is bound by
// latency when each of its phases is a launch: on 129^2 nodes an iteration is
// 7 kernels of 4 to 7 us whose work is a fraction of a microsecond.  Here one
// cluster of 16 blocks runs the PCG from overwriteRho to the E field, phases
// separated by block barriers, and by a cluster barrier only where blocks
// exchange data.
//
// Level 0 is cut into bands of node rows, one a block; block c owns a coarse
// node when it owns the fine node below it.  A block keeps x, b and the mask
// of its band of every distributed level in shared memory, with H halo rows on
// either side, and does all of a level's sweeps on the band and as much of the
// halo as they need (temporal blocking, as k_mg_down / k_mg_up: the region
// that is right shrinks by a row a sweep; the arithmetic of every node is
// theirs).  Levels of at most kClRepNodes nodes are kept whole by every block
// and worked on redundantly.  The coarsest step is a dense product with the
// inverse that PoissonState holds (k_mg_direct), its rows shared out.  Halo
// rows and shares are stored into the shared memory of the blocks that need
// them, before a cluster barrier.  On the way up the halo is wide enough that a
// level hands the next finer one all it needs.
//
// FP64 vectors stay in global memory (L2).  Each block works on whole groups of
// 32 nodes: those that start in its band.  phi, r and z of other blocks are
// read after a barrier and past L1.
//
// alpha and beta are the multi-kernel solve's bit for bit, and so is every
// iterate: r.z is summed in the order of k_mg_up's tiles, p.A p in that of
// k_pcg_pq's blocks.  |r|^2 and |b|^2, which only decide when to stop, are sums of
// the blocks' own: the two solvers end an iteration apart if a residual comes
// within some 1e-15 of the tolerance, and else give the same potential.
// A warp sums what one of their warps sums and stores it in every block, which
// then finishes the sum as reduce_finalize does.  That costs two cluster
// barriers an iteration more than sums of the blocks' own (of 129^2 nodes: 6 in
// place of 4 with each 1.3 us), but a run's particles amplify a last bit of phi
// to differences of 1e-9 in the density within some ten steps.

constexpr int kClBlocks = 16;      // a cluster (non-portable size)
// Grids up to this many nodes: beyond it the multi-kernel solve, on all SMs, is
// as fast or faster.  Measured, us a solve from zero to 1e-8, cluster / kernels:
// 33^2 nodes 44 / 88, 65^2 153 / 184, 101 x 71 224 / 246, 129^2 225 / 219, 161^2
// 276 / 250; us a step of a run (host work included): 33^2 83 / 113, 65^2 160 /
// 190, 97^2 204 / 223, 113^2 213 / 222, 129^2 226 / 222.
constexpr int64_t kClMaxNodes = 14000;
// And up to this many rows of level 0 (40 a block: every one of them is walked in
// push_rows, and narrow rows are padded).  Measured, us a solve, cluster / kernels /
// the kernels before their tiles held quads: periodic 7 x 480 cells 185 / 193 / 230,
// 16 x 640 251 / 220 / 266, 7 x 800 221 / 190 / 221, 7 x 1600 286 / 193 / 229, 10 x 1200
// 309 / 223 / 268; walls 8 x 480 310 / 310 / 336, 12 x 640 222 / 215 / 267, 8 x 1200 255 /
// 218 / 259.
constexpr int kClMaxRows = 641;
constexpr int kClThreads = 1024;
constexpr int kClMaxLevels = 8;
constexpr int kClRepNodes = 1500;  // levels up to this size are replicated
constexpr int kClDownHalo = 2 * kNu + 1;
static_assert(kNu == 2, "the cluster solve's sweeps are written for two");

// A row of a level's arrays: the red nodes ((i + j) even), then the black
// ones, each in order and padded to a multiple of four (padding counts as
// electrodes).  A half sweep then reads and writes quads of neighbouring
// nodes: 16-byte accesses, no bank conflicts, and a third of the instructions
// a node of the row-major form (whose sweeps were half of the solve's time).
struct ClLevel {
    int GX, GY;
    float cx, cy, icd, cd;
    const uint8_t* mask;
    int hw, rs;           // row layout: nodes of a colour (padded), row length = 2 hw
    uint32_t rcp_q, rcp_gx;  // ceil(2^32 / (hw / 4)), ceil(2^32 / GX): division by umulhi (the dividends are small)
    int dist;             // distributed (else every block has all rows)
    int H;                // halo rows on either side (0 when replicated)
    int U;                // rows beyond the band that the up sweep starts on
    int near;             // blocks this far away at most keep copies of a block's rows
    int ox, ob, om, oh;   // byte offsets in shared memory: x, b, mask, incoming halo rows of x
};

struct ClInst {
    int GX, GY, periodic, levels;  // levels: those above the dense one, lev[levels]
    int64_t nodes, sn;
    double cx, cy, cd, dx, dy;
    const uint8_t* mask;
    const double* dv;
    double* rho;
    double* phi;
    double* r;
    double* p;
    double* q;
    float* z;        // the V-cycle's result, for r.z (level 0 distributed)
    const double* bz;
    float4* fld;
    const float* inv;
    const int* freen;
    int nf, nfp, oc;  // free nodes of the dense level, row length of inv; offset of the right-hand side's copy
    int tx, tiles;    // k_mg_up's tiles of level 0: of a row of them, all
    int nblocks;      // blocks of k_pcg_pq
    int orz, opq;     // byte offsets of the warps' sums of r.z and p.A p, 8 a tile or block
    double* scal;
    double* host_scal;  // pinned
    double tol2;
    int maxit;
    int zero_start;  // phi starts at 0
    int overwrite;   // rho still holds the charge density (else b)
    ClLevel lev[kClMaxLevels + 1];
};

namespace cg = cooperative_groups;

// All threads of the cluster: their shared-memory and global writes before it
// are seen by the others' reads after it.  (Written out so that a warp whose
// lanes have just taken different branches may arrive lane by lane.)
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
}

struct ClShared {
    double red[2][kClThreads / 32];
    double part[3][kClBlocks][2];            // every block's partial sums, three in turn
    int start[kClMaxLevels + 1][kClBlocks + 1];  // first row of each level that each block owns
};

struct ClBlock {
    const ClInst& I;
    unsigned char* smem;
    ClShared& S;
    cg::cluster_group cluster;
    int rank, tid, slot;

    __device__ __forceinline__ float* X(int l) const { return reinterpret_cast<float*>(smem + I.lev[l].ox); }
    __device__ __forceinline__ float* B(int l) const { return reinterpret_cast<float*>(smem + I.lev[l].ob); }
    __device__ __forceinline__ float* XH(int l) const { return reinterpret_cast<float*>(smem + I.lev[l].oh); }
    __device__ __forceinline__ uint8_t* M(int l) const { return smem + I.lev[l].om; }
    __device__ __forceinline__ int start(int l, int c) const { return S.start[l][c]; }
    __device__ __forceinline__ int wrap(int l, int j) const {
        const int GY = I.lev[l].GY;
        j %= GY;
        return j < 0 ? j + GY : j;
    }

    // Sums of one or two values over the cluster (in place), the same bits in
    // every thread of every block; also a cluster barrier.  Each block stores
    // its partials in every block's table before the barrier (no remote read
    // after it).
    template <int N>
    __device__ __forceinline__ void sums(double (&v)[N]) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[n] += __shfl_xor_sync(kFull, v[n], o);
            if ((tid & 31) == 0) S.red[n][tid >> 5] = v[n];
        }
        __syncthreads();
        if (tid < 32) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
                v[n] = tid < kClThreads / 32 ? S.red[n][tid] : 0.0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v[n] += __shfl_xor_sync(kFull, v[n], o);
            }
            if (tid < kClBlocks) {
                double* to = cluster.map_shared_rank(&S.part[slot][rank][0], tid);
#pragma unroll
                for (int n = 0; n < N; ++n) to[n] = v[n];
            }
        }
        cluster_barrier();
#pragma unroll
        for (int n = 0; n < N; ++n) {
            v[n] = 0.0;
#pragma unroll
            for (int c = 0; c < kClBlocks; ++c) v[n] += S.part[slot][c][n];
        }
        slot = slot == 2 ? 0 : slot + 1;
    }

    // The sum of what the virtual warps of `blocks` blocks of 8 stored in `part`,
    // as reduce_finalize does it (at most 256 blocks); the same in every block.
    __device__ __forceinline__ double ordered_sum(const double* part, int blocks) {
        double x = 0.0;
        if (tid < kRedThreads) {
            if (tid < blocks) {
                double t = 0.0;
#pragma unroll
                for (int w = 0; w < kRedThreads / 32; ++w) t += part[tid * (kRedThreads / 32) + w];
                x += t;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
            if ((tid & 31) == 0) S.red[0][tid >> 5] = x;
        }
        __syncthreads();
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kRedThreads / 32; ++w) t += S.red[0][w];
        __syncthreads();
        return t;
    }

    // a warp's sum over its lanes, stored as entry v of `part` in every block
    __device__ __forceinline__ void share(double x, double* part, int v) const {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
        if ((tid & 31) < kClBlocks) cluster.map_shared_rank(part, tid & 31)[v] = x;
    }

    // Stores the rows of level l that this block owns, from its array `src`,
    // into the arrays of the blocks that keep a copy of them.  HALO false:
    // the same array there (all of it when the level is replicated, halo rows
    // otherwise); true: its incoming halo rows of x (U on either side).  A
    // warp a row.  (The receivers read the old values before the cluster
    // barrier that came last, the new ones after the next.)
    template <bool HALO>
    __device__ __forceinline__ void push_rows(int l, float* src) const {
        const ClLevel& L = I.lev[l];
        const int s = start(l, rank), e = start(l, rank + 1), lane = tid & 31;
        float* to = HALO ? XH(l) : src;
        // a warp an item: one of its own rows, one of the blocks near enough
        const int span = min(2 * L.near + 1, kClBlocks);
        for (int it = tid >> 5; it < (e - s) * span; it += kClThreads / 32) {
            const int jr = it / span, dd = it - jr * span - (span == kClBlocks ? 0 : L.near);
            const int j = s + jr;
            int d = span == kClBlocks ? dd : rank + dd;
            if (d < 0 || d >= kClBlocks) {
                if (!I.periodic) continue;
                d = d < 0 ? d + kClBlocks : d - kClBlocks;
            }
            const int sd = start(l, d), ed = start(l, d + 1);
            // the row itself and its images (periodic in y)
#pragma unroll 1
            for (int im = 0; im < (I.periodic && L.dist ? 3 : 1); ++im) {
                const int jj = im == 0 ? j : (im == 1 ? j - L.GY : j + L.GY);
                int lr = -1;
                if (!L.dist) lr = jj;
                else if (HALO) lr = jj >= sd - L.U && jj < sd ? jj - (sd - L.U) : (jj >= ed && jj < ed + L.U ? L.U + jj - ed : -1);
                else lr = jj >= sd - L.H && jj < ed + L.H ? jj - (sd - L.H) : -1;
                if (lr < 0 || (!HALO && d == rank && im == 0)) continue;
                const float4* row = reinterpret_cast<const float4*>(src + (L.dist ? j - (s - L.H) : j) * L.rs);
                float4* dst = reinterpret_cast<float4*>(cluster.map_shared_rank(to, d) + lr * L.rs);
#pragma unroll 2
                for (int i = lane; i < L.rs / 4; i += 32) dst[i] = row[i];
            }
        }
    }

    // index of node (i, j) of level l in a row array whose row `lr` is level row j
    __device__ __forceinline__ static int at(const ClLevel& L, int lr, int i, int j) {
        return lr * L.rs + (((i + j) & 1) ? L.hw : 0) + (i >> 1);
    }

    // one colour of Gauss-Seidel on the band and `rad` rows beyond it (all
    // rows when replicated), k_mg_rbgs's arithmetic; electrodes stay 0
    __device__ __forceinline__ void sweep(int l, int color, int rad) const {
        const ClLevel& L = I.lev[l];
        const int q = L.hw >> 2, rs = L.rs;
        const int j0 = L.dist ? start(l, rank) - rad : 0, rows = L.dist ? start(l, rank + 1) + rad - j0 : L.GY;
        const int r0 = L.dist ? L.H - rad : 0;
        float* x = X(l);
        const float* b = B(l);
        const uint8_t* m = M(l);
        for (int k = tid; k < rows * q; k += kClThreads) {
            const int jr = (int)__umulhi((uint32_t)k, L.rcp_q), h = 4 * (k - jr * q), lr = jr + r0;
            int up = lr + 1, dn = lr - 1;
            if (!L.dist) {  // rows wrap (only periodic in y; with walls rows 0 and GY - 1 are electrodes)
                up = up == L.GY ? 0 : up;
                dn = dn < 0 ? L.GY - 1 : dn;
            }
            const int own = color ? L.hw : 0, oth = L.hw - own, t = lr * rs + own + h;
            const bool odd = (j0 + jr + color) & 1;  // i = 2 h + odd
            const float* o = x + lr * rs + oth + h;
            const float4 c = *reinterpret_cast<const float4*>(o);
            const float e = odd ? o[4] : o[-1];
            const float4 u = *reinterpret_cast<const float4*>(x + up * rs + oth + h);
            const float4 d = *reinterpret_cast<const float4*>(x + dn * rs + oth + h);
            const float4 bv = *reinterpret_cast<const float4*>(b + t);
            const uint32_t mv = *reinterpret_cast<const uint32_t*>(m + t);
            // west + east: odd: c.x + c.y, ...; even: e + c.x, c.x + c.y, ...
            const float w0 = odd ? c.x : e, w1 = odd ? c.y : c.x, w2 = odd ? c.z : c.y, w3 = odd ? c.w : c.z;
            const float e3 = odd ? e : c.w;
            float4 v;
            v.x = __fmaf_rn(L.cx, w0 + w1, __fmaf_rn(L.cy, d.x + u.x, bv.x)) * L.icd;
            v.y = __fmaf_rn(L.cx, w1 + w2, __fmaf_rn(L.cy, d.y + u.y, bv.y)) * L.icd;
            v.z = __fmaf_rn(L.cx, w2 + w3, __fmaf_rn(L.cy, d.z + u.z, bv.z)) * L.icd;
            v.w = __fmaf_rn(L.cx, w3 + e3, __fmaf_rn(L.cy, d.w + u.w, bv.w)) * L.icd;
            if (mv & 0xffu) v.x = 0.0f;
            if (mv & 0xff00u) v.y = 0.0f;
            if (mv & 0xff0000u) v.z = 0.0f;
            if (mv & 0xff000000u) v.w = 0.0f;
            *reinterpret_cast<float4*>(x + t) = v;
        }
        __syncthreads();
    }

    // level l's smoothing from a zero start, then its residual's full
    // weighting into b of the level below, on the rows this block owns there
    // (all of them when l is replicated)
    __device__ __forceinline__ void down(int l) {
        const ClLevel& L = I.lev[l];
        const ClLevel& C = I.lev[l + 1];
        const int rs = L.rs, s = start(l, rank), e = start(l, rank + 1);
        float* x = X(l);
        const float* b = B(l);
        const uint8_t* m = M(l);
        {
            // red x = b / cd (as a product), black 0: quads of a row's two halves alike
            const int q = L.hw >> 2;
            const int r0 = L.dist ? L.H - kClDownHalo : 0, rows = L.dist ? e - s + 2 * kClDownHalo : L.GY;
            for (int k = tid; k < rows * q; k += kClThreads) {
                const int jr = (int)__umulhi((uint32_t)k, L.rcp_q), t = (jr + r0) * rs + 4 * (k - jr * q);
                const float4 bv = *reinterpret_cast<const float4*>(b + t);
                const uint32_t mv = *reinterpret_cast<const uint32_t*>(m + t);
                float4 v;
                v.x = (mv & 0xffu) ? 0.0f : bv.x * L.icd;
                v.y = (mv & 0xff00u) ? 0.0f : bv.y * L.icd;
                v.z = (mv & 0xff0000u) ? 0.0f : bv.z * L.icd;
                v.w = (mv & 0xff000000u) ? 0.0f : bv.w * L.icd;
                *reinterpret_cast<float4*>(x + t) = v;
                *reinterpret_cast<float4*>(x + t + L.hw) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            __syncthreads();
        }
        sweep(l, 1, kClDownHalo - 1);
        sweep(l, 0, kClDownHalo - 2);
        sweep(l, 1, kClDownHalo - 3);
        if (L.dist) push_rows<true>(l, x);
        // residual of the node at half index h of a colour in local row lr;
        // odd: its column is odd.  0 at electrodes.
        auto row = [&](int lr) {
            if (!L.dist) lr = lr < 0 ? lr + L.GY : (lr >= L.GY ? lr - L.GY : lr);
            return lr * rs;
        };
        auto residual = [&](int lr, int color, int h, int odd) -> float {
            const int own = color ? L.hw : 0, oth = L.hw - own, r = row(lr), t = r + own + h;
            if (m[t]) return 0.0f;
            return mg_residual(b[t], x[t], x[r + oth + h - 1 + odd], x[r + oth + h + odd], x[row(lr - 1) + oth + h],
                               x[row(lr + 1) + oth + h], L.cx, L.cy, L.cd);
        };
        const int Js = L.dist ? start(l + 1, rank) : 0, Je = L.dist ? start(l + 1, rank + 1) : C.GY;
        float* cb = B(l + 1);
        const uint8_t* cm = M(l + 1);
        const int clo = C.dist ? start(l + 1, rank) - C.H : 0;  // level row of the array's first row
        for (int k = tid; k < (Je - Js) * C.GX; k += kClThreads) {
            const int jr = (int)__umulhi((uint32_t)k, C.rcp_gx), a = k - jr * C.GX, J = Js + jr;
            const int t = at(C, J - clo, a, J);
            float v = 0.0f;
            if (!cm[t]) {
                // fine node (2 a, 2 J) is red; the rows beside it start with the other colour
                const int lr = L.dist ? 2 * J - (s - L.H) : 2 * J;
                v = 4.0f * residual(lr, 0, a, 0);
                v += 2.0f * (residual(lr, 1, a - 1, 1) + residual(lr, 1, a, 1) + residual(lr - 1, 1, a, 0) +
                             residual(lr + 1, 1, a, 0));
                v += residual(lr - 1, 0, a - 1, 1) + residual(lr - 1, 0, a, 1) + residual(lr + 1, 0, a - 1, 1) +
                     residual(lr + 1, 0, a, 1);
                v *= 0.0625f;
            }
            cb[t] = v;
        }
        __syncthreads();
        if (L.dist) {
            push_rows<false>(l + 1, cb);
            cluster_barrier();
        }
    }

    // coarse correction from level l + 1, then smoothing, on U rows beyond the band
    __device__ __forceinline__ void up(int l) const {
        const ClLevel& L = I.lev[l];
        const ClLevel& C = I.lev[l + 1];
        const int q = L.hw >> 2, s = start(l, rank);
        const int j0 = L.dist ? s - L.U : 0, rows = L.dist ? start(l, rank + 1) + L.U - j0 : L.GY;
        const int r0 = L.dist ? L.H - L.U : 0;
        const int clo = C.dist ? start(l + 1, rank) - C.H : 0;
        float* x = X(l);
        const float* xc = X(l + 1);
        const float* xh = XH(l);
        const uint8_t* m = M(l);
        for (int k = tid; k < rows * 2 * q; k += kClThreads) {  // quads of both colours
            const int jr2 = (int)__umulhi((uint32_t)k, L.rcp_q), jr = jr2 >> 1, color = jr2 & 1;
            const int h = 4 * (k - jr2 * q), in = (color ? L.hw : 0) + h, t = (jr + r0) * L.rs + in;
            const uint32_t mv = *reinterpret_cast<const uint32_t*>(m + t);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (mv != 0x01010101u) {
                // (the halo's own sweeps on the way down stopped short: its owners' values.
                // Rows that no block owns, outside the grid or a coarse last row past the
                // fine one, are all electrodes: their incoming rows are never written.)
                const float* from = x + t;
                if (L.dist && jr < L.U) from = xh + jr * L.rs + in;
                else if (L.dist && jr >= rows - L.U) from = xh + (jr - (rows - 2 * L.U)) * L.rs + in;
                v = *reinterpret_cast<const float4*>(from);
                int j = j0 + jr;
                const bool odd = (j + color) & 1, oy = j & 1;
                if (!C.dist && I.periodic) j = wrap(l, j);
                const int J = j >> 1, J1 = (!C.dist && J + 1 == C.GY) ? 0 : J + 1;  // wraps only periodic in y
                // coarse values at columns h .. h + 4 of rows J and J1
                float ca[5], cb[5];
#pragma unroll
                for (int n = 0; n < 5; ++n) {
                    ca[n] = (h + n < C.GX) ? xc[at(C, J - clo, h + n, J)] : 0.0f;
                    cb[n] = (oy && h + n < C.GX) ? xc[at(C, J1 - clo, h + n, J1)] : 0.0f;
                }
                float o[4];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    if (!odd && !oy) o[n] = ca[n];
                    else if (odd && !oy) o[n] = 0.5f * (ca[n] + ca[n + 1]);
                    else if (!odd) o[n] = 0.5f * (ca[n] + cb[n]);
                    else o[n] = 0.25f * (ca[n] + ca[n + 1] + cb[n] + cb[n + 1]);
                }
                if (!(mv & 0xffu)) v.x = v.x + o[0];
                if (!(mv & 0xff00u)) v.y = v.y + o[1];
                if (!(mv & 0xff0000u)) v.z = v.z + o[2];
                if (!(mv & 0xff000000u)) v.w = v.w + o[3];
            }
            *reinterpret_cast<float4*>(x + t) = v;
        }
        __syncthreads();
        sweep(l, 1, L.U - 1);
        sweep(l, 0, L.U - 2);
        sweep(l, 1, L.U - 3);
        sweep(l, 0, L.U - 4);
    }

    // the dense product: this block's rows, two a warp at a time, each value
    // stored in every block
    __device__ __forceinline__ void dense() {
        const float* b = B(I.levels);
        float* x = X(I.levels);
        float* bs = reinterpret_cast<float*>(smem + I.oc);
        const int nf = I.nf, n4 = I.nfp / 4, lane = tid & 31;
        const ClLevel& D = I.lev[I.levels];
        auto node = [&](int f) {  // free node f in the level's arrays
            const int k = __ldg(I.freen + f), jn = (int)__umulhi((uint32_t)k, D.rcp_gx);
            return at(D, jn, k - jn * D.GX, jn);
        };
        for (int j = tid; j < I.nfp; j += kClThreads) bs[direct_place(j)] = j < nf ? b[node(j)] : 0.f;
        __syncthreads();
        const float4* b4 = reinterpret_cast<const float4*>(bs);
        const int i0 = rank * nf / kClBlocks, i1 = (rank + 1) * nf / kClBlocks;
        for (int i = i0 + (tid >> 5); i < i1; i += 2 * (kClThreads / 32)) {
            const bool two = i + kClThreads / 32 < i1;
            const float4* r0 = reinterpret_cast<const float4*>(I.inv + (int64_t)i * I.nfp);
            const float4* r1 = two ? r0 + (int64_t)(kClThreads / 32) * n4 : r0;
            float v0 = 0.f, v1 = 0.f;
#pragma unroll 4
            for (int j = lane; j < n4; j += 32) {
                const float4 p = __ldg(r0 + j), q = __ldg(r1 + j), w = b4[j];
                v0 = fmaf(p.w, w.w, fmaf(p.z, w.z, fmaf(p.y, w.y, fmaf(p.x, w.x, v0))));
                v1 = fmaf(q.w, w.w, fmaf(q.z, w.z, fmaf(q.y, w.y, fmaf(q.x, w.x, v1))));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v0 += __shfl_xor_sync(kFull, v0, o);
                v1 += __shfl_xor_sync(kFull, v1, o);
            }
            // lanes 0-15: the first row's value into block `lane`; 16-31: the second's
            const int row = lane < kClBlocks ? i : i + kClThreads / 32;
            if (lane < kClBlocks || two)
                cluster.map_shared_rank(x, lane & (kClBlocks - 1))[node(row)] = lane < kClBlocks ? v0 : v1;
        }
        cluster_barrier();
    }

    // z = V-cycle of b (level 0), valid on the band and what p.A p needs beyond
    __device__ __forceinline__ void vcycle() {
        int l;
        for (l = 0; l < I.levels; ++l) down(l);
        dense();
        for (l = I.levels - 1; l >= 0; --l) up(l);
    }
};

__device__ __forceinline__ void cluster_solve(const ClInst& I, unsigned char* smem) {
    __shared__ ClShared S;
    ClBlock K{I, smem, S, cg::this_cluster(), 0, (int)threadIdx.x, 0};
    K.rank = (int)K.cluster.block_rank();
    const int tid = K.tid, GX = I.GX;
    const ClLevel& L0 = I.lev[0];
    if (tid <= kClBlocks) {
        int s = (int)((int64_t)tid * L0.GY / kClBlocks);
        for (int l = 0; l <= I.levels; ++l) {
            S.start[l][tid] = s;
            s = (s + 1) >> 1;
        }
    }
    __syncthreads();
    // masks of everything this block holds; x = 0 outside the grid and at electrodes for good
    for (int l = 0; l <= I.levels; ++l) {
        const ClLevel& L = I.lev[l];
        const int j0 = L.dist ? K.start(l, K.rank) - L.H : 0;
        const int rows = L.dist ? K.start(l, K.rank + 1) + L.H - j0 : L.GY;
        uint8_t* m = K.M(l);
        float* x = K.X(l);
        float* b = K.B(l);
#pragma unroll 4
        for (int k = tid; k < rows * (L.rs >> 2); k += kClThreads) {
            // a quad of one colour: half row k / (hw / 4), even ones red
            const int r2 = (int)__umulhi((uint32_t)k, L.rcp_q), lr = r2 >> 1, color = r2 & 1;
            const int h = 4 * (k - r2 * (L.hw >> 2)), t = lr * L.rs + (color ? L.hw : 0) + h;
            int j = j0 + lr;
            const int i0 = 2 * h + ((j + color) & 1);
            if (I.periodic) j = K.wrap(l, j);
            const bool in = j >= 0 && j < L.GY;
            const uint8_t* row = L.mask + (in ? (int64_t)j * L.GX : 0);
            uint32_t v = 0;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int i = i0 + 2 * n;
                const uint8_t w = row[i < L.GX ? i : 0];
                v |= (uint32_t)(in && i < L.GX ? (w ? 1 : 0) : 1) << (8 * n);
            }
            *reinterpret_cast<uint32_t*>(m + t) = v;
            *reinterpret_cast<float4*>(x + t) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(b + t) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    for (int k = tid; k < 8 * I.nblocks; k += kClThreads) {  // (groups past the last node)
        reinterpret_cast<double*>(smem + I.opq)[k] = 0.0;
        if (I.levels == 0) reinterpret_cast<double*>(smem + I.orz)[k] = 0.0;
    }
    cluster_barrier();  // every block's arrays are set before another stores into them
    // the nodes this block works on in FP64: the groups of 32 that start in its
    // band, [k0, k1) of the solved ones
    const int nn = (int)I.sn;
    const int s0 = K.start(0, K.rank), band0 = s0 * GX;
    const int g0 = (band0 + 31) >> 5, g1 = (min(K.start(0, K.rank + 1) * GX, nn) + 31) >> 5;
    const int k0 = min(32 * g0, nn), k1 = min(32 * g1, nn);
    double* prz = reinterpret_cast<double*>(smem + I.orz);
    double* ppq = reinterpret_cast<double*>(smem + I.opq);
    // a node's place in the level-0 arrays
    struct Place {
        int t, o, up, dn;  // the node; its row's other colour at its half index; that one and its row's neighbours above and below
        int odd;
    };
    const int lr0 = L0.dist ? L0.H : s0;
    auto place = [&](int k) {
        const int jr = (int)__umulhi((uint32_t)(k - band0), L0.rcp_gx), i = k - band0 - jr * GX, lr = lr0 + jr;
        const int black = (i + s0 + jr) & 1, own = black ? L0.hw : 0, oth = L0.hw - own, h = i >> 1;
        int up = lr + 1, dn = lr - 1;
        if (!L0.dist) {
            up = up == L0.GY ? 0 : up;
            dn = dn < 0 ? L0.GY - 1 : dn;
        }
        return Place{lr * L0.rs + own + h, lr * L0.rs + oth + h, up * L0.rs + oth + h, dn * L0.rs + oth + h, i & 1};
    };
    const uint8_t* m0 = K.M(0);
    float* b0 = K.B(0);
    const float* z0 = K.X(0);
    auto x_at = [&](int k) { return I.mask[k] ? I.dv[k] : (I.zero_start ? 0.0 : I.phi[k]); };
    // overwriteRho, the electrode potentials, r = b - A x, |r|^2 and |b_red|^2
    double rr = 0.0, bb = 0.0;
    for (int k = k0 + tid; k < k1; k += kClThreads) {
        double ri = 0.0;
        if (I.mask[k]) {
            if (I.overwrite) I.rho[k] = -I.dv[k];
            I.phi[k] = I.dv[k];
        } else {
            const double b = I.overwrite ? -I.rho[k] : I.rho[k];
            if (I.overwrite) I.rho[k] = b;
            const int up = row_up(k, nn, GX), dn = row_dn(k, nn, GX);
            ri = b - (I.cd * x_at(k) - I.cx * (x_at(k - 1) + x_at(k + 1)) - I.cy * (x_at(dn) + x_at(up)));
            const double br = b + I.cx * (dirv(I.mask, I.dv, k - 1) + dirv(I.mask, I.dv, k + 1)) +
                              I.cy * (dirv(I.mask, I.dv, dn) + dirv(I.mask, I.dv, up));
            bb += br * br;
            if (I.zero_start) I.phi[k] = 0.0;
        }
        I.r[k] = ri;
        rr += ri * ri;
    }
    if (K.rank == kClBlocks - 1)  // periodic in y: the last node row is not solved
        for (int64_t k = I.sn + tid; k < I.nodes; k += kClThreads) {
            if (I.overwrite) I.rho[k] = I.mask[k] ? -I.dv[k] : -I.rho[k];
            if (I.mask[k]) I.phi[k] = I.dv[k];
            else if (I.zero_start) I.phi[k] = 0.0;
        }
    double t0[2] = {rr, bb};
    K.sums(t0);
    rr = t0[0];
    bb = t0[1];
    const double rr0 = rr;
    double rz_old = 0.0;
    int it = 0, status = 0;
    bool go = bb > 0.0 && rr > I.tol2 * bb && it < I.maxit;
    while (go) {
        // level 0's right-hand side: r of the band and its halo
        {
            const int j0 = L0.dist ? s0 - L0.H : 0, n = (L0.dist ? K.start(0, K.rank + 1) + L0.H - j0 : L0.GY) * GX;
            for (int kk = tid; kk < n; kk += 4 * kClThreads) {
                double rv[4];
                int t[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = kk + u * kClThreads, jr = (int)__umulhi((uint32_t)k, L0.rcp_gx), i = k - jr * GX;
                    int j = j0 + jr;
                    if (I.periodic) j = K.wrap(0, j);
                    const bool in = k < n && j >= 0 && j < L0.GY;
                    t[u] = in ? ClBlock::at(L0, jr, i, j0 + jr) : -1;
                    rv[u] = in ? __ldcg(I.r + j * GX + i) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (t[u] >= 0) b0[t[u]] = (float)rv[u];
            }
            __syncthreads();
        }
        K.vcycle();
        // r.z
        if (I.levels == 0) {  // k_pcg_rz's order
            for (int g = g0 + (tid >> 5); g < g1; g += kClThreads / 32) {
                const int k = 32 * g + (tid & 31);
                double x = 0.0;
                if (k < k1) {
                    const Place P = place(k);
                    x = fma(I.r[k], m0[P.t] ? 0.0 : (double)z0[P.t], 0.0);
                }
                K.share(x, prz, g);
            }
        } else {
            if (L0.dist) {
                const int n = (K.start(0, K.rank + 1) - s0) * GX;
                for (int k = tid; k < n; k += kClThreads) I.z[band0 + k] = z0[place(band0 + k).t];
                cluster_barrier();
            }
            // warp w of a tile: 32 columns, rows w, w + 8, w + 16, w + 24 of it
            static_assert(kTileCore == 32 && kRedThreads == 256, "a warp a row of a tile");
            const int i_in = tid & 31, vw = 8 * I.tiles;
            for (int v = K.rank + kClBlocks * (tid >> 5); v < vw; v += kClBlocks * (kClThreads / 32)) {
                const int tile = v >> 3, ty = tile / I.tx, i = (tile - ty * I.tx) * kTileCore + i_in;
                const int jb = ty * kTileCore + (v & 7);
                double rv[4];
                float zv[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int j = jb + 8 * m, k = j * GX + i;
                    const bool in = i < GX && j < L0.GY && !I.mask[k];
                    rv[m] = in ? __ldcg(I.r + k) : 0.0;
                    zv[m] = !in ? 0.0f : (L0.dist ? __ldcg(I.z + k) : z0[ClBlock::at(L0, j, i, j)]);
                }
                double x = 0.0;
#pragma unroll
                for (int m = 0; m < 4; ++m) x = fma(rv[m], (double)zv[m], x);
                K.share(x, prz, v);
            }
        }
        cluster_barrier();
        const double rz = K.ordered_sum(prz, I.levels == 0 ? I.nblocks : I.tiles);
        const double beta = rz_old == 0.0 ? 0.0 : rz / rz_old;
        // p = z + beta p, q = A z + beta q (the first direction reads neither); p.q
        const int lane = tid & 31;
        for (int gg = g0 + (tid >> 5); gg < g1; gg += 4 * (kClThreads / 32)) {
            double pv[4], qv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = 32 * (gg + u * (kClThreads / 32)) + lane;
                const bool old = k < k1 && beta != 0.0;
                pv[u] = old ? I.p[k] : 0.0;
                qv[u] = old ? I.q[k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int g = gg + u * (kClThreads / 32), k = 32 * g + lane;
                if (g >= g1) break;
                double x = 0.0;
                if (k < k1) {
                    const Place P = place(k);
                    double pi = 0.0, qi = 0.0;
                    if (!m0[P.t]) {
                        const double zi = (double)z0[P.t];
                        const double az = I.cd * zi - I.cx * ((double)z0[P.o - 1 + P.odd] + (double)z0[P.o + P.odd]) -
                                          I.cy * ((double)z0[P.dn] + (double)z0[P.up]);
                        pi = beta == 0.0 ? zi : zi + beta * pv[u];
                        qi = beta == 0.0 ? az : az + beta * qv[u];
                    }
                    I.p[k] = pi;
                    I.q[k] = qi;
                    x = fma(pi, qi, 0.0);
                }
                K.share(x, ppq, g);
            }
        }
        cluster_barrier();
        const double alpha = rz / K.ordered_sum(ppq, I.nblocks);
        // x += alpha p, r -= alpha q; four nodes' loads before their stores
        double acc[1] = {0.0};
        for (int gg = g0 + (tid >> 5); gg < g1; gg += 4 * (kClThreads / 32)) {
            double xv[4], pv[4], qv[4], rw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = 32 * (gg + u * (kClThreads / 32)) + lane;
                const bool in = k < k1;
                xv[u] = in ? I.phi[k] : 0.0;
                rw[u] = in ? I.r[k] : 0.0;
                pv[u] = in ? I.p[k] : 0.0;
                qv[u] = in ? I.q[k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = 32 * (gg + u * (kClThreads / 32)) + lane;
                if (k >= k1 || m0[place(k).t]) continue;  // (r stays 0 at electrodes)
                const double ri = rw[u] - alpha * qv[u];
                I.phi[k] = xv[u] + alpha * pv[u];
                I.r[k] = ri;
                acc[0] += ri * ri;
            }
        }
        K.sums(acc);
        rr = acc[0];
        rz_old = rz;
        ++it;
        const bool finite = isfinite(rr);
        go = finite && rr > I.tol2 * bb;
        if (go && it >= I.maxit) {
            go = false;
            status = 1;
        }
        if (!finite) status = 2;
    }
    // the true residual, then the E field; phi of other blocks is read past L1
    auto phi_at = [&](int64_t k) { return __ldcg(I.phi + k); };
    double acc[1] = {0.0};
#pragma unroll 4
    for (int k = k0 + tid; k < k1; k += kClThreads) {
        const bool free = !m0[place(k).t];  // (an electrode reads only itself)
        const int w = free ? 1 : 0;
        const double ax = I.cd * phi_at(k) - I.cx * (phi_at(k - w) + phi_at(k + w)) -
                          I.cy * (phi_at(free ? row_dn(k, nn, GX) : k) + phi_at(free ? row_up(k, nn, GX) : k));
        const double ri = free ? I.rho[k] - ax : 0.0;
        acc[0] += ri * ri;
    }
    if (I.periodic && K.rank == kClBlocks - 1)
        // overwritePhi: the last row repeats row 0, then takes its own electrodes
        for (int i = tid; i < GX; i += kClThreads)
            I.phi[I.sn + i] = I.mask[I.sn + i] ? I.dv[I.sn + i] : phi_at(i);
    K.sums(acc);
    const double true_rr = acc[0];
    if (K.rank == 0 && tid == 0) {
        I.scal[S_BB] = bb;
        I.scal[S_RR] = rr;
        I.scal[S_TRUE_RR] = true_rr;
        I.scal[S_IT] = (double)it;
        I.scal[S_STATUS] = (double)status;
        I.scal[S_RR0] = rr0;
        // pinned: the host reads them after the stream's end
        I.host_scal[S_BB] = bb;
        I.host_scal[S_RR] = rr;
        I.host_scal[S_TRUE_RR] = true_rr;
        I.host_scal[S_IT] = (double)it;
        I.host_scal[S_STATUS] = (double)status;
        I.host_scal[S_RR0] = rr0;
    }
    const int kend = K.rank == kClBlocks - 1 ? (int)I.nodes : k1;
    const int GYn = (int)(I.nodes / GX);
#pragma unroll 4
    for (int k = k0 + tid; k < kend; k += kClThreads) {
        const int j = k / GX, i = k - j * GX;
        double ex, ey;
        efield_of(phi_at, GX, GYn, I.dx, I.dy, i, j, I.periodic, ex, ey);
        I.fld[k] = make_float4((float)ex, (float)ey, (float)I.bz[k], 0.0f);
    }
    cluster_barrier();  // no block leaves while another may read its shared memory
}

__global__ void __launch_bounds__(kClThreads, 1) k_cluster_solve(const __grid_constant__ ClInst I) {
    extern __shared__ __align__(16) unsigned char smem[];
    cluster_solve(I, smem);
}

// ---- host side ---------------------------------------------------------------

// A launch of one cluster.
void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, size_t smem, cudaStream_t st) {
    cfg.gridDim = dim3(kClBlocks);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClBlocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

constexpr size_t kClMaxSmem = 227 * 1024 - 4096;  // dynamic; the rest is static

// The shared-memory layout of a context's cluster solve, and whether it fits.
bool cluster_layout(pic_ctx* c, ClInst& I, size_t* bytes) {
    PoissonState& ps = c->ps;
    const int kf = ps.fused_first;
    if (!ps.mg_ok || kf > kClMaxLevels || c->nodes > kClMaxNodes || ps.levels[0].GY > kClMaxRows) return false;
    size_t off = 0;
    auto carve = [&](size_t b) {
        const size_t o = off;
        off += (b + 15) & ~(size_t)15;
        return (int)o;
    };
    I.levels = kf;
    // level 0: p and q of groups that start in the band, up to 31 nodes beyond it, read a row further
    int need = 2 + 30 / c->GX;
    bool dist = true;
    for (int l = 0; l <= kf; ++l) {
        const MGLevel& M = ps.levels[l];
        ClLevel& L = I.lev[l];
        const LevelDev D = as_dev(M);
        L.GX = M.GX;
        L.GY = M.GY;
        L.cx = D.cx;
        L.cy = D.cy;
        L.cd = D.cd;
        L.icd = D.icd;
        L.mask = M.mask;
        L.hw = std::max(8, ((M.GX + 1) / 2 + 3) & ~3);  // (at least two quads: rcp_q fits 32 bits)
        L.rs = 2 * L.hw;
        L.rcp_q = (uint32_t)((0x100000000ull + L.hw / 4 - 1) / (L.hw / 4));
        L.rcp_gx = (uint32_t)((0x100000000ull + M.GX - 1) / M.GX);
        dist = dist && l < kf && M.nodes > kClRepNodes;
        L.dist = dist ? 1 : 0;
        L.U = need + 2 * kNu;
        L.H = dist ? std::max(kClDownHalo, L.U) : 0;
        need = (L.U + 2) / 2;
        int rows = M.GY, first[kClBlocks + 1];
        L.near = kClBlocks;
        if (dist) {
            // periodic in y: a halo of more rows than the level has would hold rows
            // twice over, and push_rows stores a row and the two images next to it only
            if (c->periodic && M.GY < L.H) return false;
            rows = 0;
            for (int b = 0; b <= kClBlocks; ++b) {
                first[b] = (int)((int64_t)b * ps.levels[0].GY / kClBlocks);
                for (int k = 0; k < l; ++k) first[b] = (first[b] + 1) >> 1;
                if (b > 0) rows = std::max(rows, first[b] - first[b - 1] + 2 * L.H);
            }
            // d blocks away: the d - 1 bands between two blocks have H rows or more
            for (int d = 1; d < kClBlocks && L.near == kClBlocks; ++d) {
                int least = 1 << 30;
                for (int b = 0; b < kClBlocks; ++b) {
                    const int t = b + d;  // (past the last band: around, periodic in y)
                    if (t <= kClBlocks) least = std::min(least, first[t] - first[b]);
                    else if (c->periodic) least = std::min(least, M.GY - first[b] + first[t - kClBlocks]);
                }
                if (least >= L.H) L.near = d;
            }
        }
        const size_t n = (size_t)rows * L.rs;
        L.oh = dist ? carve((size_t)2 * L.U * L.rs * 4) : 0;
        L.ox = carve((n + 4) * 4);
        L.ob = carve(n * 4);
        L.om = carve(n);
    }
    I.oc = carve((size_t)ps.direct_nfp * 4);
    I.tx = (c->GX + kTileCore - 1) / kTileCore;
    I.tiles = I.tx * ((ps.levels[0].GY + kTileCore - 1) / kTileCore);
    I.nblocks = ps.nblocks;
    I.opq = carve((size_t)8 * I.nblocks * 8);
    I.orz = kf == 0 ? carve((size_t)8 * I.nblocks * 8) : carve((size_t)8 * I.tiles * 8);
    if (I.tiles > kRedThreads || I.nblocks > kRedThreads) return false;  // (a thread a block in the last sum)
    *bytes = off;
    return off <= kClMaxSmem;
}

// Whether the device takes such clusters (asked once a context).
bool cluster_supported() {
    if (cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClMaxSmem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, kClMaxSmem, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_cluster_solve, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n >= 1;
}

// What is the same at every solve of a context (inv: its dense coarse matrix).
void cluster_describe(pic_ctx* c, const float* inv, ClInst& I) {
    PoissonState& ps = c->ps;
    const Grid64 g = fine_grid(c);
    I.GX = c->GX;
    I.GY = c->GY;
    I.periodic = c->periodic ? 1 : 0;
    I.nodes = c->nodes;
    I.sn = c->solve_nodes;
    I.cx = g.cx;
    I.cy = g.cy;
    I.cd = g.cd;
    I.dx = c->dx;
    I.dy = c->dy;
    I.mask = c->mask;
    I.dv = c->dir_val;
    I.rho = c->rho;
    I.phi = c->phi;
    I.r = ps.r;
    I.p = ps.p[0];
    I.q = ps.q;
    I.z = ps.levels[0].x;
    I.bz = c->bz;
    I.fld = c->fld;
    I.inv = inv;
    I.freen = ps.direct_free;
    I.nf = ps.direct_nf;
    I.nfp = ps.direct_nfp;
    I.scal = ps.scal;
    I.tol2 = ps.tol * ps.tol;
    I.maxit = ps.maxit;
    I.zero_start = (ps.warm == PIC_WARM_ZERO || !ps.have_prev) ? 1 : 0;
    I.overwrite = 1;
}
