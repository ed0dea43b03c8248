// particles.cu -- cell binning, CIC deposit and gather + Boris push for
// sm_100a.
//
// Reference operators replaced (SYCL-PIC-poissonsolver):
//   * hashmap binning: InsertKernel (src/particles.cpp:227-237), map
//     delete/insert inside MoverKernel (src/mover.cpp:353-364), cleanup_map
//     (src/utils.cpp:30-44) and compact_particles (src/utils.cpp:249-372);
//   * interpolate() (src/interpolation.cpp:13-171);
//   * deterministic_mover() + MoverKernel (src/mover.cpp:103-176, 304-366).
//
// Layout: the particles of a species live in a double buffer of 20-byte
// slots, float4 {fx, fy, vx, vy} (in-cell offsets in [0,1), velocities in
// m/s) plus float vz.  Cell c (c = gy*nx + gx) owns the slots base[c] ..
// base[c+1] of both buffers with slack: its particles are a front run (the
// ones that stayed in the cell at the last push) and a back run (the ones
// that moved in), with a free gap between them.
//
// One push of a species is ONE pass over its particles (k_cells<kPush>).  A
// warp works on a few neighbouring cells at a time, 4, 8 or 16 lanes a cell
// (32 where a cell is far fuller than its neighbours); it gathers E and Bz,
// pushes, and
//   * writes a particle that stays in its cell to the front of the cell's
//     slots in the other buffer, at its rank among the cell's stayers
//     (ballot + popc: no atomics), and adds its deposit to per-lane integer
//     sums, reduced once per cell;
//   * queues a particle that leaves; every 32 of them are placed with all
//     lanes busy: each reserves a slot at the back of its new cell with one
//     atomic on the cell's back count, capped at the cell's capacity minus
//     its current count (the most stayers it can have), so front and back
//     runs never meet.
// The deposit of the particles that changed cell is a second, small pass over
// the back runs (k_cells<kArrivals>): per-cell sums again, where depositing
// each mover on its own took eight 64-bit REDs.  A mover whose target is full
// goes to a side list; a small kernel (k_fixup) then deposits it and places
// it in the free space of its target cell, or keeps it on the list (still
// part of the state: it is pushed and deposited from there at the next
// step).  When the list grows, the host rebuilds the layout from the
// per-cell counts (k_relayout_*).  Per particle-step the HBM traffic is 20 B
// read + 20 B written.
//
// Measured on a B200, push + arrivals, electrons / Ar+: the 1024^2 workload
// (1.15e8 particles each) 1.26 / 0.87 ms (with a warp a cell, 32-lane chunks
// and the movers deposited one by one: 1.83 / 1.17 ms); 512^2 at 64 a cell
// 0.23 / 0.14 ms (0.28 / 0.18); 64 grids of 128^2 .. 384^2 at 32 a cell 4.2 ms
// both (8.2 ms).  The Ar+ pass runs at 5.2 TB/s of reads and writes, 0.8 of a
// plain copy; leaving out instructions (the FP32 push, the energy sums)
// changes it by a few percent, leaving out its stores by 40 %: memory bound.
// The electrons pay 0.3 ms for placing their 18 % movers (an atomic with its
// answer, two scattered stores each) and 0.1 ms for the arrivals' pass.
//
// Determinism: the charge and energy deposits are sums of integers, so they
// do not depend on the order in which particles are processed or placed;
// the set of particles in each cell is deterministic, their order within
// the back run is not.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "pic_internal.h"

namespace picb200 {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = kWarps * 32;
constexpr int kScanTile = 2048;               // cells per scan block
constexpr uint32_t kAxisOne = 1u << kAxisBits;
constexpr float kAxisScale = (float)(1u << kAxisBits);
constexpr float kOneBelow = 0x1.fffffep-1f;   // largest float < 1
constexpr float kEnergyScale = 4194304.0f;    // eV -> 2^-22 eV units
constexpr float kFloorMagic = 12582912.0f;    // 1.5 * 2^23
constexpr uint32_t kFloorMagicBits = 0x4B400000u;
constexpr int kFixupBlocks = 148;

enum Mode { kPush = 0, kDeposit = 1, kArrivals = 2 };

// list_counts slots
enum { kOvf = 0, kLoose0 = 1, kLoose1 = 2, kTicket = 3 };

struct ListDev {
    float4* a;
    float* vz;
    uint32_t* cell;
    uint32_t* count;
    uint32_t cap;
};

__host__ __forceinline__ ListDev list_dev(const LooseList& L) {
    return ListDev{L.a, L.vz, L.cell, L.count, L.cap};
}

struct KArgs {
    int nx, ny, GX;
    int64_t ncells;
    SpeciesConsts k;
    const float4* __restrict__ fld;
    // (not __restrict__, like back_src: the arrivals' pass reads what the kernel
    // before it wrote, and may be launched before that one's end; its loads must
    // stay behind the wait)
    const float4* src_a;
    const float* src_vz;
    float4* __restrict__ dst_a;
    float* __restrict__ dst_vz;
    const uint32_t* __restrict__ base;
    const uint32_t* __restrict__ front_src;
    const uint32_t* back_src;
    uint32_t* front_dst;
    uint32_t* back_dst;
    ListDev ovf;
    unsigned long long* acc_q;
    unsigned long long* acc_e;
    unsigned long long* counters;  // [0] left exits, [1] cell limit, [2] lost particles
};

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Asynchronous global -> shared copies (cp.async) to a shared-space address.
// Only the wait orders them against the shared-memory reads of the data.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Result of one gather + Boris + position update.
struct Pushed {
    float fx, fy, vx, vy;
    float px, py;  // new position in units of the old cell (its corner at 0)
    int sx, sy;    // cell step: 0, 0 exactly when the particle keeps its cell
    // set by resolve_move
    int gx, gy;
    bool alive;  // inside the walls
    bool left;   // absorbed, and through x < 0
};

// Re-cell of the position (px, py) in units of the old cell: the integer
// part moves the cell, the remainder is the new offset.  floor without the
// conversion unit: for |p| < 2^22, p + 1.5*2^23 rounded down is floor(p) +
// 1.5*2^23 exactly, an integer held in the low mantissa bits; subtracting
// 1.5*2^23 again is exact.  The step's bits are 0 exactly when floor(p) == 0:
// for NaN or |p| >= 2^22 the sum is not 1.5*2^23, so those never read as
// staying.
__device__ __forceinline__ void recell(Pushed& o) {
    const float px = o.px, py = o.py;
    const float tx = __fadd_rd(px, kFloorMagic), ty = __fadd_rd(py, kFloorMagic);
    const float fsx = __fsub_rn(tx, kFloorMagic), fsy = __fsub_rn(ty, kFloorMagic);
    o.fx = fminf(__fsub_rn(px, fsx), kOneBelow);
    o.fy = fminf(__fsub_rn(py, fsy), kOneBelow);
    o.sx = (int)(__float_as_uint(tx) - kFloorMagicBits);
    o.sy = (int)(__float_as_uint(ty) - kFloorMagicBits);
}

// Bilinear gather of E (and Bz) from the cell's four nodes plus the Boris
// push of deterministic_mover (src/mover.cpp:123-174) in FP32.  Weights:
// (1-fx)(1-fy), fx(1-fy), (1-fx)fy, fx*fy == the reference's unnormalised
// weights divided by dx*dy.  Every operation is an explicit _rn intrinsic:
// the result does not depend on how the compiler contracts the code.
//
// push_move does the arithmetic of every particle; resolve_move the cell
// bookkeeping that only particles leaving their cell need.
// A node's field: {Ex, Ey}, with Bz (and padding) unless it is uniform.
template <bool BZU>
struct __align__(16) NodeField {
    float x, y, z, w;
    __device__ __forceinline__ static NodeField from(float4 f) { return NodeField{f.x, f.y, f.z, f.w}; }
};
template <>
struct __align__(8) NodeField<true> {
    float x, y;
    static constexpr float z = 0.f;  // not read
    __device__ __forceinline__ static NodeField from(float4 f) { return NodeField{f.x, f.y}; }
};

template <bool BZU>
__device__ __forceinline__ Pushed push_move(float4 a, NodeField<BZU> n00, NodeField<BZU> n10, NodeField<BZU> n01,
                                            NodeField<BZU> n11, const SpeciesConsts& k) {
    const float fx = a.x, fy = a.y;
    const float ofx = __fsub_rn(1.0f, fx), ofy = __fsub_rn(1.0f, fy);
    const float w00 = __fmul_rn(ofx, ofy), w10 = __fmul_rn(fx, ofy);
    const float w01 = __fmul_rn(ofx, fy), w11 = __fmul_rn(fx, fy);
    const float ex = __fmaf_rn(w11, n11.x, __fmaf_rn(w01, n01.x, __fmaf_rn(w10, n10.x, __fmul_rn(w00, n00.x))));
    const float ey = __fmaf_rn(w11, n11.y, __fmaf_rn(w01, n01.y, __fmaf_rn(w10, n10.y, __fmul_rn(w00, n00.y))));
    // Boris rotation about z (src/mover.cpp:151-162): t = h Bz, s = 2t/(1+t^2)
    float t, s;
    if (BZU) {
        t = k.bt;
        s = k.bs;
    } else {
        const float bz = __fmaf_rn(w11, n11.z, __fmaf_rn(w01, n01.z, __fmaf_rn(w10, n10.z, __fmul_rn(w00, n00.z))));
        t = __fmul_rn(k.h, bz);
        // approximate reciprocal: ~1 ulp, far below the FP32 state's error
        s = __fdividef(__fmul_rn(2.0f, t), __fmaf_rn(t, t, 1.0f));
    }
    const float ax = __fmul_rn(k.h, ex), ay = __fmul_rn(k.h, ey);
    const float vxm = __fadd_rn(a.z, ax), vym = __fadd_rn(a.w, ay);
    const float vxp = __fmaf_rn(vym, t, vxm);
    const float vyp = __fmaf_rn(-vxm, t, vym);
    Pushed o;
    o.vx = __fadd_rn(__fmaf_rn(vyp, s, vxm), ax);
    o.vy = __fadd_rn(__fmaf_rn(-vxp, s, vym), ay);
    // Position update in cell units (src/mover.cpp:164-165)
    o.px = __fmaf_rn(o.vx, k.dtdx, fx);
    o.py = __fmaf_rn(o.vy, k.dtdy, fy);
    return o;
}

// 0 <= p < 1, the particle keeps its cell in this axis: as unsigned integers
// the bits of the floats in [0, 1) are below those of 1 and every other
// float's (negative ones and NaN included) are not.  (-0 reads as leaving;
// it is then placed into its own cell again.)  The new offset is p itself.
__device__ __forceinline__ bool keeps_cell(float p) { return __float_as_uint(p) < 0x3f800000u; }

// Cell bookkeeping of a pushed particle that was in cell (gx, gy).
__device__ __forceinline__ void resolve_move(Pushed& o, const SpeciesConsts& k, int gx, int gy,
                                             int nx, int ny) {
    const float px = o.px, py = o.py;
    // beyond 2^20 cells (or NaN) a particle is lost whatever the grid
    const bool ok = fabsf(px) < 1048576.0f && fabsf(py) < 1048576.0f;
    const int sx = ok ? o.sx : 0;
    const int sy = ok ? o.sy : 0;
    o.gx = gx + sx;
    o.gy = gy + sy;
    // periodic in y (modulo(y, H), src/mover.cpp:317-320): the cell row
    // wraps, the offset stays
    if (k.pery && (unsigned)o.gy >= (unsigned)ny) {
        o.gy %= ny;
        if (o.gy < 0) o.gy += ny;
    }
    // absorbing walls (src/mover.cpp:325): outside [0,W) x [0,H)
    o.alive = ok && (unsigned)o.gx < (unsigned)nx && (unsigned)o.gy < (unsigned)ny;
    o.left = ok ? (o.gx < 0) : (px < 0.0f);
}

__device__ __forceinline__ Pushed push_one(float4 a, float4 n00, float4 n10, float4 n01,
                                           float4 n11, const SpeciesConsts& k, int gx, int gy,
                                           int nx, int ny) {
    using U = NodeField<true>;
    using V = NodeField<false>;
    Pushed o = k.bzu ? push_move<true>(a, U::from(n00), U::from(n10), U::from(n01), U::from(n11), k)
                     : push_move<false>(a, V::from(n00), V::from(n10), V::from(n01), V::from(n11), k);
    recell(o);
    resolve_move(o, k, gx, gy, nx, ny);
    return o;
}

// round(f * 2^20) for f in [0, 1): the scaling is exact, so one FMA with
// 1.5*2^23 rounds to nearest-even in the mantissa (no conversion unit).
__device__ __forceinline__ uint32_t axis_fixed(float f) {
    return __float_as_uint(__fmaf_rn(f, kAxisScale, kFloorMagic)) - kFloorMagicBits;
}

// Kinetic energy (0.5 v^2/|q/m|, src/interpolation.cpp:88-89) in units of
// 2^-22 eV, clamped below 1024 eV; escale = escale * 2^22 (a power
// of two: the product rounds as the energy in eV would).
__device__ __forceinline__ float energy_units(float vx, float vy, float vz, float escale) {
    const float v2 = __fmaf_rn(vz, vz, __fmaf_rn(vy, vy, __fmul_rn(vx, vx)));
    return fminf(__fmul_rn(v2, escale), kEnergyClampEv * kEnergyScale);
}

// Energy-weighted corner weights of one particle, rounded to integers of
// 2^-22 eV (each below 2^32): e00 <-> (gx,gy), e10 <-> (gx+1,gy),
// e01 <-> (gx,gy+1), e11 <-> (gx+1,gy+1).
struct EWeights {
    uint32_t e00, e10, e01, e11;
};

__device__ __forceinline__ EWeights energy_weights(float fx, float fy, float es) {
    const float a = __fmul_rn(es, __fsub_rn(1.0f, fx)), b = __fmul_rn(es, fx);
    const float ofy = __fsub_rn(1.0f, fy);
    EWeights w;
    w.e00 = __float2uint_rn(__fmul_rn(a, ofy));
    w.e10 = __float2uint_rn(__fmul_rn(b, ofy));
    w.e01 = __float2uint_rn(__fmul_rn(a, fy));
    w.e11 = __float2uint_rn(__fmul_rn(b, fy));
    return w;
}

// Global 64-bit integer reductions (fire-and-forget RED) into the node
// accumulators.
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
    atomicAdd(p, v);
}

// Deposit of one particle straight into the node accumulators: its four
// charge corner weights are the exact 40-bit products of the 20-bit axis
// weights (they sum to exactly 2^40).
template <bool ENERGY>
__device__ __forceinline__ void deposit_one(unsigned long long* acc_q, unsigned long long* acc_e,
                                            int GX, uint32_t n, float fx, float fy, float es) {
    const uint32_t ax = axis_fixed(fx), ay = axis_fixed(fy);
    const uint32_t bx = kAxisOne - ax, by = kAxisOne - ay;
    red_add(acc_q + n, (unsigned long long)bx * by);
    red_add(acc_q + n + 1, (unsigned long long)ax * by);
    red_add(acc_q + n + GX, (unsigned long long)bx * ay);
    red_add(acc_q + n + GX + 1, (unsigned long long)ax * ay);
    if (ENERGY) {
        const EWeights e = energy_weights(fx, fy, es);
        red_add(acc_e + n, e.e00);
        red_add(acc_e + n + 1, e.e10);
        red_add(acc_e + n + GX, e.e01);
        red_add(acc_e + n + GX + 1, e.e11);
    }
}

// Per-lane sums of the particles that stay in the lane's cell.  Charge as
// moments of the 20-bit axis weights -- sum ax, sum ay, sum ax*ay, and the
// cell's stayer count N (kept by the caller) -- from which the four corner
// sums follow exactly:
//   Q00 = N 2^40 - (SX + SY) 2^20 + SXY,  Q10 = SX 2^20 - SXY,
//   Q01 = SY 2^20 - SXY,                   Q11 = SXY.
// A lane adds at most kFlushChunks = 2^11 particles between flushes: SX, SY
// < 2^32, SXY < 2^52.  The energy mesh (a diagnostic) sums its corner weights
// as integers of 2^-22 eV (each below 2^32, rounded once per particle).
// Every sum is one of integers: no result depends on the order.
constexpr uint32_t kFlushChunks = 1u << 11;

struct StayAcc {
    uint32_t sx, sy;
    unsigned long long sxy;
    unsigned long long e[4];
};

__device__ __forceinline__ void acc_zero(StayAcc& s) {
    s.sx = s.sy = 0u;
    s.sxy = 0ull;
#pragma unroll
    for (int k = 0; k < 4; ++k) s.e[k] = 0ull;
}

// es: the particle's energy in units of 2^-22 eV
template <bool ENERGY>
__device__ __forceinline__ void acc_add(StayAcc& s, float fx, float fy, float es) {
    const uint32_t ax = axis_fixed(fx), ay = axis_fixed(fy);
    s.sx += ax;
    s.sy += ay;
    s.sxy += (unsigned long long)ax * ay;
    if (ENERGY) {
        const EWeights w = energy_weights(fx, fy, es);
        s.e[0] += w.e00;
        s.e[1] += w.e10;
        s.e[2] += w.e01;
        s.e[3] += w.e11;
    }
}

// Sums v[0..NV) over the G lanes of a group (gl: the lane's index in it) by
// recursive halving: a step exchanges half of the values still held, so the
// whole reduction is NV - 1 exchanges (not NV log2 G) and ends with lane gl
// holding the NV / G (at least one) totals from index `idx` on.  With G > NV
// the G / NV lanes of equal idx hold the same total.
template <int G, int NV>
__device__ __forceinline__ int group_reduce_scatter(unsigned long long (&v)[NV], int gl) {
    int idx = 0, cnt = NV;
#pragma unroll
    for (int d = G / 2; d >= 1; d >>= 1) {
        if (cnt > 1) {
            cnt >>= 1;
            const bool hi = (gl & d) != 0;
#pragma unroll
            for (int k = 0; k < NV / 2; ++k)
                if (k < cnt) {
                    const unsigned long long send = hi ? v[k] : v[k + cnt];
                    const unsigned long long keep = hi ? v[k + cnt] : v[k];
                    v[k] = keep + __shfl_xor_sync(kFull, send, d);
                }
            idx += hi ? cnt : 0;
        } else {
            v[0] += __shfl_xor_sync(kFull, v[0], d);
        }
    }
    return idx;
}

// Reduces the stayer sums over each cell's group of G lanes and adds them to
// the cell's four nodes (n0: its lower left node), one RED per lane for
// G = 8: lane gl of the group holds quantity gl (charge corners 00, 10, 01,
// 11, then the energy's).  N: the cell's stayer count.
template <int G, bool ENERGY>
__device__ __forceinline__ void acc_flush(StayAcc& s, const KArgs& A, uint32_t n0, int gl, uint32_t N) {
    constexpr int NV = ENERGY ? 8 : 4;
    unsigned long long v[NV];
    const unsigned long long sx = (unsigned long long)s.sx << kAxisBits, sy = (unsigned long long)s.sy << kAxisBits;
    v[3] = s.sxy;
    v[2] = sy - s.sxy;
    v[1] = sx - s.sxy;
    v[0] = s.sxy - sx - sy;
    if (ENERGY) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[NV - 4 + k] = s.e[k];
    }
    const int idx0 = group_reduce_scatter<G, NV>(v, gl);
    constexpr int kPer = NV > G ? NV / G : 1, kSame = G > NV ? G / NV : 1;
    if (N && (gl & (kSame - 1)) == 0) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int idx = idx0 + k;
            unsigned long long* acc = (ENERGY && idx >= 4) ? A.acc_e : A.acc_q;
            const uint32_t node = n0 + (idx & 1) + ((idx & 2) ? (uint32_t)A.GX : 0u);
            red_add(acc + node, idx == 0 ? v[k] + ((unsigned long long)N << (2 * kAxisBits)) : v[k]);
        }
    }
    acc_zero(s);
}

__device__ __forceinline__ void store_slot(float4* dst_a, float* dst_vz, uint32_t slot,
                                           const Pushed& p, float vz) {
    dst_a[slot] = make_float4(p.fx, p.fy, p.vx, p.vy);
    dst_vz[slot] = vz;
}

// Appends the lanes with `on` set to a side list (one atomic per warp).
__device__ __forceinline__ void list_append(const ListDev& L, bool on, uint32_t cell,
                                            const Pushed& p, float vz, unsigned lt, int lane,
                                            unsigned long long* lost) {
    const unsigned m = __ballot_sync(kFull, on);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t b = 0;
    if (lane == leader) b = atomicAdd(L.count, (uint32_t)__popc(m));
    b = __shfl_sync(kFull, b, leader);
    if (on) {
        const uint32_t s = b + __popc(m & lt);
        if (s < L.cap) {
            L.a[s] = make_float4(p.fx, p.fy, p.vx, p.vy);
            L.vz[s] = vz;
            L.cell[s] = cell;
        } else {
            atomicOr(lost, 1ull);
        }
    }
}

// One kernel body for three uses:
//   kPush    -- push, place every particle in the other buffer, deposit the
//               new positions of those that kept their cell;
//   kDeposit -- deposit the current positions (no push, nothing moves);
//   kArrivals -- deposit the back runs alone: what a push placed there.
// A block owns a tile of TX x TY cells (powers of two, at most kTileCells).
// Its prologue stages the tile's per-cell slot metadata and the node fields
// in shared memory; then each warp works on sets of 32 / G neighbouring cells
// of a row at a time, G lanes a cell: a chunk is the next 2 G particles of
// each of the set's cells, two a lane.  The chunks travel through a per-warp
// ring of kDepth chunk buffers in shared memory filled by cp.async, kDepth - 1
// chunks ahead of the one being worked on -- across sets, so the load
// pipeline never drains.
constexpr int kTileCells = 256;  // (a queued particle's old cell is 8 bits)
constexpr int kTileNodes = 2 * (kTileCells + 1);  // of the widest tile, 256 x 1 (the most nodes)

// Blocks of 4 warps, 6 an SM (80 registers a thread): with 8 warps and a ring
// of 2, and with 8 blocks of 4 warps at 64 registers, the push of the 1024^2
// workload took 3 to 8 % longer.
constexpr int kCellBlocksPerSM = 6;
constexpr int kDepth = 3;  // chunks in the ring

struct Tile {
    int ltx, lty;  // log2 of the cells in x and y
};

struct CellMeta {
    uint32_t b0, b1, nf, nb;
};

// Particles that left their cell wait in a per-warp queue in shared memory
// and are placed 32 at a time (all lanes busy): cell bookkeeping, a slot
// reserved by one atomic each, store.
constexpr int kQueue = 96;  // 31 waiting and a chunk of 64

struct MoverQueue {
    float4 a[kQueue];  // position in units of the old cell (its corner at 0), vx, vy
    float vz[kQueue];
    uint8_t cell[kQueue];  // old cell (index in the tile)
};

// Places `count` (<= 32) queued particles from entry `first` on, of the block
// with tile origin (tgx0, tgy0), one a lane: each reserves a slot at the back
// of its new cell with one atomic, capped at the cell's capacity minus its
// current count (the most stayers it can have).  Their deposit is left to
// the pass over the arrivals (kArrivals).  Returns 1 in lanes whose particle
// left through x < 0.
__device__ __forceinline__ uint32_t place_movers(const KArgs& A, MoverQueue& q,
                                                 const CellMeta* __restrict__ s_meta, Tile T, int tgx0,
                                                 int tgy0, int first, int count, int lane, unsigned lt) {
    __syncwarp();
    Pushed p{};
    float vz = 0.f;
    uint32_t left = 0, t = 0;
    bool spill = false;
    if (lane < count) {
        const float4 a = q.a[first + lane];
        const int lc = q.cell[first + lane];
        vz = q.vz[first + lane];
        p.px = a.x;
        p.py = a.y;
        p.vx = a.z;
        p.vy = a.w;
        recell(p);
        resolve_move(p, A.k, tgx0 + (lc & ((1 << T.ltx) - 1)), tgy0 + (lc >> T.ltx), A.nx, A.ny);
        if (p.alive) {
            t = (uint32_t)p.gy * (uint32_t)A.nx + (uint32_t)p.gx;
            const uint32_t k = atomicAdd(A.back_dst + t, 1u);
            // the target's slots and source counts: from the tile's shared
            // metadata when it lies in this block's tile, else from global
            // memory
            const int lx = p.gx - tgx0, ly = p.gy - tgy0;
            CellMeta m;
            if (((unsigned)lx >> T.ltx) == 0u && ((unsigned)ly >> T.lty) == 0u) {
                m = s_meta[(ly << T.ltx) + lx];
            } else {
                m.b0 = A.base[t];
                m.b1 = A.base[t + 1];
                m.nf = A.front_src[t];
                m.nb = A.back_src[t];
            }
            if (k < (m.b1 - m.b0) - (m.nf + m.nb)) {
                store_slot(A.dst_a, A.dst_vz, m.b1 - 1u - k, p, vz);
            } else {  // full: give the slot number back
                atomicSub(A.back_dst + t, 1u);
                spill = true;
            }
        } else {
            left = p.left ? 1u : 0u;
        }
    }
    list_append(A.ovf, spill, t, p, vz, lt, lane, A.counters + 2);
    __syncwarp();
    return left;
}

template <int MODE, bool BZU>
struct CellShared {
    CellMeta meta[kTileCells];
    NodeField<BZU> fld[MODE == kPush ? kTileNodes : 1];
    MoverQueue q[MODE == kPush ? kWarps : 1];
    float4 ring_a[kWarps][kDepth][2][32];
    float ring_vz[kWarps][kDepth][2][32];
};

// Whether the warps of a block would be done clearly sooner with all 32 lanes on
// a cell than with G, by the particle counts n of 32 neighbouring cells, one a
// lane: G lanes a set of 32 / G cells take as many chunks as the set's fullest
// cell needs, so a cell far fuller than its neighbours (a beam spot, a sheath) is
// walked 2 G particles at a time by one warp while the others are done.
// Measured, us a push of Ar+, 256^2 cells, 2 a cell and one of 2,000 / 8,000 /
// 40,000: 4 lanes throughout 119 / 412 / 1,974, with this 39 / 73 / 255; 512^2, 4 a
// cell and a blob of 20,000 a cell at its centre, sigma 3 cells: 990 / 205.  Where
// no tile is crowded the look at the counts costs 0.4 % (1024^2 workload, both
// species 2,138 / 2,148 us) to 1 % (512^2, 369 / 373).
template <int G>
__device__ __forceinline__ bool crowded(uint32_t n) {
    // (evenly filled cells, which is nearly all: nothing more to do)
    if (__reduce_max_sync(kFull, n) <= (__reduce_add_sync(kFull, n) >> 5) + 64u) return false;
    constexpr int kSetCells = 32 / G;
    uint32_t narrow = n;  // the fullest of the lane's set
#pragma unroll
    for (int d = 1; d < kSetCells; d <<= 1) narrow = max(narrow, __shfl_xor_sync(kFull, narrow, d));
    narrow = (narrow + 2 * G - 1) / (2 * G);
    // the sets, and the cells, that go to one warp
#pragma unroll
    for (int d = kWarps * kSetCells; d < 32; d <<= 1) narrow += __shfl_xor_sync(kFull, narrow, d);
    uint32_t wide = (n + 63) / 64;
#pragma unroll
    for (int d = kWarps; d < 32; d <<= 1) wide += __shfl_xor_sync(kFull, wide, d);
    return 4 * __reduce_max_sync(kFull, wide) <= 3 * __reduce_max_sync(kFull, narrow);
}

// The tile's cells, G lanes a cell (its metadata and fields are in S).
template <int MODE, bool ENERGY, bool BZU, int G>
__device__ __forceinline__ void cells_run(const KArgs& A, Tile T, int tgx0, int tgy0, CellShared<MODE, BZU>& S) {
    constexpr int kSetCells = 32 / G;  // cells a warp works on at a time (neighbours in a row)
    using Field = NodeField<BZU>;
    const CellMeta* s_meta = S.meta;
    const Field* s_fld = S.fld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gl = lane & (G - 1), grp = lane / G;  // lane of the group, group of the warp
    const int sets = (1 << (T.ltx + T.lty)) / kSetCells, rowlen = (1 << T.ltx) + 1;
    const unsigned lt = lanemask_lt();
    const unsigned gmask = (G == 32 ? kFull : ((1u << (G & 31)) - 1u)) << (grp * G);
    uint32_t left_exits = 0;  // per lane
    // The set being loaded: the group's cell as the source index of its j-th
    // particle (the front run for j < pnf, then the back run, index pback +
    // j), its particle count pn, and the fullest cell's count pmax.
    int pset = warp;
    uint32_t pfront = 0, pback = 0, pnf = 0, pn = 0, pmax = 0, pj = 0;
    auto p_enter = [&]() {  // the next set with particles, from pset on
        for (; pset < sets; pset += kWarps) {
            const CellMeta m = s_meta[pset * kSetCells + grp];
            pn = m.nf + m.nb;
            pmax = __reduce_max_sync(kFull, pn);
            if (pmax) {
                pfront = m.b0;
                pnf = m.nf;
                pback = m.b1 - pn;
                break;
            }
        }
        pj = gl;
    };
    const uint32_t ring_a0 = smem_u32(&S.ring_a[warp][0][0][lane]);
    const uint32_t ring_vz0 = smem_u32(&S.ring_vz[warp][0][0][lane]);
    // issues the copies of the next chunk into ring slot r; every call
    // commits one (possibly empty) copy group
    auto fetch = [&](uint32_t r) {
        if (pset < sets) {
#pragma unroll
            for (uint32_t u = 0; u < 2; ++u) {
                const uint32_t j = pj + u * G;
                if (j < pn) {
                    const uint32_t i = (j < pnf ? pfront : pback) + j;
                    cp_async16(ring_a0 + r * 1024u + u * 512u, A.src_a + i);
                    cp_async4(ring_vz0 + r * 256u + u * 128u, A.src_vz + i);
                }
            }
            pj += 2 * G;
            if (pj - gl >= pmax) {
                pset += kWarps;
                p_enter();
            }
        }
        cp_async_commit();
    };
    p_enter();

    MoverQueue& q = S.q[MODE == kPush ? warp : 0];
    int queued = 0;  // warp-uniform
    // the set being worked on: the group's cell (index lc in the tile), its
    // particle count n, its corner in the shared fields, its lower left node
    // and the next free front slot; nmax: the fullest cell's count
    int set = warp, lc = 0;
    uint32_t n = 0, nmax = 0, front = 0, front0 = 0, node = 0, cell = 0;
    bool inside = false;
    const Field* f = s_fld;
    auto enter = [&]() {  // the next set with particles; empty ones only get their front counts written
        for (; set < sets; set += kWarps) {
            lc = set * kSetCells + grp;
            const CellMeta m = s_meta[lc];
            n = m.nf + m.nb;
            nmax = __reduce_max_sync(kFull, n);
            const int lx = lc & ((1 << T.ltx) - 1), ly = lc >> T.ltx;
            const int gx = tgx0 + lx, gy = tgy0 + ly;
            inside = gx < A.nx && gy < A.ny;
            cell = (uint32_t)gy * (uint32_t)A.nx + (uint32_t)gx;
            node = (uint32_t)gy * (uint32_t)A.GX + (uint32_t)gx;
            front = front0 = m.b0;
            f = s_fld + ly * rowlen + lx;
            if (nmax) break;
            if (MODE == kPush && gl == 0 && inside) A.front_dst[cell] = 0u;
        }
    };
    enter();
    if (set < sets) {
        StayAcc acc;
        acc_zero(acc);
        uint32_t r = 0;
#pragma unroll
        for (uint32_t k = 0; k < kDepth - 1u; ++k) fetch(k);
        uint32_t j0 = 0, jstop = min(nmax, kFlushChunks * G), counted = 0;
        for (;;) {
            fetch(r == 0 ? kDepth - 1u : r - 1u);  // refill the slot freed by the previous chunk
            cp_async_wait<kDepth - 1>();
            Pushed p[2];
            float vz[2];
            bool stay[2], other[2];
            Field f00, f10, f01, f11;
            if (MODE == kPush) {
                f00 = f[0];
                f10 = f[1];
                f01 = f[rowlen];
                f11 = f[rowlen + 1];
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float4 a = S.ring_a[warp][r][u][lane];
                vz[u] = S.ring_vz[warp][r][u][lane];
                const bool valid = j0 + gl + u * G < n;
                if (MODE != kPush) {
                    p[u].fx = a.x; p[u].fy = a.y; p[u].vx = a.z; p[u].vy = a.w;
                    stay[u] = valid;
                } else {
                    p[u] = push_move<BZU>(a, f00, f10, f01, f11, A.k);
                    p[u].fx = p[u].px;
                    p[u].fy = p[u].py;
                    stay[u] = valid && keeps_cell(p[u].px) && keeps_cell(p[u].py);
                    other[u] = valid && !stay[u];
                }
            }
            r = r == kDepth - 1u ? 0u : r + 1u;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                unsigned sm = 0;
                if (MODE == kPush) sm = __ballot_sync(kFull, stay[u]) & gmask;
                if (stay[u]) {
                    const float es = ENERGY ? energy_units(p[u].vx, p[u].vy, vz[u], A.k.escale) : 0.f;
                    acc_add<ENERGY>(acc, p[u].fx, p[u].fy, es);
                    if (MODE == kPush) store_slot(A.dst_a, A.dst_vz, front + __popc(sm & lt), p[u], vz[u]);
                }
                if (MODE == kPush) front += __popc(sm);
            }
            if (MODE == kPush && __any_sync(kFull, other[0] || other[1])) {
                // the rest (moving or absorbed) is queued
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const unsigned om = __ballot_sync(kFull, other[u]);
                    if (other[u]) {
                        const int e = queued + __popc(om & lt);
                        q.a[e] = make_float4(p[u].px, p[u].py, p[u].vx, p[u].vy);
                        q.vz[e] = vz[u];
                        q.cell[e] = (uint8_t)lc;
                    }
                    queued += __popc(om);
                }
                while (queued >= 32) {
                    queued -= 32;  // the last 32 of the queue
                    left_exits += place_movers(A, q, s_meta, T, tgx0, tgy0, queued, 32, lane, lt);
                }
            }
            j0 += 2 * G;
            if (j0 >= jstop) {  // the set is done (or the per-lane sums are full)
                const uint32_t stayers = MODE == kPush ? front - front0 : min(n, j0);
                acc_flush<G, ENERGY>(acc, A, node, gl, stayers - counted);
                counted = stayers;
                if (j0 >= nmax) {
                    if (MODE == kPush && gl == 0 && inside) A.front_dst[cell] = stayers;
                    set += kWarps;
                    enter();
                    if (set >= sets) break;
                    j0 = 0;
                    counted = 0;
                }
                jstop = min(nmax, j0 + kFlushChunks * G);
            }
        }
    }
    if (MODE == kPush) {
        if (queued > 0) left_exits += place_movers(A, q, s_meta, T, tgx0, tgy0, 0, queued, lane, lt);
        const uint32_t left = __reduce_add_sync(kFull, left_exits);
        if (lane == 0 && left) atomicAdd(A.counters, (unsigned long long)left);
    }
}

template <int MODE, bool ENERGY, bool BZU, int G>
__device__ __forceinline__ void cells_body(const KArgs& A, Tile T, uint32_t tile) {
    __shared__ CellShared<MODE, BZU> S;
    const int cells = 1 << (T.ltx + T.lty);  // (a multiple of 32: whole warps below)
    // tiles in row order: the blocks resident at a time work on one stretch
    // of the slot arrays
    const uint32_t tiles_x = (uint32_t)(A.nx + (1 << T.ltx) - 1) >> T.ltx, tile_y = tile / tiles_x;
    const int tgx0 = (int)(tile - tile_y * tiles_x) << T.ltx, tgy0 = (int)tile_y << T.lty;
    bool wide = false;
    for (int i = threadIdx.x; i < cells; i += kThreads) {
        const int gx = tgx0 + (i & ((1 << T.ltx) - 1)), gy = tgy0 + (i >> T.ltx);
        CellMeta m{0u, 0u, 0u, 0u};
        if (gx < A.nx && gy < A.ny) {
            const int64_t c = (int64_t)gy * A.nx + gx;
            m.b0 = A.base[c];
            m.b1 = A.base[c + 1];
            m.nf = MODE == kArrivals ? 0u : A.front_src[c];
            m.nb = A.back_src[c];
        }
        S.meta[i] = m;
        wide = wide || crowded<G>(m.nf + m.nb);
    }
    const int rowlen = (1 << T.ltx) + 1;
    if (MODE == kPush) {
        const int nodes = rowlen * ((1 << T.lty) + 1);
        for (int i = threadIdx.x; i < nodes; i += kThreads) {
            const int ly = i / rowlen, x = tgx0 + (i - ly * rowlen), y = tgy0 + ly;
            S.fld[i] = NodeField<BZU>::from((x < A.GX && y < A.ny + 1) ? __ldg(A.fld + (int64_t)y * A.GX + x)
                                                                       : make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
    if (__syncthreads_or(wide)) cells_run<MODE, ENERGY, BZU, 32>(A, T, tgx0, tgy0, S);
    else cells_run<MODE, ENERGY, BZU, G>(A, T, tgx0, tgy0, S);
}

// The tiles of the tile shapes 1, 2 and 3 (256 cells), and the two that shape
// 0 chooses from (pick_tile).
constexpr int kNumTileShapes = 4;
constexpr int kNumTiles = 5;
constexpr Tile kTile[kNumTiles] = {{5, 0}, {8, 0}, {7, 1}, {4, 4}, {6, 0}};

template <int MODE, bool ENERGY, bool BZU, int G>
__global__ void __launch_bounds__(kThreads, kCellBlocksPerSM) k_cells(KArgs A, Tile T) {
    if (MODE == kArrivals) pdl_wait();
    cells_body<MODE, ENERGY, BZU, G>(A, T, blockIdx.x);
}

// One launch over many instances: block b works on tile work[b].y of instance
// work[b].x, whose arguments are args[work[b].x].
template <int MODE, bool ENERGY, bool BZU, int G>
__global__ void __launch_bounds__(kThreads, kCellBlocksPerSM) k_cells_batch(const KArgs* __restrict__ args,
                                                             const uint2* __restrict__ work, Tile T) {
    __shared__ KArgs s_args;
    const uint2 w = work[blockIdx.x];
    static_assert(sizeof(KArgs) % 8 == 0, "KArgs copy");
    for (int i = threadIdx.x; i < (int)(sizeof(KArgs) / 8); i += kThreads)
        reinterpret_cast<unsigned long long*>(&s_args)[i] =
            reinterpret_cast<const unsigned long long*>(args + w.x)[i];
    __syncthreads();
    cells_body<MODE, ENERGY, BZU, G>(s_args, T, w.y);
}

// ---- side lists ---------------------------------------------------------------

struct FixArgs {
    int nx, ny, GX;
    SpeciesConsts k;
    const float4* __restrict__ fld;
    float4* dst_a;
    float* dst_vz;
    const uint32_t* __restrict__ base;
    const uint32_t* front;  // final front counts of the new buffer
    uint32_t* back;                      // back counts of the new buffer
    ListDev ovf;    // pushed this step, not yet placed
    ListDev prev;   // part of the state before the push, not yet pushed
    ListDev next;   // output: pushed, did not fit
    unsigned long long* acc_q;
    unsigned long long* acc_e;
    unsigned long long* counters;
    // the end of a push (fixup_body)
    uint32_t* old_back;  // back counts of the buffer that the push read
    int64_t ncells;
    uint32_t* ticket;    // blocks done (zero between pushes)
    unsigned long long* flags;  // pinned host memory: push_report()
    uint32_t seq;
};

// Pushes the particles of the previous side list, deposits them and this
// push's spilled movers, and tries to place both in the free gap of their
// target cells; what does not fit goes to the next side list.  Block b of nb.
template <bool ENERGY>
__device__ __forceinline__ void fixup_lists(const FixArgs& F, uint32_t b, uint32_t nb) {
    const uint32_t n_prev = min(*F.prev.count, F.prev.cap);
    const uint32_t n_ovf = min(*F.ovf.count, F.ovf.cap);
    const uint32_t total = n_prev + n_ovf;
    for (uint32_t i = b * blockDim.x + threadIdx.x; i < total; i += nb * blockDim.x) {
        Pushed p;
        float vz;
        uint32_t t;
        if (i < n_prev) {
            const uint32_t c = F.prev.cell[i];
            const int gx = (int)(c % (uint32_t)F.nx), gy = (int)(c / (uint32_t)F.nx);
            const int64_t n0 = (int64_t)gy * F.GX + gx;
            vz = F.prev.vz[i];
            p = push_one(F.prev.a[i], F.fld[n0], F.fld[n0 + 1], F.fld[n0 + F.GX], F.fld[n0 + F.GX + 1],
                         F.k, gx, gy, F.nx, F.ny);
            if (!p.alive) {
                if (p.left) atomicAdd(F.counters, 1ull);
                continue;
            }
            t = (uint32_t)(p.gy * F.nx + p.gx);
        } else {
            const uint32_t e = i - n_prev;
            const float4 a = F.ovf.a[e];
            p.fx = a.x; p.fy = a.y; p.vx = a.z; p.vy = a.w;
            vz = F.ovf.vz[e];
            t = F.ovf.cell[e];
        }
        const float es = ENERGY ? energy_units(p.vx, p.vy, vz, F.k.escale) : 0.f;
        deposit_one<ENERGY>(F.acc_q, F.acc_e, F.GX, t + t / (uint32_t)F.nx, p.fx, p.fy, es);  // node = t + gy
        const uint32_t lim = (F.base[t + 1] - F.base[t]) - F.front[t];
        const uint32_t k = atomicAdd(F.back + t, 1u);
        if (k < lim) {
            store_slot(F.dst_a, F.dst_vz, F.base[t + 1] - 1u - k, p, vz);
        } else {
            atomicSub(F.back + t, 1u);
            const uint32_t s = atomicAdd(F.next.count, 1u);
            if (s < F.next.cap) {
                F.next.a[s] = make_float4(p.fx, p.fy, p.vx, p.vy);
                F.next.vz[s] = vz;
                F.next.cell[s] = t;
            } else {
                atomicOr(F.counters + 2, 1ull);
            }
        }
    }
}

// The side lists, and the end of a push: the back counts that the push read
// are cleared for the next one, and the last block to finish empties the
// consumed lists and tells the host the new list's length and the error
// counters, with the push's number, in one 8-byte store to pinned memory.
// One launch in place of three clears, two copies and an event (a push of a
// 32^2 grid, all launches: 50 us -> 17 us).
template <bool ENERGY>
__device__ __forceinline__ void fixup_body(const FixArgs& F, uint32_t b, uint32_t nb) {
    fixup_lists<ENERGY>(F, b, nb);
    for (int64_t c = (int64_t)b * blockDim.x + threadIdx.x; c < F.ncells; c += (int64_t)nb * blockDim.x)
        F.old_back[c] = 0u;
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(F.ticket, 1u) == nb - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    const volatile unsigned long long* cnt = F.counters;
    *F.ovf.count = 0u;
    *F.prev.count = 0u;
    *F.ticket = 0u;
    *(volatile unsigned long long*)F.flags =
        push_report(*(volatile uint32_t*)F.next.count, cnt[1] != 0, cnt[2] != 0, F.seq);
}

template <bool ENERGY>
__global__ void __launch_bounds__(256) k_fixup(FixArgs F) {
    pdl_wait();
    fixup_body<ENERGY>(F, blockIdx.x, gridDim.x);
}

// Deposit of the particles on a side list (stand-alone deposit).
template <bool ENERGY>
__global__ void __launch_bounds__(256) k_list_deposit(ListDev L, int nx, int GX, float escale,
                                                      unsigned long long* acc_q, unsigned long long* acc_e) {
    const uint32_t n = min(*L.count, L.cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = L.a[i];
        const uint32_t c = L.cell[i];
        const float en = ENERGY ? energy_units(a.z, a.w, L.vz[i], escale) : 0.f;
        deposit_one<ENERGY>(acc_q, acc_e, GX, c + c / (uint32_t)nx, a.x, a.y, en);  // node = c + gy
    }
}

// ---- layouts: counts, exclusive scans ------------------------------------------
//
// Slot capacity of a cell holding n particles: n + n/2 + 16 (room for a
// step's incoming movers and for the count to drift between re-layouts),
// rounded down to a multiple of 8 so that every cell's run starts on a 128-byte
// line of the float4 array and a 32-byte sector of vz (unaligned runs took
// the Ar+ push of the 1024^2 workload from 0.93 to 1.03 ms: more lines and
// sectors an access).  Down, not up: 24 slots for a cell of one particle in
// place of 16 or 17 took two fifths more memory, and grids that had fitted the
// device or the 32-bit slot indices no longer did.
__host__ __device__ __forceinline__ uint32_t cell_capacity(uint32_t n) { return (n + n / 2u + 16u) & ~7u; }

// cnt[c] = front[c] + back[c]
__global__ void k_cell_counts(const uint32_t* front, const uint32_t* back, int64_t ncells, uint32_t* cnt) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < ncells) cnt[c] = front[c] + back[c];
}

// cnt[cell] += 1 for each side-list entry
__global__ void k_list_counts(ListDev L, uint32_t* cnt) {
    const uint32_t n = min(*L.count, L.cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(cnt + L.cell[i], 1u);
}

template <bool CAP>
__device__ __forceinline__ uint32_t scan_value(const uint32_t* in, int64_t t) {
    return CAP ? cell_capacity(in[t]) : in[t];
}

// With CAP counters[3] collects the total, which may be beyond 32 bits.
template <bool CAP>
__global__ void __launch_bounds__(256) k_scan_partials(const uint32_t* in, int64_t n, uint32_t* partials,
                                                       unsigned long long* counters) {
    __shared__ uint32_t red[8];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    uint32_t s = 0;
    for (int j = threadIdx.x; j < kScanTile; j += 256) {
        const int64_t t = base + j;
        if (t >= n) break;
        s += scan_value<CAP>(in, t);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < 8; ++w) t += red[w];
        partials[blockIdx.x] = t;
        if (CAP) atomicAdd(counters + 3, (unsigned long long)t);
    }
}

// out[t] = sum of values before t, out[n] = total.  With CAP the values are
// cell capacities, and cells that want more than kMaxPerCell raise counters[1].
template <bool CAP>
__global__ void __launch_bounds__(256) k_scan_apply(const uint32_t* in, int64_t n,
                                                    const uint32_t* partials, uint32_t* out,
                                                    unsigned long long* counters) {
    __shared__ uint32_t red[8];
    __shared__ uint32_t wsum[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t pre = 0;
    for (int j = threadIdx.x; j < (int)blockIdx.x; j += 256) pre += partials[j];
    for (int o = 16; o > 0; o >>= 1) pre += __shfl_xor_sync(kFull, pre, o);
    if (lane == 0) red[warp] = pre;
    __syncthreads();
    uint32_t block_pre = 0;
    for (int w = 0; w < 8; ++w) block_pre += red[w];
    // each thread owns 8 consecutive entries
    const int64_t c0 = (int64_t)blockIdx.x * kScanTile + threadIdx.x * 8;
    uint32_t v[8];
    uint32_t tsum = 0, vmax = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t count = (c0 + j < n) ? in[c0 + j] : 0u;
        v[j] = !CAP ? count : (c0 + j < n ? cell_capacity(count) : 0u);
        tsum += v[j];
        vmax = max(vmax, count);
    }
    uint32_t incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += wsum[w];
    uint32_t run = block_pre + wpre + incl - tsum;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int64_t t = c0 + j;
        if (t < n) out[t] = run;
        run += v[j];
        if (t == n - 1) out[n] = run;
    }
    if (CAP && vmax + vmax / 2u + 16u > kMaxPerCell) atomicOr(counters + 1, 1ull);
}

// Copies every cell's particles (front run, then back run) from the old
// layout to the front of its slots in the new one; new_front = count.
__global__ void k_relayout_cells(const float4* __restrict__ src_a, const float* __restrict__ src_vz,
                                 const uint32_t* __restrict__ base, const uint32_t* __restrict__ front,
                                 const uint32_t* __restrict__ back, const uint32_t* __restrict__ nbase,
                                 int64_t ncells, float4* dst_a, float* dst_vz, uint32_t* nfront,
                                 uint32_t* nback) {
    const int64_t c = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (c >= ncells) return;
    const int lane = threadIdx.x & 31;
    const uint32_t nf = front[c], nb = back[c], b0 = base[c], back0 = base[c + 1] - nb;
    const uint32_t d0 = nbase[c];
    for (uint32_t j = lane; j < nf + nb; j += 32) {
        const uint32_t i = j < nf ? b0 + j : back0 + (j - nf);
        dst_a[d0 + j] = src_a[i];
        dst_vz[d0 + j] = src_vz[i];
    }
    if (lane == 0) {
        nfront[c] = nf + nb;
        nback[c] = 0u;
    }
}

// Side-list particles into the new layout, after the cell's own particles.
__global__ void k_relayout_list(ListDev L, const uint32_t* __restrict__ nbase, uint32_t* nfront,
                                float4* dst_a, float* dst_vz) {
    const uint32_t n = min(*L.count, L.cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = L.cell[i];
        const uint32_t s = nbase[c] + atomicAdd(nfront + c, 1u);
        dst_a[s] = L.a[i];
        dst_vz[s] = L.vz[i];
    }
}

// ---- import / export ------------------------------------------------------

// Reference Point -> cell.  The cell follows InsertKernel: gx = (int)(x *
// (1/dx)) in FP64 (src/particles.cpp:230-235); dead (pointer == -1) and
// out-of-domain points get no cell.
// Import of records (converted from reference Points on the host): count
// per cell, then place each record in its cell's front run.
__global__ void k_import_count(const PointRec* __restrict__ recs, int64_t n, uint32_t* cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t cell = recs[i].cell;
    if (cell != kNoCell) atomicAdd(cnt + cell, 1u);
}

__global__ void k_import_place(const PointRec* __restrict__ recs, int64_t n,
                               const uint32_t* __restrict__ base, uint32_t* front, float4* dst_a,
                               float* dst_vz) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const PointRec r = recs[i];
    if (r.cell == kNoCell) return;
    const uint32_t d = base[r.cell] + atomicAdd(front + r.cell, 1u);
    dst_a[d] = make_float4(r.fx, r.fy, r.vx, r.vy);
    dst_vz[d] = r.vz;
}

// Layout -> records in cell order (dense[c] = particles before cell c); the
// host expands them into reference Points.
__global__ void k_export(const float4* __restrict__ a, const float* __restrict__ vz,
                         const uint32_t* __restrict__ base, const uint32_t* __restrict__ front,
                         const uint32_t* __restrict__ back, const uint32_t* __restrict__ dense,
                         int64_t ncells, PointRec* out) {
    const int64_t c = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (c >= ncells) return;
    const int lane = threadIdx.x & 31;
    const uint32_t nf = front[c], nb = back[c], b0 = base[c], back0 = base[c + 1] - nb, d0 = dense[c];
    for (uint32_t j = lane; j < nf + nb; j += 32) {
        const uint32_t i = j < nf ? b0 + j : back0 + (j - nf);
        const float4 v = a[i];
        PointRec r;
        r.cell = (uint32_t)c;
        r.fx = v.x;
        r.fy = v.y;
        r.vx = v.z;
        r.vy = v.w;
        r.vz = vz[i];
        out[d0 + j] = r;
    }
}

// Layout -> raw arrays (cell, fx, fy, vx, vy, vz) in cell order.
__global__ void k_export_state(const float4* __restrict__ a, const float* __restrict__ vz,
                               const uint32_t* __restrict__ base, const uint32_t* __restrict__ front,
                               const uint32_t* __restrict__ back, const uint32_t* __restrict__ dense,
                               int64_t ncells, int32_t* cell, float* fx, float* fy, float* vx,
                               float* vy, float* vzo) {
    const int64_t c = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (c >= ncells) return;
    const int lane = threadIdx.x & 31;
    const uint32_t nf = front[c], nb = back[c], b0 = base[c], back0 = base[c + 1] - nb, d0 = dense[c];
    for (uint32_t j = lane; j < nf + nb; j += 32) {
        const uint32_t i = j < nf ? b0 + j : back0 + (j - nf);
        const float4 v = a[i];
        const uint32_t o = d0 + j;
        cell[o] = (int32_t)c;
        fx[o] = v.x;
        fy[o] = v.y;
        vx[o] = v.z;
        vy[o] = v.w;
        vzo[o] = vz[i];
    }
}

// Live particles per reference bucket key gy*GRID_X + gx.
__global__ void k_bin_counts(const uint32_t* __restrict__ cnt, int nx, int ny, int GX, int32_t* counts) {
    const int64_t nodes = (int64_t)GX * (ny + 1);
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nodes) return;
    const int gx = (int)(k % GX), gy = (int)(k / GX);
    counts[k] = (gx < nx && gy < ny) ? (int32_t)cnt[(int64_t)gy * nx + gx] : 0;
}

// ---- accumulators -> meshes -------------------------------------------------

// final_mesh = weighing * sum of unnormalised corner weights; rho += final *
// (-q/eps) (src/interpolation.cpp:139-171).  Resets the accumulators.
// The conversion of one species' accumulators into its final/energy mesh
// (and rho += final * chrg).
struct FlushEntry {
    int64_t nodes;
    unsigned long long* acc_q;
    unsigned long long* acc_e;
    double qscale, escale, chrg;
    double* final_mesh;
    double* energy_mesh;
    double* rho;
    int energy;
};

// kFlushNodes nodes from i0 on, `stride` apart (coalesced across a block),
// all loads issued before any store: the arrays are distinct, so the loads
// need not wait on each other's stores, and several are in flight at once.
constexpr int kFlushNodes = 4;

__device__ __forceinline__ void flush_nodes(const FlushEntry& F, int64_t i0, int stride, double (&r)[kFlushNodes]) {
    unsigned long long q[kFlushNodes], e[kFlushNodes];
#pragma unroll
    for (int u = 0; u < kFlushNodes; ++u) {
        const int64_t i = i0 + (int64_t)u * stride;
        const bool in = i < F.nodes;
        q[u] = in ? F.acc_q[i] : 0ull;
        e[u] = (in && F.energy) ? F.acc_e[i] : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kFlushNodes; ++u) {
        const int64_t i = i0 + (int64_t)u * stride;
        if (i >= F.nodes) break;
        const double f = (double)q[u] * F.qscale;
        F.acc_q[i] = 0ull;
        F.final_mesh[i] = f;
        if (F.energy) {
            F.energy_mesh[i] = (double)e[u] * F.escale;
            F.acc_e[i] = 0ull;
        } else {
            F.energy_mesh[i] = 0.0;
        }
        r[u] = r[u] + f * F.chrg;
    }
}

// ns species of one grid (the same rho), in order: rho += each one's charge,
// from zero with zero_rho.
struct FlushAll {
    FlushEntry e[PIC_MAX_SPECIES];
    int ns, zero_rho;
};

__global__ void k_flush(FlushAll F) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x * kFlushNodes + threadIdx.x, nodes = F.e[0].nodes;
    double* rho = F.e[0].rho;
    double r[kFlushNodes];
#pragma unroll
    for (int u = 0; u < kFlushNodes; ++u) {
        const int64_t i = i0 + (int64_t)u * blockDim.x;
        r[u] = (F.zero_rho || i >= nodes) ? 0.0 : rho[i];
    }
    for (int s = 0; s < F.ns; ++s) flush_nodes(F.e[s], i0, blockDim.x, r);
#pragma unroll
    for (int u = 0; u < kFlushNodes; ++u) {
        const int64_t i = i0 + (int64_t)u * blockDim.x;
        if (i < nodes) rho[i] = r[u];
    }
}

// ---- device plasma loading (Philox-4x32-10, Salmon et al., SC'11) ----------

__device__ __forceinline__ uint4 philox(uint4 ctr, uint2 key) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * ctr.x, hi0 = __umulhi(0xD2511F53u, ctr.x);
        const uint32_t lo1 = 0xCD9E8D57u * ctr.z, hi1 = __umulhi(0xCD9E8D57u, ctr.z);
        ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
        key.x += 0x9E3779B9u;
        key.y += 0xBB67AE85u;
    }
    return ctr;
}

__device__ __forceinline__ float u01(uint32_t u) { return (float)(u >> 8) * 0x1p-24f; }
__device__ __forceinline__ float u01_open(uint32_t u) { return (float)((u >> 8) + 1u) * 0x1p-24f; }

struct PlasmaArgs {
    int nx, ny;
    int ppc;
    double blob_peak, blob_cx, blob_cy, inv_two_sig2;
    float sigma_v, drift_vx, drift_vy;
    uint2 key;
    uint32_t species;
};

__device__ __forceinline__ uint32_t blob_count(const PlasmaArgs& P, int64_t c) {
    if (P.blob_peak <= 0.0) return 0;
    const int gx = (int)(c % P.nx), gy = (int)(c / P.nx);
    const double rx = gx + 0.5 - P.blob_cx, ry = gy + 0.5 - P.blob_cy;
    const double m = P.blob_peak * exp(-(rx * rx + ry * ry) * P.inv_two_sig2);
    const uint4 r = philox(make_uint4((uint32_t)c, (uint32_t)(c >> 32), P.species, 0xB10Bu), P.key);
    return (uint32_t)floor(m + (double)u01(r.x));
}

__global__ void k_plasma_counts(PlasmaArgs P, int64_t ncells, uint32_t* cnt) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    cnt[c] = (uint32_t)P.ppc + blob_count(P, c);
}

// Particle j of cell c gets the Philox counter dense[c] + j (its index in
// cell order) and the slot base[c] + j.
__global__ void k_plasma_generate(PlasmaArgs P, const uint32_t* __restrict__ dense,
                                  const uint32_t* __restrict__ base, int64_t ncells, float4* a,
                                  float* vz, uint32_t* front, uint32_t* back) {
    const int64_t c = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (c >= ncells) return;
    const int lane = threadIdx.x & 31;
    const uint32_t beg = dense[c], end = dense[c + 1], b0 = base[c];
    for (uint32_t i = beg + lane; i < end; i += 32) {
        const uint4 r0 = philox(make_uint4(i, P.species, 0u, 0x5EEDu), P.key);
        const uint4 r1 = philox(make_uint4(i, P.species, 1u, 0x5EEDu), P.key);
        const float fx = u01(r0.x), fy = u01(r0.y);
        // Box-Muller, per-component sigma = sqrt(e*T/m)
        const float m1 = P.sigma_v * sqrtf(-2.0f * logf(u01_open(r0.z)));
        const float m2 = P.sigma_v * sqrtf(-2.0f * logf(u01_open(r1.x)));
        float s1, c1, s2, c2;
        sincospif(2.0f * u01(r0.w), &s1, &c1);
        sincospif(2.0f * u01(r1.y), &s2, &c2);
        const bool blob = (i - beg) >= (uint32_t)P.ppc;
        float vx = m1 * c1, vy = m1 * s1, vzz = m2 * c2;
        if (blob) {
            vx += P.drift_vx;
            vy += P.drift_vy;
        }
        const uint32_t s = b0 + (i - beg);
        a[s] = make_float4(fx, fy, vx, vy);
        vz[s] = vzz;
    }
    if (lane == 0) {
        front[c] = end - beg;
        back[c] = 0u;
    }
}

inline unsigned grid1d(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

constexpr unsigned long long kMaxSlots = 0xF0000000ull;  // of a species

// out[0..n] = exclusive scan of in (CAP: of cell capacities); returns the
// total through *total when not null (synchronises).  Capacities beyond the
// 32-bit slot indices are an error.
template <bool CAP>
int scan_cells(pic_ctx* c, Species& sp, const uint32_t* in, uint32_t* out, uint32_t* total) {
    const int64_t n = c->ncells;
    const int nparts = (int)((n + kScanTile - 1) / kScanTile);
    if (CAP) PIC_CUDA(cudaMemsetAsync(sp.counters + 3, 0, 8, c->stream));
    k_scan_partials<CAP><<<nparts, 256, 0, c->stream>>>(in, n, c->scan_partials, sp.counters);
    k_scan_apply<CAP><<<nparts, 256, 0, c->stream>>>(in, n, c->scan_partials, out, sp.counters);
    c->launches += 2;
    PIC_CUDA(cudaGetLastError());
    if (total) {
        unsigned long long t = 0;
        if (CAP) PIC_CUDA(cudaMemcpyAsync(&t, sp.counters + 3, 8, cudaMemcpyDeviceToHost, c->stream));
        else PIC_CUDA(cudaMemcpyAsync(&t, out + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
        PIC_CUDA(cudaStreamSynchronize(c->stream));
        if (t > kMaxSlots && CAP)
            return fail(PIC_ERR_CAPACITY, "a species holds at most 4.0e9 particle slots (32-bit indices)");
        *total = (uint32_t)t;
    }
    return PIC_OK;
}

// Species constants for a push, with the Boris factors of a uniform Bz.
SpeciesConsts push_consts(const pic_ctx* c, const Species& sp) {
    SpeciesConsts k = sp.k;
    k.bzu = c->bz_uniform ? 1 : 0;
    k.pery = c->periodic ? 1 : 0;
    const float t = k.h * (float)c->bz_value;
    k.bt = t;
    k.bs = (float)(2.0 * (double)t / (1.0 + (double)t * (double)t));
    return k;
}

KArgs make_args(pic_ctx* c, Species& sp) {
    KArgs A{};
    A.nx = c->nx;
    A.ny = c->ny;
    A.GX = c->GX;
    A.ncells = c->ncells;
    A.k = push_consts(c, sp);
    A.fld = c->fld;
    A.src_a = sp.buf[sp.cur].a;
    A.src_vz = sp.buf[sp.cur].vz;
    A.dst_a = sp.buf[sp.cur ^ 1].a;
    A.dst_vz = sp.buf[sp.cur ^ 1].vz;
    A.base = sp.base;
    A.front_src = sp.front[sp.cur];
    A.back_src = sp.back[sp.cur];
    A.front_dst = sp.front[sp.cur ^ 1];
    A.back_dst = sp.back[sp.cur ^ 1];
    A.ovf = list_dev(sp.ovf);
    A.acc_q = sp.acc_q;
    A.acc_e = sp.acc_e;
    A.counters = sp.counters;
    return A;
}

// What a push leaves to do after k_cells: from the state before it.
FixArgs fix_args(pic_ctx* c, Species& sp, unsigned long long* flags, uint32_t seq) {
    const int dst = sp.cur ^ 1;
    FixArgs F{};
    F.nx = c->nx;
    F.ny = c->ny;
    F.GX = c->GX;
    F.k = push_consts(c, sp);
    F.fld = c->fld;
    F.dst_a = sp.buf[dst].a;
    F.dst_vz = sp.buf[dst].vz;
    F.base = sp.base;
    F.front = sp.front[dst];
    F.back = sp.back[dst];
    F.ovf = list_dev(sp.ovf);
    F.prev = list_dev(sp.loose[sp.lcur]);
    F.next = list_dev(sp.loose[sp.lcur ^ 1]);
    F.acc_q = sp.acc_q;
    F.acc_e = sp.acc_e;
    F.counters = sp.counters;
    F.old_back = sp.back[sp.cur];
    F.ncells = c->ncells;
    F.ticket = sp.list_counts + kTicket;
    F.flags = flags;
    F.seq = seq;
    return F;
}

// The deposit of a push's arrivals reads the buffer that the push wrote.
KArgs arrivals_args(const KArgs& push) {
    KArgs A = push;
    A.src_a = push.dst_a;
    A.src_vz = push.dst_vz;
    A.back_src = push.back_dst;
    return A;
}

unsigned num_tiles(const pic_ctx* c, Tile T) {
    return ((unsigned)(c->nx + (1 << T.ltx) - 1) >> T.ltx) * ((unsigned)(c->ny + (1 << T.lty) - 1) >> T.lty);
}

// The tile of a shape for a species (or batch) of `ppc` particles a cell on
// grids that 64 x 1 tiles cut into `tiles64`.  Shape 0 takes short one-row
// tiles: the blocks resident at a time then work on one short stretch of the
// slot arrays, and the last wave is short.  64 cells when they are sparse (a
// block's prologue is shared by more work: 64 instances of 32 particles a
// cell 3.67 ms a push of both species, 3.85 with 32 cells) and still fill
// the device twice over; 32 otherwise (the 1024^2 workload 1.99 ms, 64 cells
// 2.06, 256 x 1 2.21, 128 x 2 2.41, 16 x 16 2.90).
int pick_tile(int shape, double ppc, int64_t tiles64) {
    if (shape != 0) return shape;
    return ppc < 48.0 && tiles64 >= 2 * 6 * 148 ? 4 : 0;
}

// Lanes a cell of a push.  Few lanes: a warp's set has more cells, so the
// per-set work (metadata, reduction, REDs) is shared by more of them and
// sparse cells leave fewer lanes idle; many lanes: longer contiguous runs an
// access.  (By the mean: tiles with cells far fuller than the rest see to
// themselves, crowded().)  Measured, electron + ion push of a 512^2 grid in us with 4 / 8 /
// 16 lanes: 4 particles a cell 100 / 114 / 169, 8: 118 / 126 / 174, 16: 168 /
// 162 / 189, 32: 254 / 230 / 240, 48: 355 / 313 / 309, 64: 430 / 374 / 366.
int pick_lanes(double ppc) { return ppc >= 48.0 ? 16 : (ppc >= 12.0 ? 8 : 4); }

// What a launch of the cell kernels needs to know besides its arguments.
struct CellLaunch {
    int tile;   // index into kTile
    int lanes;  // lanes a cell of a push
    bool bzu;   // uniform Bz
};

CellLaunch cell_launch(const pic_ctx* c, const Species& sp) {
    return CellLaunch{pick_tile(c->tile_shape, sp.ppc, num_tiles(c, kTile[4])), pick_lanes(sp.ppc),
                      c->bz_uniform};
}

// A tenth to a fifth of a cell's electrons arrive a step, few of its ions:
// 4 lanes (with the push's 16, arrivals of the 512^2 workload took 43 us of
// mostly idle lanes instead of 22).
constexpr int kDepositLanes = 8, kArrivalLanes = 4;

// f(lanes a cell, uniform Bz) with both as compile-time constants
template <typename F>
void with_lanes(const CellLaunch& L, F&& f) {
    auto go = [&](auto g) {
        if (L.bzu) f(g, std::true_type());
        else f(g, std::false_type());
    };
    if (L.lanes == 16) go(std::integral_constant<int, 16>());
    else if (L.lanes == 8) go(std::integral_constant<int, 8>());
    else go(std::integral_constant<int, 4>());
}

template <int MODE, bool ENERGY>
void launch_cells(const CellLaunch& L, const pic_ctx* c, const KArgs& A) {
    const Tile T = kTile[L.tile];
    if constexpr (MODE == kPush) {
        with_lanes(L, [&](auto g, auto bzu) {
            k_cells<MODE, ENERGY, decltype(bzu)::value, decltype(g)::value><<<num_tiles(c, T), kThreads, 0, c->stream>>>(A, T);
        });
    } else {
        constexpr int G = MODE == kDeposit ? kDepositLanes : kArrivalLanes;
        if (MODE == kArrivals)
            launch_pdl(k_cells<MODE, ENERGY, true, G>, num_tiles(c, T), kThreads, 0, c->stream, A, T);
        else
            k_cells<MODE, ENERGY, true, G><<<num_tiles(c, T), kThreads, 0, c->stream>>>(A, T);
    }
}

template <int MODE, bool ENERGY>
void launch_cells_batch(const CellLaunch& L, unsigned nblocks, cudaStream_t st, const KArgs* args, const uint2* work) {
    const Tile T = kTile[L.tile];
    if constexpr (MODE == kPush) {
        with_lanes(L, [&](auto g, auto bzu) {
            k_cells_batch<MODE, ENERGY, decltype(bzu)::value, decltype(g)::value><<<nblocks, kThreads, 0, st>>>(args, work, T);
        });
    } else {
        constexpr int G = MODE == kDeposit ? kDepositLanes : kArrivalLanes;
        k_cells_batch<MODE, ENERGY, true, G><<<nblocks, kThreads, 0, st>>>(args, work, T);
    }
}

int check_flags(pic_ctx* c, Species& sp, bool sync);

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static int list_alloc(LooseList& L, uint32_t cap, uint32_t* count) {
    cudaFree(L.a);
    cudaFree(L.vz);
    cudaFree(L.cell);
    L = LooseList{};
    L.count = count;  // (a list without room is an empty one to the kernels)
    PIC_CUDA(cudaMalloc(&L.a, (size_t)cap * sizeof(float4)));
    PIC_CUDA(cudaMalloc(&L.vz, (size_t)cap * sizeof(float)));
    PIC_CUDA(cudaMalloc(&L.cell, (size_t)cap * sizeof(uint32_t)));
    L.cap = cap;
    return PIC_OK;
}

static void list_free(LooseList& L) {
    cudaFree(L.a);
    cudaFree(L.vz);
    cudaFree(L.cell);
    L = LooseList{};
}

static int grow_store(pic_ctx* c, int s, int64_t capacity);
static int grow_lists(pic_ctx* c, int s);

// Side lists hold up to 1/16 of the slots (at least 2^20 particles).
static uint32_t list_capacity(int64_t slots) {
    return (uint32_t)std::min<int64_t>(std::max<int64_t>(slots / 16, 1 << 20), 0x40000000ll);
}

int species_setup(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    sp.desc = c->cfg.species[s];
    if (sp.desc.mass <= 0 || sp.desc.sim_count <= 0)
        return fail(PIC_ERR_CONFIG, "species mass and SimulationParticles must be positive");
    sp.ctom = sp.desc.charge / sp.desc.mass;  // initCtoM, src/particles.cpp:298-300
    const double surf = c->cfg.surf_area > 0 ? c->cfg.surf_area : c->cfg.xmax * c->cfg.ymax;
    // updateWeighingFactor, src/particles.cpp:303-305
    sp.weighing = sp.desc.actual_count * surf / (sp.desc.sim_count * c->dx * c->dy * c->dx * c->dy);
    sp.k.h = (float)(0.5 * sp.ctom * c->cfg.dt);
    sp.k.dtdx = (float)(c->cfg.dt / c->dx);
    sp.k.dtdy = (float)(c->cfg.dt / c->dy);
    sp.k.escale = sp.ctom != 0 ? (float)(0.5 / std::fabs(sp.ctom)) * kEnergyScale : 0.f;
    const size_t nc = (size_t)c->ncells;
    PIC_CUDA(cudaMalloc(&sp.base, (nc + 1) * sizeof(uint32_t)));
    PIC_CUDA(cudaMalloc(&sp.base_next, (nc + 1) * sizeof(uint32_t)));
    for (int b = 0; b < 2; ++b) {
        PIC_CUDA(cudaMalloc(&sp.front[b], nc * sizeof(uint32_t)));
        PIC_CUDA(cudaMalloc(&sp.back[b], nc * sizeof(uint32_t)));
        PIC_CUDA(cudaMemsetAsync(sp.front[b], 0, nc * sizeof(uint32_t), c->stream));
        PIC_CUDA(cudaMemsetAsync(sp.back[b], 0, nc * sizeof(uint32_t), c->stream));
    }
    PIC_CUDA(cudaMalloc(&sp.cnt, nc * sizeof(uint32_t)));
    PIC_CUDA(cudaMalloc(&sp.dense, (nc + 1) * sizeof(uint32_t)));
    PIC_CUDA(cudaMalloc(&sp.list_counts, 4 * sizeof(uint32_t)));
    PIC_CUDA(cudaMemsetAsync(sp.list_counts, 0, 4 * sizeof(uint32_t), c->stream));
    PIC_CUDA(cudaMalloc(&sp.acc_q, (size_t)c->nodes * 2 * sizeof(unsigned long long)));
    sp.acc_e = sp.acc_q + c->nodes;
    PIC_CUDA(cudaMalloc(&sp.final_mesh, (size_t)c->nodes * sizeof(double)));
    PIC_CUDA(cudaMalloc(&sp.energy_mesh, (size_t)c->nodes * sizeof(double)));
    PIC_CUDA(cudaMalloc(&sp.counters, 4 * sizeof(unsigned long long)));
    PIC_CUDA(cudaMallocHost(&sp.flags, sizeof(unsigned long long)));
    *sp.flags = push_report(0u, false, false, 0u);
    PIC_CUDA(cudaMemsetAsync(sp.acc_q, 0, (size_t)c->nodes * 16, c->stream));
    PIC_CUDA(cudaMemsetAsync(sp.final_mesh, 0, (size_t)c->nodes * 8, c->stream));
    PIC_CUDA(cudaMemsetAsync(sp.energy_mesh, 0, (size_t)c->nodes * 8, c->stream));
    PIC_CUDA(cudaMemsetAsync(sp.counters, 0, 4 * sizeof(unsigned long long), c->stream));
    // an empty layout: every cell owns cell_capacity(0) slots
    PIC_CUDA(cudaMemsetAsync(sp.cnt, 0, nc * sizeof(uint32_t), c->stream));
    uint32_t total = 0;
    PIC_TRY(scan_cells<true>(c, sp, sp.cnt, sp.base, &total));
    PIC_TRY(grow_store(c, s, total));
    PIC_TRY(grow_lists(c, s));
    sp.acc_fresh = true;  // zero particles: the zero accumulator is their deposit
    return PIC_OK;
}

void species_free(Species& sp) {
    cudaFree(sp.store);
    cudaFree(sp.base);
    cudaFree(sp.base_next);
    for (int b = 0; b < 2; ++b) {
        cudaFree(sp.front[b]);
        cudaFree(sp.back[b]);
    }
    cudaFree(sp.cnt);
    cudaFree(sp.dense);
    cudaFree(sp.list_counts);
    list_free(sp.ovf);
    list_free(sp.loose[0]);
    list_free(sp.loose[1]);
    if (sp.flags) cudaFreeHost(sp.flags);
    cudaFree(sp.acc_q);
    cudaFree(sp.final_mesh);
    cudaFree(sp.energy_mesh);
    cudaFree(sp.counters);
    sp = Species{};
}

// Grows the buffers to `capacity` slots each, keeping the current buffer's
// contents (same layout).
static int grow_store(pic_ctx* c, int s, int64_t capacity) {
    Species& sp = c->sp[s];
    if (capacity <= sp.capacity && sp.store) return PIC_OK;
    // multiples of 64 slots keep both buffers' float4 arrays 256-byte aligned
    capacity = (capacity + 63) & ~(int64_t)63;
    if (capacity > (int64_t)kMaxSlots)
        return fail(PIC_ERR_CAPACITY, "a species holds at most 4.0e9 particle slots (32-bit indices)");
    float* store = nullptr;
    PIC_CUDA(cudaMalloc(&store, (size_t)capacity * 2 * 5 * sizeof(float)));
    ParticleSoA nb[2];
    for (int b = 0; b < 2; ++b) {
        nb[b].a = reinterpret_cast<float4*>(store + (size_t)b * capacity * 5);
        nb[b].vz = store + (size_t)b * capacity * 5 + (size_t)capacity * 4;
    }
    if (sp.store && sp.capacity > 0) {
        PIC_CUDA(cudaMemcpyAsync(nb[sp.cur].a, sp.buf[sp.cur].a, (size_t)sp.capacity * sizeof(float4),
                                 cudaMemcpyDeviceToDevice, c->stream));
        PIC_CUDA(cudaMemcpyAsync(nb[sp.cur].vz, sp.buf[sp.cur].vz, (size_t)sp.capacity * sizeof(float),
                                 cudaMemcpyDeviceToDevice, c->stream));
        PIC_CUDA(cudaStreamSynchronize(c->stream));
    }
    cudaFree(sp.store);
    sp.store = store;
    sp.buf[0] = nb[0];
    sp.buf[1] = nb[1];
    sp.capacity = capacity;
    return PIC_OK;
}

// Sizes the side lists for the current capacity; only called while they
// are empty.
static int grow_lists(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    const uint32_t lc = list_capacity(sp.capacity);
    if (lc <= std::min({sp.ovf.cap, sp.loose[0].cap, sp.loose[1].cap})) return PIC_OK;
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    PIC_TRY(list_alloc(sp.ovf, lc, sp.list_counts + kOvf));
    PIC_TRY(list_alloc(sp.loose[0], lc, sp.list_counts + kLoose0));
    PIC_TRY(list_alloc(sp.loose[1], lc, sp.list_counts + kLoose1));
    return PIC_OK;
}

static int normalize(pic_ctx* c, int s);

int species_reserve(pic_ctx* c, int s, int64_t capacity) {
    Species& sp = c->sp[s];
    if (sp.store) PIC_TRY(normalize(c, s));  // side lists empty before they are resized
    PIC_TRY(grow_store(c, s, capacity));
    return grow_lists(c, s);
}

namespace {

// The error flags that the last push leaves in pinned memory (k_fixup).
// sync: wait for them; otherwise only look when they are already there.
int check_flags(pic_ctx* c, Species& sp, bool sync) {
    if (!sp.flags_pending) return PIC_OK;
    if (sync) PIC_CUDA(cudaStreamSynchronize(c->stream));
    const unsigned long long f = *(volatile unsigned long long*)sp.flags;
    if (report_seq(f) != (sp.push_seq & kReportSeqMask)) {
        if (sync) return fail(PIC_ERR_CUDA, "a push did not report its end");
        return PIC_OK;
    }
    sp.flags_pending = false;
    sp.loose_count = report_loose(f);
    if (report_cell_limit(f)) return fail(PIC_ERR_CAPACITY, "a cell exceeds the per-cell particle limit");
    if (report_lost(f)) return fail(PIC_ERR_CAPACITY, "particle side list overflowed: particles were lost");
    return PIC_OK;
}

}  // namespace

// Particles a cell, on average, of a layout of `slots` slots (cell_capacity).
static double mean_count(const pic_ctx* c, uint32_t slots) {
    return std::max(0.0, ((double)slots / (double)c->ncells - 12.5) / 1.5);
}

// Rebuilds the layout from the current per-cell counts (cell runs plus the
// side list): every cell gets cell_capacity(count) slots with its particles
// at the front.  Synchronises.
static int relayout(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    const int64_t nc = c->ncells;
    const int src = sp.cur;
    const ListDev L = list_dev(sp.loose[sp.lcur]);
    k_cell_counts<<<grid1d(nc, 256), 256, 0, c->stream>>>(sp.front[src], sp.back[src], nc, sp.cnt);
    k_list_counts<<<kFixupBlocks, 256, 0, c->stream>>>(L, sp.cnt);
    c->launches += 2;
    uint32_t total = 0;
    PIC_TRY(scan_cells<true>(c, sp, sp.cnt, sp.base_next, &total));
    sp.ppc = mean_count(c, total);
    const int dst = src ^ 1;
    if ((int64_t)total > sp.capacity) {
        // grow: a fresh store, the old current buffer copied into its buffer
        // `src` first (same layout), then rebuilt into `dst` as usual
        PIC_TRY(grow_store(c, s, (int64_t)total + total / 8));
    }
    k_relayout_cells<<<grid1d(nc, 8), 256, 0, c->stream>>>(
        sp.buf[src].a, sp.buf[src].vz, sp.base, sp.front[src], sp.back[src], sp.base_next, nc,
        sp.buf[dst].a, sp.buf[dst].vz, sp.front[dst], sp.back[dst]);
    k_relayout_list<<<kFixupBlocks, 256, 0, c->stream>>>(L, sp.base_next, sp.front[dst], sp.buf[dst].a,
                                                         sp.buf[dst].vz);
    c->launches += 2;
    PIC_CUDA(cudaGetLastError());
    PIC_CUDA(cudaMemsetAsync(sp.back[src], 0, (size_t)nc * 4, c->stream));  // as a push leaves them
    PIC_CUDA(cudaMemsetAsync(sp.list_counts, 0, 4 * sizeof(uint32_t), c->stream));
    std::swap(sp.base, sp.base_next);
    sp.cur = dst;
    sp.lcur = 0;
    sp.flags_pending = false;
    sp.loose_count = 0u;
    unsigned long long flags[3] = {0, 0, 0};
    PIC_CUDA(cudaMemcpyAsync(flags, sp.counters, sizeof(flags), cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    if (flags[1]) return fail(PIC_ERR_CAPACITY, "a cell exceeds the per-cell particle limit");
    if (flags[2]) return fail(PIC_ERR_CAPACITY, "particle side list overflowed: particles were lost");
    return grow_lists(c, s);
}

// Every particle in a cell run (side list empty).  Synchronises.
static int normalize(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    PIC_TRY(check_flags(c, sp, true));
    uint32_t n = 0;
    PIC_CUDA(cudaMemcpyAsync(&n, sp.list_counts + kLoose0 + sp.lcur, sizeof(uint32_t),
                             cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    if (n > 0) PIC_TRY(relayout(c, s));
    return PIC_OK;
}

// cnt = particles per cell, dense = its exclusive scan; *total = particles.
static int count_cells(pic_ctx* c, int s, int64_t* total) {
    Species& sp = c->sp[s];
    PIC_TRY(normalize(c, s));
    k_cell_counts<<<grid1d(c->ncells, 256), 256, 0, c->stream>>>(sp.front[sp.cur], sp.back[sp.cur],
                                                                 c->ncells, sp.cnt);
    c->launches += 1;
    uint32_t t = 0;
    PIC_TRY(scan_cells<false>(c, sp, sp.cnt, sp.dense, &t));
    *total = t;
    return PIC_OK;
}

int ensure_staging(pic_ctx* c, size_t bytes) {
    if (bytes <= c->staging_bytes) return PIC_OK;
    // whole 32 MiB granules: requests of nearly the same size (an export,
    // then an import of the same particles) reuse the buffer
    constexpr size_t kGranule = 32u << 20;
    bytes = (bytes + kGranule - 1) / kGranule * kGranule;
    cudaFree(c->staging);
    c->staging = nullptr;
    c->staging_bytes = 0;
    PIC_CUDA(cudaMalloc(&c->staging, bytes));
    c->staging_bytes = bytes;
    return PIC_OK;
}

int particles_import_staging(pic_ctx* c, int64_t n, PointRec** dev_recs) {
    PIC_TRY(ensure_staging(c, (size_t)n * sizeof(PointRec)));
    *dev_recs = static_cast<PointRec*>(c->staging);
    return PIC_OK;
}

// Leaves a species without particles, and without room for any: after its
// buffers were given up and larger ones, or larger lists, could not be had.
static int drop_particles(pic_ctx* c, Species& sp) {
    const size_t bytes = (size_t)c->ncells * 4;
    cudaGetLastError();
    PIC_CUDA(cudaMemsetAsync(sp.base, 0, bytes + 4, c->stream));
    for (int b = 0; b < 2; ++b) {
        PIC_CUDA(cudaMemsetAsync(sp.front[b], 0, bytes, c->stream));
        PIC_CUDA(cudaMemsetAsync(sp.back[b], 0, bytes, c->stream));
    }
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    sp.acc_fresh = false;
    return PIC_OK;
}

// Installs a fresh layout from sp.cnt (particles per cell): base from the
// cell capacities, growing the buffers when needed.  The current buffer's
// contents are dropped, unless the counts are refused.
static int fresh_layout(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    uint32_t total = 0;
    PIC_TRY(scan_cells<true>(c, sp, sp.cnt, sp.base_next, &total));
    unsigned long long flags[2] = {0, 0};
    PIC_CUDA(cudaMemcpyAsync(flags, sp.counters, sizeof(flags), cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    if (flags[1]) {
        PIC_CUDA(cudaMemsetAsync(sp.counters + 1, 0, 8, c->stream));
        return fail(PIC_ERR_CAPACITY, "a cell exceeds the per-cell particle limit");
    }
    std::swap(sp.base, sp.base_next);
    PIC_CUDA(cudaMemsetAsync(sp.list_counts, 0, 4 * sizeof(uint32_t), c->stream));
    sp.lcur = 0;
    sp.flags_pending = false;
    sp.loose_count = 0u;
    sp.ppc = mean_count(c, total);
    int st = PIC_OK;
    if ((int64_t)total > sp.capacity) {
        PIC_CUDA(cudaStreamSynchronize(c->stream));
        cudaFree(sp.store);
        sp.store = nullptr;
        sp.capacity = 0;
        st = grow_store(c, s, total);
    }
    if (st == PIC_OK) st = grow_lists(c, s);
    if (st != PIC_OK) {
        const std::string why = pic_last_error();
        PIC_TRY(drop_particles(c, sp));
        return fail(st, why);
    }
    return PIC_OK;
}

int particles_import(pic_ctx* c, int s, int64_t n) {
    Species& sp = c->sp[s];
    if ((size_t)n * sizeof(PointRec) > c->staging_bytes)
        return fail(PIC_ERR_STATE, "import staging too small");
    const PointRec* recs = static_cast<const PointRec*>(c->staging);
    PIC_CUDA(cudaMemsetAsync(sp.cnt, 0, (size_t)c->ncells * 4, c->stream));
    if (n > 0) k_import_count<<<grid1d(n, 256), 256, 0, c->stream>>>(recs, n, sp.cnt);
    PIC_TRY(fresh_layout(c, s));
    const int b = sp.cur;
    PIC_CUDA(cudaMemsetAsync(sp.front[b], 0, (size_t)c->ncells * 4, c->stream));
    PIC_CUDA(cudaMemsetAsync(sp.back[b], 0, (size_t)c->ncells * 4, c->stream));
    if (n > 0)
        k_import_place<<<grid1d(n, 256), 256, 0, c->stream>>>(recs, n, sp.base, sp.front[b],
                                                              sp.buf[b].a, sp.buf[b].vz);
    c->launches += 2;
    PIC_CUDA(cudaGetLastError());
    sp.acc_fresh = false;
    return PIC_OK;
}

int particles_export(pic_ctx* c, int s, PointRec* dev_out, int64_t* n_out) {
    Species& sp = c->sp[s];
    int64_t n = 0;
    PIC_TRY(count_cells(c, s, &n));
    *n_out = n;
    if (n == 0) return PIC_OK;
    const int b = sp.cur;
    k_export<<<grid1d(c->ncells, 8), 256, 0, c->stream>>>(sp.buf[b].a, sp.buf[b].vz, sp.base,
                                                          sp.front[b], sp.back[b], sp.dense,
                                                          c->ncells, dev_out);
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

int particles_export_state(pic_ctx* c, int s, void* dev, int64_t n) {
    Species& sp = c->sp[s];
    int64_t m = 0;
    PIC_TRY(count_cells(c, s, &m));
    if (m != n) return fail(PIC_ERR_STATE, "particle count changed during export");
    if (n == 0) return PIC_OK;
    int32_t* cell = static_cast<int32_t*>(dev);
    float* f = reinterpret_cast<float*>(cell + n);
    const int b = sp.cur;
    k_export_state<<<grid1d(c->ncells, 8), 256, 0, c->stream>>>(
        sp.buf[b].a, sp.buf[b].vz, sp.base, sp.front[b], sp.back[b], sp.dense, c->ncells, cell, f,
        f + n, f + 2 * n, f + 3 * n, f + 4 * n);
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

int particles_count(pic_ctx* c, int s, int64_t* n) { return count_cells(c, s, n); }

int particles_bin_counts(pic_ctx* c, int s, int32_t* dev_counts) {
    Species& sp = c->sp[s];
    int64_t n = 0;
    PIC_TRY(count_cells(c, s, &n));
    k_bin_counts<<<grid1d(c->nodes, 256), 256, 0, c->stream>>>(sp.cnt, c->nx, c->ny, c->GX, dev_counts);
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

int particles_load_plasma(pic_ctx* c, int s, const pic_plasma_desc* d) {
    Species& sp = c->sp[s];
    if (d->ppc < 0 || d->temperature_ev < 0 || d->blob_peak_ppc < 0)
        return fail(PIC_ERR_ARG, "plasma description has a negative count or temperature");
    PlasmaArgs P{};
    P.nx = c->nx;
    P.ny = c->ny;
    P.ppc = d->ppc;
    P.blob_peak = d->blob_peak_ppc;
    P.blob_cx = d->blob_cx;
    P.blob_cy = d->blob_cy;
    P.inv_two_sig2 = d->blob_sigma > 0 ? 1.0 / (2.0 * d->blob_sigma * d->blob_sigma) : 0.0;
    P.sigma_v = (float)std::sqrt(1.602176634e-19 * d->temperature_ev / sp.desc.mass);
    P.drift_vx = (float)d->drift_vx;
    P.drift_vy = (float)d->drift_vy;
    P.key = make_uint2((uint32_t)d->seed, (uint32_t)(d->seed >> 32));
    P.species = (uint32_t)s;
    k_plasma_counts<<<grid1d(c->ncells, 256), 256, 0, c->stream>>>(P, c->ncells, sp.cnt);
    c->launches += 1;
    PIC_TRY(scan_cells<false>(c, sp, sp.cnt, sp.dense, nullptr));
    PIC_TRY(fresh_layout(c, s));
    const int b = sp.cur;
    k_plasma_generate<<<grid1d(c->ncells, 8), 256, 0, c->stream>>>(P, sp.dense, sp.base, c->ncells,
                                                                    sp.buf[b].a, sp.buf[b].vz,
                                                                    sp.front[b], sp.back[b]);
    c->launches += 1;
    PIC_CUDA(cudaGetLastError());
    sp.acc_fresh = false;
    return PIC_OK;
}

// Zeroes a species' accumulators, unless they are (a flush leaves them so).
static int clear_accumulators(pic_ctx* c, Species& sp) {
    if (sp.acc_clear) return PIC_OK;
    PIC_CUDA(cudaMemsetAsync(sp.acc_q, 0, (size_t)c->nodes * 16, c->stream));  // acc_q and acc_e
    sp.acc_clear = true;
    return PIC_OK;
}

int particles_deposit(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    PIC_TRY(clear_accumulators(c, sp));
    sp.acc_clear = false;
    KArgs A = make_args(c, sp);
    const bool energy = c->cfg.deposit_energy != 0;
    const ListDev L = list_dev(sp.loose[sp.lcur]);
    prof_begin(c, PIC_PHASE_DEPOSIT);
    const CellLaunch cl = cell_launch(c, sp);
    if (energy) {
        launch_cells<kDeposit, true>(cl, c, A);
        k_list_deposit<true><<<kFixupBlocks, 256, 0, c->stream>>>(L, c->nx, c->GX, sp.k.escale,
                                                                  sp.acc_q, sp.acc_e);
    } else {
        launch_cells<kDeposit, false>(cl, c, A);
        k_list_deposit<false><<<kFixupBlocks, 256, 0, c->stream>>>(L, c->nx, c->GX, sp.k.escale,
                                                                   sp.acc_q, sp.acc_e);
    }
    prof_end(c, PIC_PHASE_DEPOSIT);
    c->launches += 2;
    PIC_CUDA(cudaGetLastError());
    sp.acc_fresh = true;
    return PIC_OK;
}

static FlushEntry flush_entry(const pic_ctx* c, const Species& sp) {
    const double area = c->dx * c->dy;
    return FlushEntry{c->nodes, sp.acc_q, sp.acc_e, kChargeUnit * area * sp.weighing, kEnergyUnit * area * sp.weighing,
                      -sp.desc.charge / c->cfg.epsilon, sp.final_mesh, sp.energy_mesh, c->rho,
                      c->cfg.deposit_energy ? 1 : 0};
}

int particles_flush(pic_ctx* c, int s0, int ns, bool zero_rho) {
    FlushAll F{};
    F.ns = ns;
    F.zero_rho = zero_rho ? 1 : 0;
    for (int k = 0; k < ns; ++k) F.e[k] = flush_entry(c, c->sp[s0 + k]);
    prof_begin(c, PIC_PHASE_FLUSH);
    c->launches += 1;
    k_flush<<<grid1d(c->nodes, 256 * kFlushNodes), 256, 0, c->stream>>>(F);
    prof_end(c, PIC_PHASE_FLUSH);
    PIC_CUDA(cudaGetLastError());
    for (int k = 0; k < ns; ++k) {
        c->sp[s0 + k].acc_fresh = false;
        c->sp[s0 + k].acc_clear = true;
    }
    return PIC_OK;
}

int particles_push(pic_ctx* c, int s) {
    Species& sp = c->sp[s];
    // a side list that keeps growing means the layout no longer fits the
    // particle distribution: rebuild it (looked at without waiting)
    PIC_TRY(check_flags(c, sp, false));
    if (!sp.flags_pending && sp.loose_count > sp.loose[0].cap / 8u) {
        prof_begin(c, PIC_PHASE_RELAYOUT);
        PIC_TRY(relayout(c, s));
        prof_end(c, PIC_PHASE_RELAYOUT);
    }
    KArgs A = make_args(c, sp);
    const CellLaunch cl = cell_launch(c, sp);
    const bool energy = c->cfg.deposit_energy != 0;
    const int dst = sp.cur ^ 1;
    // the accumulators collect the deposit of the new positions (back[dst] is
    // clear: the push before, or whatever made the layout, left it so)
    PIC_TRY(clear_accumulators(c, sp));
    sp.acc_clear = false;
    prof_begin(c, PIC_PHASE_PUSH);
    if (energy)
        launch_cells<kPush, true>(cl, c, A);
    else
        launch_cells<kPush, false>(cl, c, A);
    // the deposit of the particles that changed cell, from the back runs
    const KArgs B = arrivals_args(A);
    if (energy)
        launch_cells<kArrivals, true>(cl, c, B);
    else
        launch_cells<kArrivals, false>(cl, c, B);
    prof_end(c, PIC_PHASE_PUSH);
    PIC_CUDA(cudaGetLastError());
    const FixArgs F = fix_args(c, sp, sp.flags, ++sp.push_seq);
    prof_begin(c, PIC_PHASE_FIXUP);
    if (energy)
        launch_pdl(k_fixup<true>, kFixupBlocks, 256, 0, c->stream, F);
    else
        launch_pdl(k_fixup<false>, kFixupBlocks, 256, 0, c->stream, F);
    prof_end(c, PIC_PHASE_FIXUP);
    PIC_CUDA(cudaGetLastError());
    c->launches += 3;
    sp.lcur ^= 1;
    sp.cur = dst;
    sp.flags_pending = true;
    sp.acc_fresh = true;
    return PIC_OK;
}

}  // namespace picb200

// ---------------------------------------------------------------------------
// Tile-shape autotuning
// ---------------------------------------------------------------------------
namespace picb200 {

int particles_num_tile_shapes() { return kNumTileShapes; }

// Times `reps` push passes of every species with each tile shape on the
// current particles, without committing them (no buffer swap, no side-list
// placement), then restores what the passes touched: the side-list count,
// the counters, and the accumulators (marked stale, so the next
// charge_deposition redeposits).  ms[k] = mean milliseconds of one pass over
// all species with shape k.
int particles_time_shapes(pic_ctx* c, int reps, double* ms) {
    if (!c->fields_valid) PIC_TRY(fields_from_phi(c));
    const int ns = c->cfg.num_species;
    unsigned long long* saved = nullptr;
    PIC_CUDA(cudaMalloc(&saved, (size_t)ns * 4 * sizeof(unsigned long long)));
    for (int s = 0; s < ns; ++s)
        PIC_CUDA(cudaMemcpyAsync(saved + 4 * s, c->sp[s].counters, 4 * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToDevice, c->stream));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    PIC_CUDA(cudaEventCreate(&e0));
    PIC_CUDA(cudaEventCreate(&e1));
    int status = PIC_OK;
    const bool energy = c->cfg.deposit_energy != 0;
    for (int sh = 0; sh < kNumTileShapes && status == PIC_OK; ++sh) {
        float total = 0.f;
        for (int r = -1; r < reps; ++r) {  // r = -1: warm-up
            cudaEventRecord(e0, c->stream);
            for (int s = 0; s < ns; ++s) {
                Species& sp = c->sp[s];
                KArgs A = make_args(c, sp);
                CellLaunch cl = cell_launch(c, sp);
                cl.tile = pick_tile(sh, sp.ppc, num_tiles(c, kTile[4]));
                cudaMemsetAsync(sp.back[sp.cur ^ 1], 0, (size_t)c->ncells * 4, c->stream);
                cudaMemsetAsync(sp.list_counts + kOvf, 0, sizeof(uint32_t), c->stream);
                if (energy)
                    launch_cells<kPush, true>(cl, c, A);
                else
                    launch_cells<kPush, false>(cl, c, A);
            }
            cudaEventRecord(e1, c->stream);
            if (cudaEventSynchronize(e1) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
                status = fail(PIC_ERR_CUDA, "autotune: push launch failed");
                break;
            }
            float t = 0.f;
            cudaEventElapsedTime(&t, e0, e1);
            if (r >= 0) total += t;
        }
        if (ms) ms[sh] = total / (float)std::max(reps, 1);
    }
    for (int s = 0; s < ns; ++s) {
        Species& sp = c->sp[s];
        cudaMemcpyAsync(sp.counters, saved + 4 * s, 4 * sizeof(unsigned long long),
                        cudaMemcpyDeviceToDevice, c->stream);
        cudaMemsetAsync(sp.list_counts + kOvf, 0, sizeof(uint32_t), c->stream);
        cudaMemsetAsync(sp.back[sp.cur ^ 1], 0, (size_t)c->ncells * 4, c->stream);
        sp.acc_fresh = sp.acc_clear = false;
    }
    cudaStreamSynchronize(c->stream);
    cudaFree(saved);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    PIC_CUDA(cudaGetLastError());
    return status;
}

}  // namespace picb200

// ---------------------------------------------------------------------------
// Batched particle phases: one launch per phase over the contexts of an
// ensemble (same device, same stream).  Per-instance arguments live in
// device tables rebuilt by the host before each step; the kernels only read
// them, so a captured step replays with the tables of the next step.
// ---------------------------------------------------------------------------
namespace picb200 {
namespace {

struct ZeroEntry {
    uint32_t* ptr;
    uint64_t words;  // 4-byte words
};

__global__ void k_batch_zero(const ZeroEntry* __restrict__ e, int n) {
    const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t gsize = (int64_t)gridDim.x * blockDim.x;
    for (int i = 0; i < n; ++i) {
        const ZeroEntry z = e[i];
        for (int64_t w = gtid; w < (int64_t)z.words; w += gsize) z.ptr[w] = 0u;
    }
}

// Every species of every instance: block (x, i) works on kFlushNodes x 256
// nodes of instance i, each thread on the same nodes of every species in
// turn (species order; rho starts from zero).
// e[s * n + i]: species s of instance i.
__global__ void k_batch_flush(const FlushEntry* __restrict__ e, int n, int ns) {
    const int i = blockIdx.y;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x * kFlushNodes + threadIdx.x, nodes = e[i].nodes;
    if (i0 >= nodes) return;
    double r[kFlushNodes] = {};
    for (int s = 0; s < ns; ++s) flush_nodes(e[(size_t)s * n + i], i0, blockDim.x, r);
    double* rho = e[i].rho;
#pragma unroll
    for (int u = 0; u < kFlushNodes; ++u)
        if (i0 + (int64_t)u * blockDim.x < nodes) rho[i0 + (int64_t)u * blockDim.x] = r[u];
}

constexpr int kFixupBlocksPerInstance = 4;

template <bool ENERGY>
__global__ void __launch_bounds__(256) k_fixup_batch(const FixArgs* __restrict__ args) {
    const FixArgs F = args[blockIdx.x / kFixupBlocksPerInstance];
    fixup_body<ENERGY>(F, blockIdx.x % kFixupBlocksPerInstance, kFixupBlocksPerInstance);
}

}  // namespace

struct ParticleBatchImpl {
    int n = 0, ns = 0;
    // each tile shape's {instance, tile} of every block: the instances whose Bz is
    // uniform first, the others from block nuniform on
    uint2* work[kNumTiles] = {};
    unsigned nblocks[kNumTiles] = {}, nuniform[kNumTiles] = {};
    std::vector<bool> uniform;  // each instance's Bz when the lists were made
    int64_t lists_made = 0;
    KArgs* d_args = nullptr;      // [ns][n] pushes, then [ns][n] deposits of arrivals
    FixArgs* d_fix = nullptr;     // [ns][n]
    FlushEntry* d_flush = nullptr;  // [ns][n]
    ZeroEntry* d_zero = nullptr;  // [ns][2n]: what the tuner clears before a push
    // pinned host mirrors (one upload per step)
    char* h_tables = nullptr;
    char* d_tables = nullptr;
    size_t table_bytes = 0;
    unsigned long long* h_flags = nullptr;  // pinned, [ns][n]: push_report() of each push
    int64_t max_nodes = 0;  // nodes of the largest instance
    double ppc = 0;         // particles a cell, over all instances and species
};

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Makes the work lists, unless every instance's Bz is of the kind that it was
// when they were made.  (Their lengths do not change.)
static int batch_work(ParticleBatchImpl* B, pic_ctx** cs, cudaStream_t st) {
    std::vector<bool> uniform;
    for (int i = 0; i < B->n; ++i) uniform.push_back(cs[i]->bz_uniform);
    if (B->lists_made && uniform == B->uniform) return PIC_OK;
    for (int sh = 0; sh < kNumTiles; ++sh) {
        std::vector<uint2> w;
        for (const bool kind : {true, false}) {
            for (int i = 0; i < B->n; ++i) {
                if (uniform[i] != kind) continue;
                const unsigned tiles = num_tiles(cs[i], kTile[sh]);
                for (unsigned t = 0; t < tiles; ++t) w.push_back(make_uint2((uint32_t)i, t));
            }
            if (kind) B->nuniform[sh] = (unsigned)w.size();
        }
        B->nblocks[sh] = (unsigned)w.size();
        if (!B->work[sh]) PIC_CUDA(cudaMalloc(&B->work[sh], w.size() * sizeof(uint2)));
        PIC_CUDA(cudaMemcpyAsync(B->work[sh], w.data(), w.size() * sizeof(uint2), cudaMemcpyHostToDevice, st));
    }
    PIC_CUDA(cudaStreamSynchronize(st));
    B->uniform = uniform;
    B->lists_made += 1;
    return PIC_OK;
}

int batch_create(pic_ctx** cs, int n, ParticleBatchImpl** out) {
    auto* B = new ParticleBatchImpl();
    *out = B;
    B->n = n;
    B->ns = cs[0]->cfg.num_species;
    for (int i = 0; i < n; ++i) B->max_nodes = std::max<int64_t>(B->max_nodes, cs[i]->nodes);
    PIC_TRY(batch_work(B, cs, cs[0]->stream));
    const int ns = B->ns;
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        const size_t o = off;
        off += align256(bytes);
        return o;
    };
    const size_t o_args = carve(sizeof(KArgs) * 2 * ns * n), o_fix = carve(sizeof(FixArgs) * ns * n);
    const size_t o_flush = carve(sizeof(FlushEntry) * ns * n), o_zero = carve(sizeof(ZeroEntry) * ns * 2 * n);
    B->table_bytes = off;
    PIC_CUDA(cudaMalloc(&B->d_tables, off));
    PIC_CUDA(cudaMallocHost(&B->h_tables, off));
    std::memset(B->h_tables, 0, off);
    B->d_args = reinterpret_cast<KArgs*>(B->d_tables + o_args);
    B->d_fix = reinterpret_cast<FixArgs*>(B->d_tables + o_fix);
    B->d_flush = reinterpret_cast<FlushEntry*>(B->d_tables + o_flush);
    B->d_zero = reinterpret_cast<ZeroEntry*>(B->d_tables + o_zero);
    PIC_CUDA(cudaMallocHost(&B->h_flags, sizeof(unsigned long long) * ns * n));
    std::memset(B->h_flags, 0, sizeof(unsigned long long) * ns * n);
    return PIC_OK;
}

void batch_destroy(ParticleBatchImpl* B) {
    if (!B) return;
    for (auto* w : B->work) cudaFree(w);
    cudaFree(B->d_tables);
    if (B->h_tables) cudaFreeHost(B->h_tables);
    if (B->h_flags) cudaFreeHost(B->h_flags);
    delete B;
}

// Host part before a step: side-list checks (and rare re-layouts) per
// instance, then the tables of this step, uploaded on `st`.
int batch_prepare(ParticleBatchImpl* B, pic_ctx** cs, cudaStream_t st) {
    const int n = B->n, ns = B->ns;
    for (int i = 0; i < n; ++i)
        for (int s = 0; s < ns; ++s) {
            Species& sp = cs[i]->sp[s];
            unsigned long long& f = B->h_flags[(size_t)s * n + i];
            if (report_cell_limit(f)) return fail(PIC_ERR_CAPACITY, "a cell exceeds the per-cell particle limit");
            if (report_lost(f)) return fail(PIC_ERR_CAPACITY, "particle side list overflowed: particles were lost");
            if (report_loose(f) > sp.loose[0].cap / 8u) {
                PIC_TRY(relayout(cs[i], s));
                f = push_report(0u, false, false, 0u);
            }
        }
    const size_t o_args = 0, o_fix = align256(sizeof(KArgs) * 2 * ns * n);
    const size_t o_flush = o_fix + align256(sizeof(FixArgs) * ns * n);
    const size_t o_zero = o_flush + align256(sizeof(FlushEntry) * ns * n);
    KArgs* ha = reinterpret_cast<KArgs*>(B->h_tables + o_args);
    FixArgs* hf = reinterpret_cast<FixArgs*>(B->h_tables + o_fix);
    FlushEntry* hl = reinterpret_cast<FlushEntry*>(B->h_tables + o_flush);
    ZeroEntry* hz = reinterpret_cast<ZeroEntry*>(B->h_tables + o_zero);
    PIC_TRY(batch_work(B, cs, st));
    double cells = 0, count = 0;
    for (int i = 0; i < n; ++i) {
        pic_ctx* c = cs[i];
        for (int s = 0; s < ns; ++s) {
            cells += (double)c->ncells;
            count += (double)c->ncells * c->sp[s].ppc;
        }
        for (int s = 0; s < ns; ++s) {
            Species& sp = c->sp[s];
            const size_t k = (size_t)s * n + i;
            const int dst = sp.cur ^ 1;
            ha[k] = make_args(c, sp);
            ha[(size_t)ns * n + k] = arrivals_args(ha[k]);
            hf[k] = fix_args(c, sp, B->h_flags + k, 0u);
            hl[k] = flush_entry(c, sp);
            // the tuner's clears: back counts of the new buffer, the spill list
            hz[(size_t)s * 2 * n + i] = ZeroEntry{sp.back[dst], (uint64_t)c->ncells};
            hz[(size_t)s * 2 * n + n + i] = ZeroEntry{sp.list_counts + kOvf, 1};
        }
    }
    B->ppc = count / cells;
    PIC_CUDA(cudaMemcpyAsync(B->d_tables, B->h_tables, B->table_bytes, cudaMemcpyHostToDevice, st));
    return PIC_OK;
}

static CellLaunch batch_launch(const ParticleBatchImpl* B, int shape) {
    return CellLaunch{pick_tile(shape, B->ppc, B->nblocks[4]), pick_lanes(B->ppc), true};
}

// The kernels that a push of the batch launches, as a number: a captured
// step is good for as long as it does not change.
int64_t batch_kernels(const ParticleBatchImpl* B, int shape) {
    const CellLaunch L = batch_launch(B, shape);
    return (B->lists_made * kNumTiles + L.tile) * 64 + L.lanes;
}

// The push pass of species s of every instance: one launch for the instances
// whose Bz is uniform, one for the others.  (An instance's push is then the one
// that it has in a context of its own, whatever the others' Bz.)
template <bool ENERGY>
static void launch_push_batch(const ParticleBatchImpl* B, CellLaunch L, int s, cudaStream_t st) {
    const unsigned nu = B->nuniform[L.tile], nv = B->nblocks[L.tile] - nu;
    const KArgs* args = B->d_args + (size_t)s * B->n;
    L.bzu = true;
    if (nu) launch_cells_batch<kPush, ENERGY>(L, nu, st, args, B->work[L.tile]);
    L.bzu = false;
    if (nv) launch_cells_batch<kPush, ENERGY>(L, nv, st, args, B->work[L.tile] + nu);
}

// Flush the accumulators of every species of every instance into final/energy
// mesh and rho (from zero), leaving them clear for the push.
int batch_deposit(ParticleBatchImpl* B, cudaStream_t st) {
    const int n = B->n, ns = B->ns;
    const dim3 fg(grid1d(B->max_nodes, 256 * kFlushNodes), (unsigned)n);
    k_batch_flush<<<fg, 256, 0, st>>>(B->d_flush, n, ns);
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

// push every species of every instance; each reports its end in B->h_flags
int batch_push(ParticleBatchImpl* B, int shape, bool energy, cudaStream_t st) {
    const int n = B->n, ns = B->ns;
    const CellLaunch cl = batch_launch(B, shape);
    for (int s = 0; s < ns; ++s) {
        if (energy) launch_push_batch<true>(B, cl, s, st);
        else launch_push_batch<false>(B, cl, s, st);
        if (energy)
            launch_cells_batch<kArrivals, true>(cl, B->nblocks[cl.tile], st, B->d_args + (size_t)(ns + s) * n, B->work[cl.tile]);
        else
            launch_cells_batch<kArrivals, false>(cl, B->nblocks[cl.tile], st, B->d_args + (size_t)(ns + s) * n, B->work[cl.tile]);
        if (energy)
            k_fixup_batch<true><<<n * kFixupBlocksPerInstance, 256, 0, st>>>(B->d_fix + (size_t)s * n);
        else
            k_fixup_batch<false><<<n * kFixupBlocksPerInstance, 256, 0, st>>>(B->d_fix + (size_t)s * n);
    }
    PIC_CUDA(cudaGetLastError());
    return PIC_OK;
}

// Host bookkeeping after a step (the buffers and lists every push flips).
void batch_commit(pic_ctx** cs, int n) {
    for (int i = 0; i < n; ++i)
        for (int s = 0; s < cs[i]->cfg.num_species; ++s) {
            Species& sp = cs[i]->sp[s];
            sp.cur ^= 1;
            sp.lcur ^= 1;
            sp.acc_fresh = true;
            sp.acc_clear = false;
            sp.flags_pending = false;
        }
}

}  // namespace picb200

namespace picb200 {

// Times `reps` batched push passes of all species with each tile shape on the
// current particles of every instance, without committing them; restores
// the counters and side-list counts the passes touched and marks the
// accumulators stale.  Tables must be prepared (batch_prepare).
int batch_time_shapes(ParticleBatchImpl* B, pic_ctx** cs, cudaStream_t st, int reps, bool energy,
                      double* ms) {
    const int n = B->n, ns = B->ns;
    unsigned long long* saved = nullptr;
    PIC_CUDA(cudaMalloc(&saved, (size_t)n * ns * 4 * sizeof(unsigned long long)));
    for (int i = 0; i < n; ++i)
        for (int s = 0; s < ns; ++s)
            PIC_CUDA(cudaMemcpyAsync(saved + 4 * ((size_t)i * ns + s), cs[i]->sp[s].counters,
                                     4 * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    PIC_CUDA(cudaEventCreate(&e0));
    PIC_CUDA(cudaEventCreate(&e1));
    int status = PIC_OK;
    for (int sh = 0; sh < kNumTileShapes && status == PIC_OK; ++sh) {
        const CellLaunch cl = batch_launch(B, sh);
        float total = 0.f;
        for (int r = -1; r < reps; ++r) {
            cudaEventRecord(e0, st);
            for (int s = 0; s < ns; ++s) {
                k_batch_zero<<<296, 256, 0, st>>>(B->d_zero + (size_t)s * 2 * n, 2 * n);
                if (energy) launch_push_batch<true>(B, cl, s, st);
                else launch_push_batch<false>(B, cl, s, st);
            }
            cudaEventRecord(e1, st);
            if (cudaEventSynchronize(e1) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
                status = fail(PIC_ERR_CUDA, "autotune: batched push launch failed");
                break;
            }
            float t = 0.f;
            cudaEventElapsedTime(&t, e0, e1);
            if (r >= 0) total += t;
        }
        if (ms) ms[sh] = total / (float)std::max(reps, 1);
    }
    for (int i = 0; i < n; ++i)
        for (int s = 0; s < ns; ++s) {
            Species& sp = cs[i]->sp[s];
            cudaMemcpyAsync(sp.counters, saved + 4 * ((size_t)i * ns + s), 4 * sizeof(unsigned long long),
                            cudaMemcpyDeviceToDevice, st);
            cudaMemsetAsync(sp.list_counts + kOvf, 0, sizeof(uint32_t), st);
            cudaMemsetAsync(sp.back[sp.cur ^ 1], 0, (size_t)cs[i]->ncells * 4, st);
            sp.acc_fresh = sp.acc_clear = false;
        }
    cudaStreamSynchronize(st);
    cudaFree(saved);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    PIC_CUDA(cudaGetLastError());
    return status;
}

}  // namespace picb200

// ---------------------------------------------------------------------------
// Particle sources: generate_new_electrons and generate_pairs
// (SYCL-PIC-poissonsolver/src/utils.cpp:374-777, called per step by
// src/sycl_pic_ctypes.cpp:212-236).  New particles are drawn on the device
// (Philox-4x32-10, counter = (call, particle, stream)) and appended to the
// species' side list: they are part of the state at once (deposited into
// the accumulators when those hold the current positions) and are placed in
// their cells by the next push or re-layout.
// ---------------------------------------------------------------------------
namespace picb200 {
namespace {

struct SourceArgs {
    int nx, ny, GX;
    double dx, dy, W, H;
    double x_reinject;
    double x11, x22, xm;
    double ve, vi;  // sqrt(2|q/m|T) of electrons and ions
    uint32_t n_reinject, n_pairs;
    uint2 key;
    uint32_t call;
    ListDev e_list, i_list;
    unsigned long long* e_acc_q;
    unsigned long long* e_acc_e;
    unsigned long long* i_acc_q;
    unsigned long long* i_acc_e;
    int deposit_e, deposit_i, energy;
    float e_escale, i_escale;
    unsigned long long* e_counters;
    unsigned long long* i_counters;
    unsigned* accepted;  // pairs created
};

__device__ __forceinline__ double u01d(uint32_t a, uint32_t b) {
    // 53-bit uniform in [0, 1)
    return (double)(((uint64_t)a << 21) ^ (uint64_t)(b >> 11)) * (1.0 / 9007199254740992.0);
}

// the reference's Maxwellian draw: v * sqrt(-ln u) * (cos, sin)(2 pi u'),
// u clamped below at 1e-10 as ran2 (src/utils.cpp:51-56)
__device__ __forceinline__ void maxwell(double v, uint4 r0, uint4 r1, double& vx, double& vy, double& vz) {
    const double u1 = fmax(u01d(r0.x, r0.y), 1e-10), u2 = u01d(r0.z, r0.w);
    const double u3 = fmax(u01d(r1.x, r1.y), 1e-10), u4 = u01d(r1.z, r1.w);
    const double z1 = sqrt(-log(u1)), z3 = sqrt(-log(u3));
    double s, c;
    sincospi(2.0 * u2, &s, &c);
    vx = v * z1 * c;
    vy = v * z1 * s;
    sincospi(2.0 * u4, &s, &c);
    vz = v * z3 * c;
}

// Appends one particle (FP64 position) to a side list, deposit included.
template <bool ENERGY>
__device__ __forceinline__ void append_point(const SourceArgs& S, const ListDev& L, double x, double y,
                                             double vx, double vy, double vz, bool deposit,
                                             unsigned long long* acc_q, unsigned long long* acc_e,
                                             float escale, unsigned long long* counters) {
    const double sx = x * (1.0 / S.dx), sy = y * (1.0 / S.dy);
    if (!(sx >= 0.0 && sy >= 0.0 && sx < (double)S.nx && sy < (double)S.ny)) return;
    const int gx = (int)sx, gy = (int)sy;
    const float fx = fminf((float)(sx - gx), kOneBelow), fy = fminf((float)(sy - gy), kOneBelow);
    const uint32_t s = atomicAdd(L.count, 1u);
    if (s >= L.cap) {
        atomicOr(counters + 2, 1ull);
        return;
    }
    L.a[s] = make_float4(fx, fy, (float)vx, (float)vy);
    L.vz[s] = (float)vz;
    L.cell[s] = (uint32_t)(gy * S.nx + gx);
    if (deposit) {
        const float en = ENERGY ? energy_units((float)vx, (float)vy, (float)vz, escale) : 0.f;
        deposit_one<ENERGY>(acc_q, acc_e, S.GX, (uint32_t)(gy * S.GX + gx), fx, fy, en);
    }
}

template <bool ENERGY>
__global__ void k_sources(SourceArgs S) {
    const uint32_t total = S.n_reinject + S.n_pairs;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
        const uint4 r0 = philox(make_uint4(k, S.call, 0u, 0x50u), S.key);
        const uint4 r1 = philox(make_uint4(k, S.call, 1u, 0x50u), S.key);
        if (k < S.n_reinject) {
            // generate_new_electrons (src/utils.cpp:397-425): x fixed, y uniform
            double vx, vy, vz;
            maxwell(S.ve, r0, r1, vx, vy, vz);
            const uint4 r2 = philox(make_uint4(k, S.call, 2u, 0x50u), S.key);
            append_point<ENERGY>(S, S.e_list, S.x_reinject, S.H * u01d(r2.x, r2.y), vx, vy, vz, S.deposit_e,
                                 S.e_acc_q, S.e_acc_e, S.e_escale, S.e_counters);
        } else {
            // generate_pairs (src/utils.cpp:517-566): one electron and one
            // ion at x = xm + asin(2u-1)(x22-x11)/pi, y uniform, kept inside (0, W)
            const uint4 r2 = philox(make_uint4(k, S.call, 2u, 0x50u), S.key);
            const uint4 r3 = philox(make_uint4(k, S.call, 3u, 0x50u), S.key);
            const uint4 r4 = philox(make_uint4(k, S.call, 4u, 0x50u), S.key);
            const double x = S.xm + asin(2.0 * u01d(r2.x, r2.y) - 1.0) * (S.x22 - S.x11) * (1.0 / 3.14159265358979323846);
            const double y = S.H * u01d(r2.z, r2.w);
            if (!(x > 0.0 && x < S.W)) continue;
            double vx, vy, vz;
            maxwell(S.ve, r0, r1, vx, vy, vz);
            append_point<ENERGY>(S, S.e_list, x, y, vx, vy, vz, S.deposit_e, S.e_acc_q, S.e_acc_e,
                                 S.e_escale, S.e_counters);
            maxwell(S.vi, r3, r4, vx, vy, vz);
            append_point<ENERGY>(S, S.i_list, x, y, vx, vy, vz, S.deposit_i, S.i_acc_q, S.i_acc_e,
                                 S.i_escale, S.i_counters);
            atomicAdd(S.accepted, 1u);
        }
    }
}

}  // namespace

int particles_generate(pic_ctx* c, const pic_source_desc* d, int64_t* n_e, int64_t* n_p) {
    if (c->cfg.num_species < 2) return fail(PIC_ERR_STATE, "particle sources need electrons (species 0) and ions (1)");
    Species& E = c->sp[0];
    Species& I = c->sp[1];
    // re-injection count: electron exits through x < 0 beyond the ions'
    unsigned long long ex[2] = {0, 0};
    PIC_CUDA(cudaMemcpyAsync(&ex[0], E.counters, 8, cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA(cudaMemcpyAsync(&ex[1], I.counters, 8, cudaMemcpyDeviceToHost, c->stream));
    PIC_CUDA(cudaStreamSynchronize(c->stream));
    int64_t num_new = 0;
    if (d->reinject) {
        num_new = std::max<int64_t>((int64_t)ex[0] - (int64_t)ex[1], 0);
        PIC_CUDA(cudaMemsetAsync(E.counters, 0, 8, c->stream));
        PIC_CUDA(cudaMemsetAsync(I.counters, 0, 8, c->stream));
    }
    int64_t target = 0;
    if (d->pairs) {
        // fn = H dt (2/pi) (x22 - x11) ionimax / rate_div (src/utils.cpp:502)
        const double fn = c->cfg.ymax * c->cfg.dt * (2.0 / 3.14159265358979323846) * (d->x22 - d->x11) *
                          d->ionimax / d->rate_div;
        if (fn > 0) target = (int64_t)std::ceil(fn);
    }
    if (n_e) *n_e = 0;
    if (n_p) *n_p = 0;
    if (num_new + target == 0) return PIC_OK;
    if (num_new + target > 0x7fffffffll) return fail(PIC_ERR_CAPACITY, "too many new particles in one call");
    // the side lists must hold them: make room first if needed
    for (Species* sp : {&E, &I}) {
        uint32_t n = 0;
        PIC_CUDA(cudaMemcpy(&n, sp->list_counts + 1 + sp->lcur, 4, cudaMemcpyDeviceToHost));
        if ((int64_t)n + num_new + target > (int64_t)sp->loose[sp->lcur].cap)
            return fail(PIC_ERR_CAPACITY, "particle sources: more new particles than the side list holds");
    }
    unsigned* accepted = nullptr;
    PIC_CUDA(cudaMalloc(&accepted, sizeof(unsigned)));
    PIC_CUDA(cudaMemsetAsync(accepted, 0, sizeof(unsigned), c->stream));
    SourceArgs S{};
    S.nx = c->nx;
    S.ny = c->ny;
    S.GX = c->GX;
    S.dx = c->dx;
    S.dy = c->dy;
    S.W = c->cfg.xmax;
    S.H = c->cfg.ymax;
    S.x_reinject = d->reinject_x;
    S.x11 = d->x11;
    S.x22 = d->x22;
    S.xm = d->xm;
    S.ve = std::sqrt(2.0 * std::fabs(E.ctom) * d->te_ev);
    S.vi = std::sqrt(2.0 * std::fabs(I.ctom) * d->ti_ev);
    S.n_reinject = (uint32_t)num_new;
    S.n_pairs = (uint32_t)target;
    S.key = make_uint2((uint32_t)d->seed, (uint32_t)(d->seed >> 32));
    S.call = (uint32_t)c->source_calls++;
    S.e_list = list_dev(E.loose[E.lcur]);
    S.i_list = list_dev(I.loose[I.lcur]);
    S.e_acc_q = E.acc_q;
    S.e_acc_e = E.acc_e;
    S.i_acc_q = I.acc_q;
    S.i_acc_e = I.acc_e;
    S.deposit_e = E.acc_fresh ? 1 : 0;
    S.deposit_i = I.acc_fresh ? 1 : 0;
    S.e_escale = E.k.escale;
    S.i_escale = I.k.escale;
    S.e_counters = E.counters;
    S.i_counters = I.counters;
    S.accepted = accepted;
    const unsigned blocks = (unsigned)std::min<int64_t>((num_new + target + 255) / 256, 148 * 8);
    if (c->cfg.deposit_energy)
        k_sources<true><<<blocks, 256, 0, c->stream>>>(S);
    else
        k_sources<false><<<blocks, 256, 0, c->stream>>>(S);
    c->launches += 1;
    unsigned acc_h = 0;
    cudaMemcpyAsync(&acc_h, accepted, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream);
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    cudaFree(accepted);
    if (e != cudaSuccess) return fail(PIC_ERR_CUDA, std::string("particle sources: ") + cudaGetErrorString(e));
    // the new particles make the side lists' host-side counts stale
    E.flags_pending = I.flags_pending = false;
    if (n_e) *n_e = num_new;
    if (n_p) *n_p = acc_h;
    return PIC_OK;
}

}  // namespace picb200
