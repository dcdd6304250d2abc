// Structured-grid triangular substitution: the line pipeline.
//
// For factors whose strict-lower part couples row r = X + nx (Y + ny Z) only to rows
// r - 1 (X > 0), r - nx (Y > 0) and r - nx ny (Z > 0) — a 7-point (3-D) or 5-point (2-D:
// ny = 1, the second offset taken as the plane offset) stencil in natural order, ILU(0) —
// and whose strict-upper part is the mirror image, every row depends on its three
// predecessors along x, y and z.  The sweeps then run on a fixed software pipeline
// instead of level sets:
//
// * in sweep coordinates (x', y', z') — the natural ones for L, mirrored for U — a lane
//   owns one grid line (y', z') and walks it in x', so the x-dependency is the lane's
//   own previous result, in a register;
// * a warp holds wy x wz lines (lane = zz wy + yy) and lane (yy, zz) works on
//   x' = s - (yy + zz) at step s: its y- and z-predecessors at the same x' were computed
//   by lanes (yy - 1, zz) and (yy, zz - 1) one step earlier and arrive by warp shuffles;
// * a CTA holds by x bz compute warps; a warp's first lanes along y / z take their
//   predecessors from a face in shared memory that the previous warp of the CTA fills
//   ([x][wz] / [x][wy] values per warp, value-as-flag: reset to the sentinel per block);
// * faces of a block's first warps are filled by the previous block: through distributed
//   shared memory inside a thread-block cluster, else through an exchange buffer in L2 of
//   the same layout that a halo warp polls and hands back at the sentinel.
//
// What bounds it: the chain of nx + ny + nz steps.  The vectors lie in natural order, so a
// lane's own accesses would touch 32 cache lines per warp and step; they were 64 of the ~70
// L1 wavefronts of a step, and with four warps per SM they set its pace (176 ns per FP32
// step).  So each compute warp has a helper warp on its scheduler that moves the operands and
// the results in chunks of 8 steps through shared memory: the coefficient stream by bulk
// copies, right-hand side and results 8 consecutive rows of a line at a time (the first
// product with `scale` included).  The compute warp touches only staged values, its faces
// and the shuffles, a step is 70 ns (FP32) or 160 / 265 ns (FP64 forward / backward, whose
// FP64 instructions alone take 93 / 186 ns on a scheduler), and a handoff between warps costs
// two to three steps.  Inside GMRES, forward / backward, us: 128^3 FP32 89 / 83 (151 / 137
// with a lane's own accesses), FP64 135 / 194 (247 / 622, block-local backward 492); 256^2
// FP32 45 / 40 (95 / 84), FP64 72 / 129 (204 / block-local 313).
//
// Blocks are taken from a ticket counter in dependency order (anti-diagonals of the block
// grid), so a block only waits for blocks of smaller tickets, whose CTAs are running or
// done; inside a block a warp only waits for warps of smaller index along y or z (all
// resident), whose faces never wait on their consumers.  Every wait is bounded.
//
// A missing neighbour at the grid's boundary has coefficient 0 and value 0, and
// fma(-0, 0, acc) == acc exactly, so the results are bit-identical to the level-ordered
// and block-local kernels (src/ilu_solver.cpp:687-696 for L, 719-729 for U).
#pragma once

#include "common.cuh"
#include "division.cuh"
#include "ilu_kernels.cuh"

namespace gb300 {

constexpr int kLineMaxWarps = 4;  // compute warps per CTA of the line kernels, one per scheduler (each with
                                  // a helper warp)
// Steps staged at a time per compute warp (between its synchronisations with its helper),
// and chunks in flight (two were 15 - 25 % slower, four no faster).
constexpr int kLineChunk = 8;
constexpr int kLineSlots = 3;
// Staged right-hand side and results: per lane a chunk's steps (16-byte accesses by the
// compute warps) and 16 bytes more, which spread the lanes over the banks.
template <class T>
constexpr int kLinePitch = kLineChunk + 16 / static_cast<int>(sizeof(T));
constexpr int kLineWarmLines = 700;  // FP32, 2-D: lines
constexpr int kLineWarmDepth = 280;  // 3-D: lines along y and z
constexpr int kLineStepAlign = 8;  // steps of a warp are rounded up to a multiple of this

struct LineGeom {
    int nx = 0, ny = 0, nz = 0;
    int wy = 1, wz = 32;  // lanes of a warp along y / z (wy * wz == 32)
    int by = 1, bz = 1;   // warps of a CTA along y / z
    int nby = 1, nbz = 1; // blocks along y / z
    int steps = 0;        // steps of a warp: nx + wy + wz - 2 ...
    int psteps = 0;       // ... rounded up to a multiple of kLineStepAlign
    int nblk = 0;         // nby * nbz
    int cl = 0;           // CTAs per thread-block cluster (consecutive blocks along z), 0: none
    int nbzc = 0;         // clusters along z: ceil(nbz / cl)
    __host__ __device__ int nw() const { return by * bz; }
    __host__ __device__ int halo_warps() const { return ny > 1 ? 2 : 1; }
    __host__ __device__ int threads() const { return (2 * nw() + halo_warps()) * 32; }
    // Slot of lane `lane` of warp w of block b at step s in the packed operand stream.
    __host__ __device__ long long slot(int b, int w, int s, int lane) const {
        return ((static_cast<long long>(b) * nw() + w) * psteps + s) * 32 + lane;
    }
    __host__ __device__ long long slots() const { return static_cast<long long>(nblk) * nw() * psteps * 32; }
    // Positions of a face: x' = -pad .. psteps (a lane's x' runs from -(wy + wz - 2) to
    // psteps - 1, faces are read one step ahead).  Only x' in [0, nx) is ever waited for.
    __host__ __device__ int pad() const { return wy + wz - 2; }
    __host__ __device__ int face_len() const { return psteps + pad() + 1; }
    __host__ __device__ int face_y() const { return ny > 1 ? face_len() * wz : 0; }  // values of one y-face
    __host__ __device__ int face_z() const { return face_len() * wy; }
    // Exchange buffer of a block: its first warps' faces, y then z.
    __host__ __device__ long long xch_block() const { return static_cast<long long>(bz) * face_y() + by * face_z(); }
};

template <class T>
struct LineTri {
    LineGeom g;
    const int* order = nullptr;  // [nblk] block (iy + nby iz, sweep coordinates) of each ticket;
                                 // with clusters [nby nbzc]: cluster (iy + nby izc) of each ticket
    const T* coef = nullptr;     // per slot c_z, c_y, c_x, and for U the reciprocal RN(1 / u_ii),
                                 // in the order of line_coef_at
    const T* div = nullptr;      // FP64 U: [slots] u_ii (line_quotient)
    T* xch = nullptr;            // [nblk][xch_block()] faces handed over through L2, at the sentinel
                                 // between launches (in x' in [0, nx))
    unsigned long long* tl = nullptr;  // per-block timeline [nblk][kLineTimeline] (null: off)
};

// Timeline record of one block (nanoseconds of %globaltimer): [0] compute start (faces
// reset, after the CTA barrier), [1] SM id, [2 + w] end of compute warp w (w < nw), [2 +
// nw] end of the halo warp; unused entries 0.
constexpr int kLineTimeline = 12;

__device__ __forceinline__ unsigned sm_id() {
    unsigned r;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
    return r;
}
template <class T>
__device__ __forceinline__ void line_stamp_start(const LineTri<T>& P, int blk) {
    if (P.tl != nullptr && threadIdx.x == 0) {
        unsigned long long* r = P.tl + static_cast<long long>(blk) * kLineTimeline;
        r[0] = global_ns();
        r[1] = sm_id();
    }
}
template <class T>
__device__ __forceinline__ void line_stamp_end(const LineTri<T>& P, int blk, int entry) {
    if (P.tl != nullptr && (threadIdx.x & 31) == 0)
        P.tl[static_cast<long long>(blk) * kLineTimeline + entry] = global_ns();
}

// Shared memory by its 32-bit address.
__device__ __forceinline__ unsigned shared_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void lds(unsigned a, float& v) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void lds(unsigned a, double& v) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); }
__device__ __forceinline__ void lds_polled(unsigned a, float& v) {
    asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ void lds_polled(unsigned a, double& v) {
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
__device__ __forceinline__ void lds16(unsigned a, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a));
}
__device__ __forceinline__ void lds16(unsigned a, double (&v)[2]) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a));
}
__device__ __forceinline__ void sts16(unsigned a, const float (&v)[4]) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
}
__device__ __forceinline__ void sts16(unsigned a, const double (&v)[2]) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]));
}
// Relaxed store through a generic address: the next warp's face (this CTA's shared
// memory), the next CTA's (distributed shared memory) or an exchange buffer (global).
__device__ __forceinline__ void st_relaxed_generic(bool on, double* p, double v) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %0, 0; @q st.relaxed.gpu.f64 [%1], %2; }" ::"r"(static_cast<unsigned>(on)), "l"(p), "d"(v));
}
__device__ __forceinline__ void st_relaxed_generic(bool on, float* p, float v) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %0, 0; @q st.relaxed.gpu.f32 [%1], %2; }" ::"r"(static_cast<unsigned>(on)), "l"(p), "f"(v));
}
// Generic address of `p` (this CTA's shared memory) in cluster CTA `rank`.
template <class T>
__device__ __forceinline__ T* map_generic_rank(T* p, unsigned rank) {
    unsigned long long r;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return reinterpret_cast<T*>(r);
}

// mbarriers between a compute warp and its helper (arrivals by lane 0 after a warp barrier).  Their arrivals release the warp's shared-memory writes without waiting for
// its global loads and stores in flight; a st.release flag did wait for them, which cost
// the compute warps a memory round trip per chunk.
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b))), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long* b) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b))) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b))) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(b))),
                 "r"(bytes)
                 : "memory");
}
// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) into this CTA's
// shared memory, completed on the mbarrier `b`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(bytes), "r"(static_cast<unsigned>(__cvta_generic_to_shared(b)))
                 : "memory");
}
// (test_wait, not try_wait: a warp that try_wait had suspended for about 100 us took 5 us
// to come back)
__device__ __forceinline__ bool mbar_test(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(static_cast<unsigned>(__cvta_generic_to_shared(b))), "r"(parity)
                 : "memory");
    return ok != 0u;
}
// Waits (bounded) for the completion of the barrier's phase of this parity; false when the
// wait gave up.  The clock is read as rarely as in line_wait_shared.
static __device__ __noinline__ bool mbar_wait_long(unsigned long long* b, unsigned parity, int* status) {
    WaitBudget wb;
    for (;;) {
        for (int polls = 0; polls < 2048; ++polls)
            if (mbar_test(b, parity)) return true;
        wb.polls |= 1023;  // so that expired() looks at the clock and at the status word
        if (wb.expired(status)) {
            atomicExch(status + kStatusTimeout, 1);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity, int* status) {
    return mbar_test(b, parity) || mbar_wait_long(b, parity, status);
}
// Waits for a bulk copy that has been issued to land: a block's barriers are initialised again, and
// its shared memory given back, only then, also when a wait elsewhere gave up.  A copy comes to
// its end whatever else happens; the bound is for form.
__device__ __forceinline__ void mbar_land(unsigned long long* b, unsigned parity) {
    for (int polls = 0; polls < (1 << 24) && !mbar_test(b, parity); ++polls) {
    }
}

// A value that may be stored where others poll for the sentinel: the sentinel's own bit
// pattern (a NaN) becomes the canonical NaN.  Integer compares: an FP64 compare would
// take 64 cycles of GB300's FP64 pipe in every step.
__device__ __forceinline__ float off_sentinel(float v) {
    return __float_as_uint(v) == 0xFFFFFFFFu ? __uint_as_float(0x7FC00000u) : v;
}
__device__ __forceinline__ double off_sentinel(double v) {
    return __double2hiint(v) == -1 ? __longlong_as_double(0x7FF8000000000000ll) : v;
}

// Waits (bounded) until the value at the shared address `a` is no longer the sentinel.
// The clock is read rarely, and not before kLinePollsFree polls (about 40 us): a read
// takes as long as several steps, and a warp never makes up for a delay, because its
// predecessor runs at the same pace (with a read every 64 polls each handoff between two
// warps cost 40 steps instead of 8).  After many polls it sleeps between polls (a block
// far behind).
constexpr int kLinePollsFree = 2048;
template <class T>
__device__ __noinline__ T line_wait_shared(unsigned a, int* status) {
    T v;
    for (int polls = 0; polls < kLinePollsFree; ++polls) {
        lds_polled(a, v);
        if (!Sentinel<T>::is(v)) return v;
    }
    WaitBudget wb;
    for (;;) {
        for (int polls = 0; polls < 1024; ++polls) {
            lds_polled(a, v);
            if (!Sentinel<T>::is(v)) return v;
        }
        wb.polls |= 1023;  // so that expired() looks at the clock and at the status word
        if (wb.expired(status)) {
            atomicExch(status + kStatusTimeout, 1);
            return T(0);
        }
    }
}

// Whether a face value has not arrived (lanes without a face hold zeros).
__device__ __forceinline__ bool line_late(float y, float z) { return max(__float_as_uint(y), __float_as_uint(z)) == 0xFFFFFFFFu; }
__device__ __forceinline__ bool line_late(double y, double z) {
    // (only the sentinel has these upper words: published values are off it)
    return max(static_cast<unsigned>(__double2hiint(y)), static_cast<unsigned>(__double2hiint(z))) == 0xFFFFFFFFu;
}

// Whether waiting warps keep their instructions warm (WARM, line_compute), chosen per grid,
// type (elem bytes) and sweep.  us, without / with:
// * 2-D: 1000^2 (blocks wait for 300 us and more) forward and backward FP32 214 / 156 and 195 /
//   139, FP64 392 / 267 and 694 / 405.  FP32 loses up to 600 lines (100 x 300 39 / 41 and 35 / 38,
//   500^2 79 / 83 and 70 / 77, 100 x 600 58 / 62 and 53 / 57) and gains from 800 (100 x 800 82 / 75 and
//   73 / 70, 800^2 130 / 127 and 115 / 118, 64 x 1500 171 / 117 and 167 / 110).
// * 3-D backward: FP32 40 x 40 x 500 353 / 129, 64 x 64 x 200 89 / 75, 128^3 85 / 85, 96^3 63 / 63;
//   FP64 96^3 143 / 128.
// * 3-D forward: FP32 gains from about 300 lines along y and z (60 x 100 x 200 146 / 96, 32 x 32 x
//   300 110 / 80, 24 x 24 x 1000 801 / 223; 160^3 and 200^3 lose, 126 / 131 and 193 / 200) and
//   loses below (128^3 87 / 90, 96^3 63 / 66, 64 x 64 x 200 70 / 75); FP64, whose blocks are
//   smaller, gains on narrow grids alone, where few blocks share an SM (20 x 20 x 300 265 / 117, 24
//   x 24 x 1000 645 / 399; 40 x 40 x 500 218 / 230, 128^3 128 / 135).
inline bool line_stays_warm(const LineGeom& g, int elem, bool upper) {
    if (g.ny == 1) return elem == 8 || g.nz > kLineWarmLines;
    if (upper) return true;
    return g.ny + g.nz > kLineWarmDepth && (elem == 4 || g.nby <= 2);
}
// Polls a warp's faces at its first step for about 20 us; whether all have arrived.
template <class T>
__device__ __forceinline__ bool line_first_faces(unsigned fy, unsigned fz) {
    for (int i = 0; i < 640; ++i) {
        T y, z;
        lds_polled(fy, y);
        lds_polled(fz, z);
        if (!__any_sync(0xffffffffu, line_late(y, z))) return true;
    }
    return false;
}

// Bound of a warp's wait made of many polls at a time: the clock is read every 16th time.  All
// lanes call it together and get one answer, whatever time each of them reads: shuffles and
// votes of the whole warp follow.
struct LineWait {
    WaitBudget wb;
    int calls = 0;
    __device__ __forceinline__ bool expired(int* status) {
        if ((++calls & 15) != 0) return false;
        return __any_sync(0xffffffffu, slow(status));
    }
    __device__ __noinline__ bool slow(int* status) {
        wb.polls |= 1023;  // so that expired() looks at the clock and at the status word
        const bool out = wb.expired(status);
        if (out) atomicExch(status + kStatusTimeout, 1);
        return out;
    }
};

// Coefficients of one row in the packed stream: c_z, c_y, c_x and for U the reciprocal.  A
// step's 32 rows lie together: FP32 four values (16 bytes) per lane; FP64 pairs (c_z, c_y)
// per lane, then for U pairs (c_x, reciprocal), for L c_x alone.
template <class T>
struct LineCoef {
    T cz, cy, cx, d;
};
template <class T, bool UPPER>
__host__ __device__ constexpr int line_step_values() {
    return sizeof(T) == 8 && !UPPER ? 96 : 128;
}
template <class T, bool UPPER>
__host__ __device__ constexpr long long line_coef_at(long long slot, int e) {
    const long long step = (slot / 32) * line_step_values<T, UPPER>();
    const int lane = static_cast<int>(slot % 32);
    if (sizeof(T) == 4) return step + lane * 4 + e;
    if (e < 2) return step + lane * 2 + e;
    return step + 64 + (UPPER ? lane * 2 + (e - 2) : lane);
}
// (a: shared address of the step)
template <bool UPPER>
__device__ __forceinline__ void line_load_coef(unsigned a, int lane, LineCoef<float>& c) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(c.cz), "=f"(c.cy), "=f"(c.cx), "=f"(c.d) : "r"(a + lane * 16));
}
template <bool UPPER>
__device__ __forceinline__ void line_load_coef(unsigned a, int lane, LineCoef<double>& c) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(c.cz), "=d"(c.cy) : "r"(a + lane * 16));
    if constexpr (UPPER)
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(c.cx), "=d"(c.d) : "r"(a + lane * 16 + 512));
    else
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(c.cx) : "r"(a + lane * 8 + 512));
}

// Shared memory of a CTA: per compute warp and slot a chunk of the coefficient stream
// (and for FP64 of the divisors) and its right-hand side [lane][kLinePitch]; per
// compute warp a ring of kLineSlots + 1 chunks of results [lane][kLinePitch]; then the faces (consumer-indexed: slot w holds what warp w reads;
// y-faces [nw][face_y()], z-faces [nw][face_z()]); then kLineIdle zeros that lanes without
// a face read (so that no load needs a predicate) and kLineIdle values, the address of lanes
// without a consumer, whose stores are predicated off; then per compute warp and slot two mbarriers: [0] the chunk is staged (and the result ring has room for it), [1] the
// chunk is computed.
template <class T, bool UPPER>
struct LineStage {
    static constexpr int kCoef = kLineChunk * line_step_values<T, UPPER>();
    static constexpr int kDiv = UPPER && sizeof(T) == 8 ? kLineChunk * 32 : 0;
    static constexpr int kVec = 32 * kLinePitch<T>;
    static constexpr int kSlot = kCoef + kDiv + kVec;  // a multiple of 16 bytes
    static constexpr int kWarp = kLineSlots * kSlot + (kLineSlots + 1) * kVec;
};
constexpr int kLineIdle = kLineStepAlign * 32 + 32;  // offsets within a chunk stay inside
template <class T, bool UPPER>
__host__ __device__ inline long long line_bar_offset(const LineGeom& g) {
    return (((g.nw() * (static_cast<long long>(LineStage<T, UPPER>::kWarp) + g.face_y() + g.face_z()) + 2 * kLineIdle) *
             static_cast<long long>(sizeof(T))) + 15) & ~15ll;
}
template <class T, bool UPPER>
__host__ __device__ inline long long line_smem_bytes(const LineGeom& g) {
    return line_bar_offset<T, UPPER>(g) + 2ll * g.nw() * kLineSlots * static_cast<long long>(sizeof(unsigned long long));
}

template <class T, bool UPPER>
struct LineSmem {
    T *stage, *face_y, *face_z, *idle;
    unsigned long long* bar;
    __device__ __forceinline__ T* slot(int w, int k) const {
        return stage + w * LineStage<T, UPPER>::kWarp + (k % kLineSlots) * LineStage<T, UPPER>::kSlot;
    }
    __device__ __forceinline__ T* result(int w, int k) const {
        return stage + w * LineStage<T, UPPER>::kWarp + kLineSlots * LineStage<T, UPPER>::kSlot +
               (k % (kLineSlots + 1)) * LineStage<T, UPPER>::kVec;
    }
    __device__ __forceinline__ unsigned long long* full(int w, int k) const {
        return bar + w * 2 * kLineSlots + k % kLineSlots;
    }
    __device__ __forceinline__ unsigned long long* done(int w, int k) const { return full(w, k) + kLineSlots; }
    static __device__ __forceinline__ unsigned parity(int k) { return (k / kLineSlots) & 1; }
};
template <class T, bool UPPER>
__device__ __forceinline__ LineSmem<T, UPPER> line_smem_view(const LineGeom& g, unsigned char* base) {
    LineSmem<T, UPPER> m;
    m.stage = reinterpret_cast<T*>(base);
    m.face_y = m.stage + static_cast<long long>(g.nw()) * LineStage<T, UPPER>::kWarp;
    m.face_z = m.face_y + static_cast<long long>(g.nw()) * g.face_y();
    m.idle = m.face_z + static_cast<long long>(g.nw()) * g.face_z();
    m.bar = reinterpret_cast<unsigned long long*>(base + line_bar_offset<T, UPPER>(g));
    return m;
}

// One compute warp's share of block `blk`: wy x wz lines over psteps steps.  Slots without
// a row hold zero coefficients and a zero right-hand side, so a lane outside its line
// computes zeros (or, past the line's end, values that nobody reads) and needs no
// predicate.  to_y / to_z: the face (generic address, this warp's lane pattern) that its
// last lanes along y / z fill, null: none.
//
// False (WARM) when the first faces have not arrived: then only the first chunk was
// run, on the idle area, and the caller tries again.  A warp that only polls for about 50 us
// finds the instructions of its steps gone from the cache, and its first chunk took 8 us.
template <class T, bool UPPER, int WY, bool D3, bool WARM>
__device__ __forceinline__ bool line_compute(const LineTri<T>& P, int blk, int w, const LineSmem<T, UPPER>& M, T* to_y, T* to_z,
                                             LineWait& wait, int* status) {
    constexpr int WZ = 32 / WY;
    constexpr int PAD = WY + WZ - 2;
    constexpr int C = kLineChunk;
    using St = LineStage<T, UPPER>;
    constexpr bool DIV = UPPER && sizeof(T) == 8;
    const int lane = threadIdx.x & 31;
    const int yy = lane % WY, zz = lane / WY;
    const int shift = PAD - (yy + zz);  // face position of step 0
    const bool y_edge = D3 && yy == 0;
    const bool z_edge = zz == 0;
    constexpr unsigned Z = sizeof(T);
    const unsigned idle = shared_addr(M.idle);
    unsigned fy = y_edge ? shared_addr(M.face_y + static_cast<long long>(w) * P.g.face_y() + shift * WZ + zz) : idle;
    unsigned fz = z_edge ? shared_addr(M.face_z + static_cast<long long>(w) * P.g.face_z() + shift * WY + yy) : idle;
    const bool dry = WARM && !line_first_faces<T>(fy, fz) && !wait.expired(status);
    if (dry) fy = fz = idle;
    const unsigned fy_adv = y_edge ? C * WZ * Z : 0u, fz_adv = z_edge ? C * WY * Z : 0u;
    const bool has_y = !dry && D3 && to_y != nullptr && yy == WY - 1;
    const bool has_z = !dry && to_z != nullptr && zz == WZ - 1;
    T* oy = has_y ? to_y + shift * WZ + zz : M.idle + kLineIdle;
    T* oz = has_z ? to_z + shift * WY + yy : M.idle + kLineIdle;
    const int oy_adv = has_y ? C * WZ : 0, oz_adv = has_z ? C * WY : 0;
    const int nchunk = dry ? 1 : P.g.psteps / C;

    mbar_wait(M.full(w, 0), 0u, status);
    __syncwarp();
    constexpr int V = 16 / sizeof(T);  // steps per access of the right-hand side and the results
    constexpr unsigned kDiv = St::kCoef * Z, kB = kDiv + St::kDiv * Z, kStep = line_step_values<T, UPPER>() * Z;
    const unsigned laneZ = lane * Z, laneP = lane * (kLinePitch<T> * Z);
    unsigned row = shared_addr(M.slot(w, 0));
    // operands: coefficients loaded two steps ahead, right-hand side by groups of V steps,
    // faces one step ahead
    LineCoef<T> c[2];
    T d[2] = {T(0), T(0)}, bc[V], bn[V], res[V];
    T pfy = T(0), pfz;
    auto load = [&](unsigned slot, int step, int e) {
        line_load_coef<UPPER>(slot + step * kStep, lane, c[e]);
        if constexpr (DIV) lds(slot + laneZ + (kDiv + step * 32 * Z), d[e]);
    };
    load(row, 0, 0);
    load(row, 1, 1);
    lds16(row + laneP + kB, bc);
    if (D3) lds_polled(fy, pfy);
    lds_polled(fz, pfz);
    T prev = T(0), sh_y = T(0), sh_z = T(0);  // the previous step's results: own, y- and z-neighbour
    auto shuffle = [&](T r, T& y, T& z) {
        if (D3 && WY > 1) y = __shfl_up_sync(0xffffffffu, r, 1);
        z = __shfl_up_sync(0xffffffffu, r, WY);
    };
#pragma unroll 1
    for (int k = 0; k < nchunk; ++k) {
        unsigned next = row;
        const unsigned out = shared_addr(M.result(w, k)) + laneP;
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const LineCoef<T> q = c[i % 2];
            const T qd = d[i % 2], a0 = bc[i % V];
            const T fyv = pfy, fzv = pfz;
            // the row, as if every predecessor were there and the quotient final
            T acc;
            auto solve = [&](T fy_v, T fz_v) -> T {
                acc = fma(-q.cz, z_edge ? fz_v : sh_z, a0);
                if (D3) acc = fma(-q.cy, y_edge ? fy_v : sh_y, acc);
                acc = fma(-q.cx, prev, acc);
                if constexpr (DIV) return line_quotient(acc, qd, q.d);  // the reference's division
                if constexpr (UPPER) return acc * q.d;
                return acc;
            };
            T r = solve(fyv, fzv);
            T ny = T(0), nz;
            shuffle(r, ny, nz);
            if (i == C - 2 && k + 1 < nchunk) {
                mbar_wait(M.full(w, k + 1), M.parity(k + 1), status);
                __syncwarp();
                next = shared_addr(M.slot(w, k + 1));
            }
            if (D3) lds_polled(fy + (i + 1) * WZ * Z, pfy);
            lds_polled(fz + (i + 1) * WY * Z, pfz);
            // (after the last step values that nothing uses)
            load(i + 2 < C ? row : next, (i + 2) % C, i % 2);
            if (i % V == V - 2) lds16((i + 2 < C ? row : next) + laneP + (kB + (i + 2) % C * Z), bn);
            // otherwise: wait for the faces, divide again
            if (__any_sync(0xffffffffu, line_late(fyv, fzv) || (DIV && line_quotient_bad(r, acc)))) {
                T fy_v = fyv, fz_v = fzv;
                if (D3 && Sentinel<T>::is(fyv)) fy_v = line_wait_shared<T>(fy + i * WZ * Z, status);
                if (Sentinel<T>::is(fzv)) fz_v = line_wait_shared<T>(fz + i * WY * Z, status);
                __syncwarp();
                r = solve(fy_v, fz_v);
                if constexpr (DIV) {
                    if (line_quotient_bad(r, acc)) r = line_divide(acc, qd);
                    __syncwarp();
                }
                shuffle(r, ny, nz);
            }
            prev = r;
            sh_y = ny;
            sh_z = nz;
            // only the stored copies, which others poll, are kept off the sentinel
            const T rs = off_sentinel(r);
            if (D3) st_relaxed_generic(has_y, oy + i * WZ, rs);
            st_relaxed_generic(has_z, oz + i * WY, rs);
            res[i % V] = rs;
            if (i % V == V - 1) {
                sts16(out + (i - (V - 1)) * Z, res);
#pragma unroll
                for (int e = 0; e < V; ++e) bc[e] = bn[e];
            }
        }
        __syncwarp();
        if (lane == 0 && !dry) mbar_arrive(M.done(w, k));
        row = next;
        fy += fy_adv;
        fz += fz_adv;
        oy += oy_adv;
        oz += oz_adv;
    }
    return !dry;
}

// The helper of compute warp w: stages the operands chunk by chunk (the coefficients by
// bulk copies; the right-hand side times `sc`, and written back so, when GMRES normalises
// its new Krylov vector in the forward sweep) and writes the results out.  Its lanes take
// kLineChunk consecutive rows of 32 / kLineChunk lines at a time.
template <class T, bool UPPER>
__device__ __forceinline__ void line_helper(const LineTri<T>& P, int blk, int w, const LineSmem<T, UPPER>& M, T* in, bool scaled,
                                            T sc, T* out, int* status) {
    constexpr int C = kLineChunk;
    constexpr int S = kLineSlots;
    constexpr int Q = 32 / C;  // lines per access
    using St = LineStage<T, UPPER>;
    const int lane = threadIdx.x & 31;
    const int i = lane % C, q = lane / C;
    const int nx = P.g.nx, ny = P.g.ny, nz = P.g.nz;
    const int wyi = w % P.g.by, wzi = w / P.g.by;
    const int iy = blk % P.g.nby, iz = blk / P.g.nby;
    constexpr int sx = UPPER ? -1 : 1;
    int x0[C], row0[C];  // x' and row of this lane's value of chunk 0 on line Q r + q
#pragma unroll
    for (int r = 0; r < C; ++r) {
        const int l = Q * r + q;
        const int yy = l % P.g.wy, zz = l / P.g.wy;
        const int yq = (iy * P.g.by + wyi) * P.g.wy + yy;
        const int zq = (iz * P.g.bz + wzi) * P.g.wz + zz;
        const bool ok = yq < ny && zq < nz;
        const int Y = UPPER ? ny - 1 - yq : yq;
        const int Z = UPPER ? nz - 1 - zq : zq;
        const int x = i - (yy + zz);
        x0[r] = ok ? x : -(1 << 30);
        row0[r] = ok ? static_cast<int>((UPPER ? nx - 1 : 0) + sx * x + static_cast<long long>(nx) * (Y + static_cast<long long>(ny) * Z)) : 0;
    }
    const int nchunk = P.g.psteps / C;
    const long long first = P.g.slot(blk, w, 0, 0);
    auto valid = [&](int r, int k) { return static_cast<unsigned>(x0[r] + C * k) < static_cast<unsigned>(nx); };
    auto fetch = [&](int k, T (&v)[C]) {
#pragma unroll
        for (int r = 0; r < C; ++r) v[r] = valid(r, k) ? in[row0[r] + sx * C * k] : T(0);
    };
    auto flush = [&](int k) {
        const T* const o = M.result(w, k) + q * kLinePitch<T> + i;
#pragma unroll
        for (int r = 0; r < C; ++r)
            if (valid(r, k)) out[row0[r] + sx * C * k] = o[Q * r * kLinePitch<T>];
    };
    // chunk k, its right-hand side in v; v is left with that of chunk k + 2.  False when the
    // slot's previous chunk is not computed in time: then nothing more is staged, and the
    // compute warp's waits give up as well.
    auto stage = [&](int k, T (&v)[C]) -> bool {
        if (k >= S && !__all_sync(0xffffffffu, mbar_wait(M.done(w, k - S), M.parity(k - S), status))) return false;
        T* const slot = M.slot(w, k);
        unsigned long long* const full = M.full(w, k);
        if (lane == 0) {
            constexpr unsigned cb = St::kCoef * sizeof(T);
            constexpr unsigned db = St::kDiv * sizeof(T);
            mbar_arrive_expect(full, cb + db);
            bulk_load(slot, P.coef + line_coef_at<T, UPPER>(first + static_cast<long long>(k) * C * 32, 0), cb, full);
            if (db > 0) bulk_load(slot + St::kCoef, P.div + first + static_cast<long long>(k) * C * 32, db, full);
        }
        T* const b = slot + St::kCoef + St::kDiv + q * kLinePitch<T> + i;
#pragma unroll
        for (int r = 0; r < C; ++r) {
            if (scaled) v[r] = v[r] * sc;
            b[Q * r * kLinePitch<T>] = v[r];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(full);
        if (scaled) {
#pragma unroll
            for (int r = 0; r < C; ++r)
                if (valid(r, k)) in[row0[r] + sx * C * k] = v[r];
        }
        if (k + 2 < nchunk) fetch(k + 2, v);
        if (k >= S) flush(k - S);
        return true;
    };
    // right-hand sides are loaded two chunks ahead: a chunk's loads take as long as the
    // rest of the work on a chunk
    T va[C], vb[C];
    fetch(0, va);
    if (nchunk > 1) fetch(1, vb);
    int staged = 0;
    while (staged < nchunk && stage(staged, va) && ++staged < nchunk && stage(staged, vb)) ++staged;
    for (int k = max(0, staged - S); k < staged; ++k) {
        mbar_wait(M.done(w, k), M.parity(k), status);
        __syncwarp();
        flush(k);
        mbar_land(M.full(w, k), M.parity(k));
    }
    __syncwarp();
}

// A halo warp of block `blk`: copies faces that the previous block hands over through its
// exchange buffer into shared memory as they arrive, and puts the buffer back to the
// sentinel.  Lane e owns line e of the face (at most 32: `width` lines in each of the
// `nslot` warps' faces, a warp's face being `face` values, and face slots `stride` warps
// apart) and walks it in x' with its own cursor; a round loads the next kLineHalo
// positions (one L2 round trip) and retires, in order, those that have arrived.
constexpr int kLineHalo = 8;

template <class T>
__device__ __forceinline__ void line_halo(T* xch, T* faces, int face, int stride, int nslot, int width, int pad, int nx,
                                          int* status) {
    const int lane = threadIdx.x & 31;
    const int slot = lane / width;
    const bool on = slot < nslot;
    T* const src = xch + static_cast<long long>(on ? slot : 0) * face + pad * width + lane % width;
    T* const dst = faces + static_cast<long long>(on ? slot : 0) * stride * face + pad * width + lane % width;
    int x = on ? 0 : nx;
    bool idle = true;  // nothing arrived in the last round: poll one position per lane only
    WaitBudget wb;
    while (__any_sync(0xffffffffu, x < nx)) {
        T v[kLineHalo];
#pragma unroll
        for (int u = 0; u < kLineHalo; ++u)
            v[u] = x + u < nx && (u == 0 || !idle) ? ld_relaxed_nb(src + (x + u) * width) : Sentinel<T>::value();
        int adv = 0;
        bool stop = false;
#pragma unroll
        for (int u = 0; u < kLineHalo; ++u) {
            stop = stop || Sentinel<T>::is(v[u]);
            if (!stop) {
                st_volatile_shared(dst + (x + u) * width, v[u]);
                src[(x + u) * width] = Sentinel<T>::value();
                ++adv;
            }
        }
        x += adv;
        idle = !__any_sync(0xffffffffu, adv > 0);
        if (!idle) {
            wb = WaitBudget();
        } else if (wb.expired(status)) {
            atomicExch(status + kStatusTimeout, 1);
            // unblock the compute warps: the remaining entries become 0
            for (; x < nx; ++x) st_volatile_shared(dst + x * width, T(0));
        }
    }
}

// Resets a block's faces, each warp whole faces: the sentinel where a value will be
// written (x' in [0, nx)), 0 elsewhere and in the faces of lines at the grid's boundary;
// and the mbarriers (`again`: they were used before).
template <class T, bool UPPER>
__device__ __forceinline__ void line_reset(const LineGeom& g, int iy, int iz, const LineSmem<T, UPPER>& M, bool again) {
    const int lane = threadIdx.x & 31;
    const int nwarp = static_cast<int>(blockDim.x >> 5);
    const int nw = g.nw();
    for (int f = static_cast<int>(threadIdx.x >> 5); f < (g.ny > 1 ? 2 * nw : nw); f += nwarp) {
        const bool z = f < nw;
        const int w = z ? f : f - nw;
        const int width = z ? g.wy : g.wz;
        const int len = z ? g.face_z() : g.face_y();
        T* const p = (z ? M.face_z : M.face_y) + static_cast<long long>(w) * len;
        const bool zero = z ? (iz == 0 && w / g.by == 0) : (iy == 0 && w % g.by == 0);
        const int lo = zero ? len : g.pad() * width, hi = (g.pad() + g.nx) * width;
        for (int j = lane; j < len; j += 32) p[j] = j >= lo && j < hi ? Sentinel<T>::value() : T(0);
    }
    constexpr int S = kLineSlots;
    for (int j = threadIdx.x; j < kLineIdle; j += blockDim.x) M.idle[j] = T(0);
    for (int j = threadIdx.x; j < 2 * nw * S; j += blockDim.x) {
        if (again) mbar_inval(M.bar + j);
        mbar_init(M.bar + j, j % (2 * S) < S ? 2 : 1);  // staged: bulk copies and right-hand side
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");  // (before the bulk copies use them)
}

// Block `blk` by this CTA (faces reset, all threads past a barrier).  next_z: the faceZ of
// the next CTA along z in distributed shared memory (null: through L2); z_from_l2: this
// CTA's first warps along z take their predecessors from the exchange buffer.
template <class T, bool UPPER, int WY, bool D3, bool WARM>
__device__ __forceinline__ void line_block(const LineTri<T>& P, int blk, const LineSmem<T, UPPER>& M, T* in, bool scaled, T sc,
                                           T* out, T* next_z, bool z_from_l2, int* status) {
    const LineGeom& g = P.g;
    const int nw = g.nw();
    const int w = threadIdx.x >> 5;
    const int iy = blk % g.nby, iz = blk / g.nby;
    line_stamp_start(P, blk);
    if (w < nw) {
        LineWait wait;
        for (bool done = false; !done;) {
            // (addresses are worked out anew rather than held in registers through the steps)
            int b = blk, cw = w;
            if (WARM) asm volatile("" : "+r"(b), "+r"(cw));
            const int by = b % g.nby, bz = b / g.nby;
            const int wyi = cw % g.by, wzi = cw / g.by;
            T* to_y = nullptr;
            T* to_z = nullptr;
            if (D3) {
                if (wyi + 1 < g.by)
                    to_y = M.face_y + static_cast<long long>(cw + 1) * g.face_y();
                else if (by + 1 < g.nby)
                    to_y = P.xch + (b + 1) * g.xch_block() + static_cast<long long>(wzi) * g.face_y();
            }
            if (wzi + 1 < g.bz)
                to_z = M.face_z + static_cast<long long>(cw + g.by) * g.face_z();
            else if (next_z != nullptr)
                to_z = next_z + static_cast<long long>(wyi) * g.face_z();
            else if (bz + 1 < g.nbz)
                to_z = P.xch + (b + g.nby) * g.xch_block() + static_cast<long long>(g.bz) * g.face_y() +
                       static_cast<long long>(wyi) * g.face_z();
            done = line_compute<T, UPPER, WY, D3, WARM>(P, b, cw, M, to_y, to_z, wait, status);
        }
        line_stamp_end(P, blk, 2 + w);
    } else if (w < 2 * nw) {
        line_helper<T, UPPER>(P, blk, w - nw, M, in, scaled, sc, out, status);
    } else if (w == 2 * nw) {
        T* const x = P.xch + blk * g.xch_block() + static_cast<long long>(g.bz) * g.face_y();
        if (iz > 0 && z_from_l2) line_halo(x, M.face_z, g.face_z(), 1, g.by, WY, g.pad(), g.nx, status);
        line_stamp_end(P, blk, 2 + nw);
    } else if (D3) {
        T* const x = P.xch + blk * g.xch_block();
        if (iy > 0) line_halo(x, M.face_y, g.face_y(), g.by, g.bz, 32 / WY, g.pad(), g.nx, status);
    }
}

// Streams the block's operands into L2 (they come from HBM: the Krylov vectors evict them
// between sweeps).
template <class T, bool UPPER>
__device__ __forceinline__ void line_prefetch(const LineTri<T>& P, int blk) {
    const int w = threadIdx.x >> 5;
    if (w >= P.g.nw()) return;
    const long long s0 = P.g.slot(blk, w, 0, 0);
    const long long n = static_cast<long long>(P.g.psteps) * static_cast<long long>(sizeof(T));
    prefetch_l2_range(P.coef + line_coef_at<T, UPPER>(s0, 0), n * line_step_values<T, UPPER>(), threadIdx.x & 31);
    if (UPPER && sizeof(T) == 8) prefetch_l2_range(P.div + s0, n * 32, threadIdx.x & 31);
}

// Forward (UPPER = false): out = L^{-1} (scale * in), in rescaled in place when `scale`
// is given; backward (UPPER = true): out = U^{-1} in.  in / out in natural order; what out
// holds on entry does not matter.  g.threads() threads: compute warps, their helpers, halo
// warps; dynamic shared memory line_smem_bytes.
template <class T, bool UPPER, int WY, bool D3, bool WARM>
__global__ void __launch_bounds__((2 * kLineMaxWarps + 2) * kWarp, sizeof(T) == 4 ? 2 : 1)
    sptrsv_line_kernel(LineTri<T> P, T* in, const double* scale, T* out, unsigned* counter, int* status,
                       const int* gate, int step) {
    if (gate_closed(gate, step)) return;
    extern __shared__ __align__(16) unsigned char line_smem[];
    const LineSmem<T, UPPER> M = line_smem_view<T, UPPER>(P.g, line_smem);
    __shared__ int s_ticket;
    const bool scaled = !UPPER && scale != nullptr;
    const T sc = scaled ? static_cast<T>(*scale) : T(1);
    bool again = false;
    for (int tk = draw_block_ticket(counter, P.g.nblk, &s_ticket); tk < P.g.nblk;
         tk = draw_block_ticket(counter, P.g.nblk, &s_ticket)) {
        const int blk = P.order[tk];
        line_reset<T, UPPER>(P.g, blk % P.g.nby, blk / P.g.nby, M, again);
        again = true;
        line_prefetch<T, UPPER>(P, blk);
        __syncthreads();
        line_block<T, UPPER, WY, D3, WARM>(P, blk, M, in, scaled, sc, out, nullptr, true, status);
    }
}

// Cluster variant: launched with clusters of g.cl CTAs; the cluster of ticket q takes the
// blocks (iy, izc cl + rank) of cluster q (tickets along anti-diagonals of the cluster
// grid: a cluster only waits for clusters of smaller tickets, whose CTAs are running or
// done; the CTAs of one cluster are co-scheduled).  A CTA's last warps along z push
// their results into the next CTA's face in distributed shared memory, so only the first
// CTA of a cluster and the y-direction take their predecessors from L2 (halo warps).
template <class T, bool UPPER, int WY, bool D3, bool WARM>
__global__ void __launch_bounds__((2 * kLineMaxWarps + 2) * kWarp, sizeof(T) == 4 ? 2 : 1)
    sptrsv_line_cluster_kernel(LineTri<T> P, T* in, const double* scale, T* out, unsigned* counter, int* status,
                               const int* gate, int step) {
    if (gate_closed(gate, step)) return;
    extern __shared__ __align__(16) unsigned char line_smem[];
    const LineSmem<T, UPPER> M = line_smem_view<T, UPPER>(P.g, line_smem);
    __shared__ int s_ticket;
    const bool scaled = !UPPER && scale != nullptr;
    const T sc = scaled ? static_cast<T>(*scale) : T(1);
    const unsigned rank = cluster_rank_u32();
    const unsigned CL = cluster_size_u32();
    const int nq = P.g.nby * P.g.nbzc;
    const int nclusters = static_cast<int>(gridDim.x / CL);
    bool again = false;
    for (;;) {
        // the previous round is complete in every CTA of the cluster (no push in flight)
        // before the ticket and the faces are reset
        cluster_sync_all();
        if (rank == 0 && threadIdx.x == 0) {
            const int q = static_cast<int>(atomicAdd(counter, 1u));
            if (q == nq + nclusters - 1) atomicExch(counter, 0u);
            for (unsigned r = 0; r < CL; ++r) st_cluster(map_shared_rank(&s_ticket, r), q);
        }
        cluster_sync_all();
        const int q = *reinterpret_cast<volatile int*>(&s_ticket);
        if (q >= nq) break;
        const int cb = P.order[q];
        const int iy = cb % P.g.nby;
        const int iz = (cb / P.g.nby) * static_cast<int>(CL) + static_cast<int>(rank);
        const bool active = iz < P.g.nbz;
        const int blk = iy + P.g.nby * iz;
        if (active) {
            line_reset<T, UPPER>(P.g, iy, iz, M, again);
            again = true;
            line_prefetch<T, UPPER>(P, blk);
            }
        __syncthreads();
        // every face of the cluster is reset before any CTA pushes into it
        cluster_sync_all();
        if (active) {
            const bool push = rank + 1 < CL && iz + 1 < P.g.nbz;
            T* const next = push ? map_generic_rank(M.face_z, rank + 1) : nullptr;
            line_block<T, UPPER, WY, D3, WARM>(P, blk, M, in, scaled, sc, out, next, rank == 0, status);
        }
        __syncthreads();
    }
}

// Packs the operand stream of a structured factor from its CSR values: one thread per
// slot.  L: c_z, c_y, c_x are the row's strict-lower entries (columns ascending:
// r - nx ny, r - nx, r - 1, each present only inside the grid).  U: c_z, c_y, c_x are the
// strict-upper entries r + nx ny, r + nx, r + 1 (columns descending) and the reciprocal of
// u_ii: FP32 RN(1 / u_ii), computed in FP64 and rounded once (as the other FP32 kernels);
// FP64 line_reciprocal, and u_ii itself.  Slots without a row hold zeros.
template <class T, bool UPPER>
__global__ void line_pack_kernel(LineGeom g, const int* __restrict__ rp, const int* __restrict__ diag,
                                 const double* __restrict__ lu, T* __restrict__ dst, T* __restrict__ div) {
    const long long total = g.slots();
    const int nw = g.nw();
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int lane = static_cast<int>(i & 31);
        long long t = i >> 5;
        const int s = static_cast<int>(t % g.psteps);
        t /= g.psteps;
        const int w = static_cast<int>(t % nw);
        const int b = static_cast<int>(t / nw);
        const int wyi = w % g.by, wzi = w / g.by;
        const int yy = lane % g.wy, zz = lane / g.wy;
        const int iy = b % g.nby, iz = b / g.nby;
        const int yq = (iy * g.by + wyi) * g.wy + yy;
        const int zq = (iz * g.bz + wzi) * g.wz + zz;
        const int xq = s - (yy + zz);
        double cz = 0.0, cy = 0.0, cx = 0.0, d = 0.0, u = 0.0;
        if (yq < g.ny && zq < g.nz && xq >= 0 && xq < g.nx) {
            const int X = UPPER ? g.nx - 1 - xq : xq;
            const int Y = UPPER ? g.ny - 1 - yq : yq;
            const int Z = UPPER ? g.nz - 1 - zq : zq;
            const long long r = X + static_cast<long long>(g.nx) * (Y + static_cast<long long>(g.ny) * Z);
            if constexpr (!UPPER) {
                int p = rp[r];
                if (Z > 0) cz = lu[p++];
                if (Y > 0) cy = lu[p++];
                if (X > 0) cx = lu[p++];
            } else {
                int p = diag[r];
                u = lu[p++];
                if (X < g.nx - 1) cx = lu[p++];
                if (Y < g.ny - 1) cy = lu[p++];
                if (Z < g.nz - 1) cz = lu[p++];
                d = sizeof(T) == 4 ? 1.0 / u : line_reciprocal(u);
            }
        }
        dst[line_coef_at<T, UPPER>(i, 0)] = static_cast<T>(cz);
        dst[line_coef_at<T, UPPER>(i, 1)] = static_cast<T>(cy);
        dst[line_coef_at<T, UPPER>(i, 2)] = static_cast<T>(cx);
        if constexpr (UPPER || sizeof(T) == 4) dst[line_coef_at<T, UPPER>(i, 3)] = static_cast<T>(d);
        if constexpr (UPPER && sizeof(T) == 8) div[i] = u;
    }
}

template <class T>
__global__ void line_fill_kernel(long long n, T* p, T v) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        p[i] = v;
}

}  // namespace gb300
