// ILU(0) of a full 7- / 5-point stencil in natural order: the line pipeline of
// line_sweep.cuh applied to the factorisation.
//
// On such a grid (nx >= 3, and ny >= 3 in 3-D) the row elimination of
// src/ilu_solver.cpp:553-589 changes the diagonal only: no pivot row's strict-upper part
// meets row i anywhere but at i itself, so
//     l_ij = a_ij / d_j,   d_i = ((a_ii - l_iz a_zi) - l_iy a_yi) - l_ix a_xi
// over the lower neighbours z, y, x in ascending column order (the reference's order, an
// FMA each as ilu_factor_kernel) and the strict-upper entries stay those of A.  That is the
// forward sweep's dependency structure, and the kernel is laid out like it: a lane per grid
// line, skewed lanes, faces between warps and blocks, helper warps that stage the operands
// by bulk copies.
//
// What bounds it: the FP64 instructions of a row on one scheduler (64 cycles each, whatever
// the lanes).  A division takes nine; here a row computes the reciprocal of its own pivot once
// (four, line_pivot_reciprocal) and hands it on with the pivot, so each of the quotients takes
// three (line_quotient) and a 3-D row 16 instructions, 1024 cycles, of which eight lie on the
// chain along x.  The results are written to the operand stream, coalesced
// (a lane's rows lie a line apart in the CSR values: 32 sectors per entry), and a second
// kernel takes them to the CSR values.  The warp-per-row kernel pays an L2 handoff and a
// division chain per level.  Whole factorisations (packs of the sweeps included), ms, before
// (warp per row) and now: 128^3 4.6 / 0.79, 101 x 90 x 75 2.4 / 0.36, 200^3 14.5 / 2.3, 384 x
// 301 4.2 / 0.47, 1024^2 13.0 / 1.4, 32^2 0.35 / 0.07; a step takes 0.58 us.  A CTA of one warp
// fits in shared memory up to nx = 910 in 3-D (its faces hold 192 B per cell along x, its
// stages 48 KB) and nx = 11,000 in 2-D; longer lines are factorised by the warp-per-row kernel
// (900 x 12 x 12 0.82 ms, 950 x 12 x 12 3.8 ms).
#pragma once

#include "line_sweep.cuh"

namespace gb300 {

constexpr int kLineFactorWarps = 2;  // compute warps per CTA
constexpr int kLineFactorRow = 8;    // staged values per row: a_ii, a_iz, a_iy, a_ix, a_zi, a_yi, a_xi, unused;
                                     // on return d_i, l_iz, l_iy, l_ix
constexpr int kLinePivotParts = 2;   // values handed on per row: the pivot and its reciprocal
constexpr int kLineFactorSlots = 3;
constexpr int kLineFactorPolls = 16;  // (about 1 us)

struct LineFactor {
    LineGeom g;
    const int* order = nullptr;      // blocks (clusters) by ticket, as LineTri
    double* rows = nullptr;          // operand stream, line_factor_at
    double* xch = nullptr;           // [nblk][kLinePivotParts][xch_block()]
};

// Value e of a slot in the operand stream: a step's 32 rows lie together, four 16-byte parts
// per lane.
__host__ __device__ constexpr long long line_factor_at(long long slot, int e) {
    return (slot / 32) * (32 * kLineFactorRow) + (e / 2) * 64 + (slot % 32) * 2 + e % 2;
}

struct LinePivot {
    double d, z;  // z: its reciprocal
};

__device__ __forceinline__ bool line_late(const LinePivot& y, const LinePivot& z) {
    return line_late(y.d, z.d) || line_late(y.z, z.z);
}

// Shared memory: per compute warp the staged rows; the faces of every warp; the
// idle area; mbarriers (staged, computed) per warp and slot.
__host__ __device__ inline long long line_factor_stage() {
    return static_cast<long long>(kLineFactorSlots) * kLineChunk * 32 * kLineFactorRow;
}
__host__ __device__ inline long long line_factor_bar_offset(const LineGeom& g) {
    return (((g.nw() * (line_factor_stage() + kLinePivotParts * (g.face_y() + g.face_z())) + kLineIdle) * 8) + 15) & ~15ll;
}
__host__ __device__ inline long long line_factor_smem_bytes(const LineGeom& g) {
    return line_factor_bar_offset(g) + 2ll * g.nw() * kLineFactorSlots * 8;
}
struct LineFactorSmem {
    double *stage, *face_y, *face_z, *idle;  // faces: [warp][kLinePivotParts][face]
    unsigned long long* bar;
    __device__ __forceinline__ double* slot(int w, int k) const {
        return stage + (w * kLineFactorSlots + k % kLineFactorSlots) * (kLineChunk * 32 * kLineFactorRow);
    }
    __device__ __forceinline__ unsigned long long* full(int w, int k) const {
        return bar + w * 2 * kLineFactorSlots + k % kLineFactorSlots;
    }
    __device__ __forceinline__ unsigned long long* done(int w, int k) const { return full(w, k) + kLineFactorSlots; }
    static __device__ __forceinline__ unsigned parity(int k) { return (k / kLineFactorSlots) & 1; }
};
__device__ __forceinline__ LineFactorSmem line_factor_smem(const LineGeom& g, unsigned char* base) {
    LineFactorSmem m;
    m.stage = reinterpret_cast<double*>(base);
    m.face_y = m.stage + g.nw() * line_factor_stage();
    m.face_z = m.face_y + static_cast<long long>(kLinePivotParts) * g.nw() * g.face_y();
    m.idle = m.face_z + static_cast<long long>(kLinePivotParts) * g.nw() * g.face_z();
    m.bar = reinterpret_cast<unsigned long long*>(base + line_factor_bar_offset(g));
    return m;
}

// One compute warp's rows of block `blk`.  to_y / to_z: the faces (face_y() / face_z()
// values apart) that its last lanes along y / z fill.
template <int WY, bool D3>
__device__ __forceinline__ void line_factor_compute(const LineFactor& P, int blk, int w, const LineFactorSmem& M, double* to_y,
                                                    double* to_z, int* status) {
    constexpr int WZ = 32 / WY;
    constexpr int PAD = WY + WZ - 2;
    constexpr int C = kLineChunk;
    constexpr unsigned Z = 8, kStep = 32 * kLineFactorRow * Z;
    const LineGeom& g = P.g;
    const int lane = threadIdx.x & 31;
    const int yy = lane % WY, zz = lane / WY;
    const int shift = PAD - (yy + zz);
    const bool y_edge = D3 && yy == 0, z_edge = zz == 0;
    const int nchunk = g.psteps / C;
    const int ylen = g.face_y(), zlen = g.face_z();
    const unsigned idle = shared_addr(M.idle);
    unsigned fy = y_edge ? shared_addr(M.face_y + static_cast<long long>(kLinePivotParts) * w * ylen + shift * WZ + zz) : idle;
    unsigned fz = z_edge ? shared_addr(M.face_z + static_cast<long long>(kLinePivotParts) * w * zlen + shift * WY + yy) : idle;
    const unsigned fy_adv = y_edge ? WZ * Z : 0u, fz_adv = z_edge ? WY * Z : 0u;
    const unsigned fy_comp = y_edge ? ylen * Z : 0u, fz_comp = z_edge ? zlen * Z : 0u;
    const bool has_y = D3 && to_y != nullptr && yy == WY - 1;
    const bool has_z = to_z != nullptr && zz == WZ - 1;
    double* oy = to_y + shift * WZ + zz;
    double* oz = to_z + shift * WY + yy;
    double* result = P.rows + line_factor_at(g.slot(blk, w, 0, lane), 0);

    // operands and faces one step ahead
    double v[kLineFactorRow];
    LinePivot prev{1.0, 1.0};  // the previous row of the line (none: its coefficient is 0)
    LinePivot sy = prev, sz = prev, fyv{}, fzv{};
    auto load = [&](unsigned a) {
#pragma unroll
        for (int e = 0; e < kLineFactorRow; e += 2) {
            if (!D3 && e == 4) continue;  // (a_zi)
            double p[2];
            lds16(a + lane * 16 + e / 2 * 512, p);
            v[e] = p[0];
            v[e + 1] = p[1];
        }
    };
    auto face = [&](unsigned a, unsigned comp, LinePivot& f) {
        lds_polled(a, f.d);
        lds_polled(a + comp, f.z);
    };
    auto shuffle = [&](const LinePivot& p, LinePivot& y, LinePivot& z) {
        if (D3 && WY > 1) {
            y.d = __shfl_up_sync(0xffffffffu, p.d, 1);
            y.z = __shfl_up_sync(0xffffffffu, p.z, 1);
        }
        z.d = __shfl_up_sync(0xffffffffu, p.d, WY);
        z.z = __shfl_up_sync(0xffffffffu, p.z, WY);
    };
    mbar_wait(M.full(w, 0), 0u, status);
    __syncwarp();
    unsigned row = shared_addr(M.slot(w, 0));
    load(row);
    if (D3) face(fy, fy_comp, fyv);
    face(fz, fz_comp, fzv);
    LineWait wait;
    int left = C;  // steps left in the chunk
#pragma unroll 1
    for (int k = 0; k < nchunk;) {
        // Faces that have not arrived are polled for a while; then the row is solved with
        // what there is and the result dropped: a warp that only polls finds its step's
        // instructions gone from the cache (after about 50 us its first steps took 2.1 us
        // each instead of 0.6)
        bool late = __any_sync(0xffffffffu, line_late(fyv, fzv));
        if (late) {
            for (int polls = 0; late && polls < kLineFactorPolls; ++polls) {
                if (D3) face(fy, fy_comp, fyv);
                face(fz, fz_comp, fzv);
                late = __any_sync(0xffffffffu, line_late(fyv, fzv));
            }
            if (!late) wait = LineWait();
        }
        // the row, as if the quotients were final
        const LinePivot pz = z_edge ? fzv : sz, py = y_edge ? fyv : sy;
        LinePivot np, ny, nz;
        double lz, ly = 0.0, lx;
        auto quotient = [&](double a, const LinePivot& p, bool exact, bool& bad) {
            double l = line_quotient(a, p.d, p.z);
            if (line_quotient_bad(l, a)) {
                bad = true;
                if (exact) l = line_divide(a, p.d);
            }
            return l;
        };
        auto solve = [&](bool exact) {
            bool bad = false;
            lz = quotient(v[1], pz, exact, bad);
            np.d = fma(-v[D3 ? 4 : 7], lz, v[0]);
            if (D3) {
                ly = quotient(v[2], py, exact, bad);
                np.d = fma(-v[5], ly, np.d);
            }
            lx = quotient(v[3], prev, exact, bad);
            np.d = fma(-v[6], lx, np.d);
            np.z = line_pivot_reciprocal(np.d);
            return bad;
        };
        const bool bad = solve(false);
        shuffle(np, ny, nz);
        if (late) {
            if (!wait.expired(status)) continue;
            // give up: zeros in place of what did not arrive
            if (line_late(fyv, fyv)) fyv = LinePivot{0.0, 0.0};
            if (line_late(fzv, fzv)) fzv = LinePivot{0.0, 0.0};
            __syncwarp();
            continue;
        }
        if (__any_sync(0xffffffffu, bad)) {
            solve(true);
            __syncwarp();
            shuffle(np, ny, nz);
        }
        fy += fy_adv;
        fz += fz_adv;
        if (D3) face(fy, fy_comp, fyv);
        face(fz, fz_comp, fzv);
        prev = np;
        sy = ny;
        sz = nz;
        // only the stored copies, which others poll, are kept off the sentinel
        const double pd = off_sentinel(np.d), pz_out = off_sentinel(np.z);
        if (D3) {
            st_relaxed_generic(has_y, oy, pd);
            st_relaxed_generic(has_y, oy + ylen, pz_out);
            oy += WZ;
        }
        st_relaxed_generic(has_z, oz, pd);
        st_relaxed_generic(has_z, oz + zlen, pz_out);
        oz += WY;
        row += kStep;
        if (--left == 0) {
            left = C;
            __syncwarp();
            if (lane == 0) mbar_arrive(M.done(w, k));
            if (++k < nchunk) {
                mbar_wait(M.full(w, k), M.parity(k), status);
                __syncwarp();
                row = shared_addr(M.slot(w, k));
            } else {
                row -= kStep;  // (values that nothing uses)
            }
        }
        load(row);
        *reinterpret_cast<double2*>(result) = make_double2(np.d, lz);
        *reinterpret_cast<double2*>(result + 64) = make_double2(ly, lx);
        result += 32 * kLineFactorRow;
    }
}

template <int WY, bool D3>
__device__ __forceinline__ void line_factor_block(const LineFactor& P, int blk, const LineFactorSmem& M, double* next_z,
                                                  bool z_from_l2, int* status) {
    const LineGeom& g = P.g;
    const int nw = g.nw();
    const int w = threadIdx.x >> 5;
    const int iy = blk % g.nby, iz = blk / g.nby;
    constexpr long long parts = kLinePivotParts;
    const long long xb = parts * g.xch_block();
    if (w < nw) {
        const int wyi = w % g.by, wzi = w / g.by;
        double* to_y = nullptr;
        double* to_z = nullptr;
        if (D3) {
            if (wyi + 1 < g.by)
                to_y = M.face_y + parts * (w + 1) * g.face_y();
            else if (iy + 1 < g.nby)
                to_y = P.xch + (blk + 1) * xb + parts * wzi * g.face_y();
        }
        if (wzi + 1 < g.bz)
            to_z = M.face_z + parts * (w + g.by) * g.face_z();
        else if (next_z != nullptr)
            to_z = next_z + parts * wyi * g.face_z();
        else if (iz + 1 < g.nbz)
            to_z = P.xch + (blk + g.nby) * xb + parts * g.bz * g.face_y() + parts * wyi * g.face_z();
        line_factor_compute<WY, D3>(P, blk, w, M, to_y, to_z, status);
    } else if (w < 2 * nw) {  // helper: bulk copies of the staged rows
        const int cw = w - nw;
        const int nchunk = g.psteps / kLineChunk;
        const long long first = g.slot(blk, cw, 0, 0);
        int k = 0;
        for (; k < nchunk; ++k) {
            // (given up: nothing more is staged, and the compute warp's waits give up as well)
            if (k >= kLineFactorSlots && !__all_sync(0xffffffffu, mbar_wait(M.done(cw, k - kLineFactorSlots),
                                                                            M.parity(k - kLineFactorSlots), status)))
                break;
            if ((threadIdx.x & 31) == 0) {
                constexpr unsigned bytes = kLineChunk * 32 * kLineFactorRow * 8;
                mbar_arrive_expect(M.full(cw, k), bytes);
                bulk_load(M.slot(cw, k), P.rows + line_factor_at(first + static_cast<long long>(k) * kLineChunk * 32, 0), bytes,
                          M.full(cw, k));
            }
            __syncwarp();
        }
        for (int q = max(0, k - kLineFactorSlots); q < k; ++q) mbar_land(M.full(cw, q), M.parity(q));
        __syncwarp();
    } else {
        // halo warps: the components of a face one after the other, a warp each for
        // y and z would wait for the first to end; so each component has its own warp
        const int h = w - 2 * nw;
        const int comp = h % kLinePivotParts;
        if (h < kLinePivotParts) {
            double* const x = P.xch + blk * xb + parts * g.bz * g.face_y() + static_cast<long long>(comp) * g.face_z();
            if (iz > 0 && z_from_l2)
                line_halo(x, M.face_z + static_cast<long long>(comp) * g.face_z(), kLinePivotParts * g.face_z(), 1, g.by, WY, g.pad(), g.nx, status);
        } else if (D3) {
            double* const x = P.xch + blk * xb + static_cast<long long>(comp) * g.face_y();
            if (iy > 0)
                line_halo(x, M.face_y + static_cast<long long>(comp) * g.face_y(), kLinePivotParts * g.face_y(), g.by, g.bz, 32 / WY, g.pad(), g.nx,
                          status);
        }
    }
}
__host__ __device__ inline int line_factor_threads(const LineGeom& g) { return (2 * g.nw() + (g.ny > 1 ? 2 : 1) * kLinePivotParts) * 32; }

__device__ __forceinline__ void line_factor_reset(const LineGeom& g, int iy, int iz, const LineFactorSmem& M, bool again) {
    const int lane = threadIdx.x & 31;
    const int nwarp = static_cast<int>(blockDim.x >> 5);
    const int nw = g.nw();
    for (int f = static_cast<int>(threadIdx.x >> 5); f < kLinePivotParts * (g.ny > 1 ? 2 * nw : nw); f += nwarp) {
        const bool z = f < kLinePivotParts * nw;
        const int c = z ? f : f - kLinePivotParts * nw;  // kLinePivotParts w + component
        const int w = c / kLinePivotParts;
        const int width = z ? g.wy : g.wz;
        const int len = z ? g.face_z() : g.face_y();
        double* const p = (z ? M.face_z : M.face_y) + static_cast<long long>(c) * len;
        const bool zero = z ? (iz == 0 && w / g.by == 0) : (iy == 0 && w % g.by == 0);
        const int lo = zero ? len : g.pad() * width, hi = (g.pad() + g.nx) * width;
        for (int j = lane; j < len; j += 32) p[j] = j >= lo && j < hi ? Sentinel<double>::value() : 0.0;
    }
    for (int j = threadIdx.x; j < kLineIdle; j += blockDim.x) M.idle[j] = 0.0;
    for (int j = threadIdx.x; j < 2 * nw * kLineFactorSlots; j += blockDim.x) {
        if (again) mbar_inval(M.bar + j);
        mbar_init(M.bar + j, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Factorises the operand stream in place.  Launched with clusters of g.cl CTAs along z
// (CLUSTER), or without.
template <int WY, bool D3, bool CLUSTER>
__global__ void __launch_bounds__((2 * kLineFactorWarps + 2 * kLinePivotParts) * kWarp, 1)
    ilu_factor_line_kernel(LineFactor P, unsigned* counter, int* status) {
    extern __shared__ __align__(16) unsigned char line_smem[];
    const LineFactorSmem M = line_factor_smem(P.g, line_smem);
    __shared__ int s_ticket;
    bool again = false;
    if constexpr (!CLUSTER) {
        for (int tk = draw_block_ticket(counter, P.g.nblk, &s_ticket); tk < P.g.nblk;
             tk = draw_block_ticket(counter, P.g.nblk, &s_ticket)) {
            const int blk = P.order[tk];
            line_factor_reset(P.g, blk % P.g.nby, blk / P.g.nby, M, again);
            again = true;
            __syncthreads();
            line_factor_block<WY, D3>(P, blk, M, nullptr, true, status);
        }
    } else {
        const unsigned rank = cluster_rank_u32();
        const unsigned CL = cluster_size_u32();
        const int nq = P.g.nby * P.g.nbzc;
        const int nclusters = static_cast<int>(gridDim.x / CL);
        for (;;) {
            // (the barriers as in sptrsv_line_cluster_kernel)
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
                line_factor_reset(P.g, iy, iz, M, again);
                again = true;
            }
            __syncthreads();
            cluster_sync_all();
            if (active) {
                const bool push = rank + 1 < CL && iz + 1 < P.g.nbz;
                double* const next = push ? map_generic_rank(M.face_z, rank + 1) : nullptr;
                line_factor_block<WY, D3>(P, blk, M, next, rank == 0, status);
            }
            __syncthreads();
        }
    }
}

// Row of thread i of the two kernels below, and its slot; -1: no row.  A warp takes four
// neighbouring lines by eight rows, so that both the CSR values (a line's rows lie together)
// and the stream (a step's lanes lie together) are read and written in whole sectors.
__device__ __forceinline__ long long line_factor_row(const LineGeom& g, long long i, long long& slot, int& x, int& y, int& z) {
    const int lane = static_cast<int>((i >> 3) & 31);
    long long t = i >> 8;
    const int chunks = g.psteps / 8, nw = g.nw();
    const int s = static_cast<int>(t % chunks) * 8 + static_cast<int>(i & 7);
    t /= chunks;
    const int w = static_cast<int>(t % nw);
    const int b = static_cast<int>(t / nw);
    const int yy = lane % g.wy, zz = lane / g.wy;
    slot = g.slot(b, w, s, lane);
    y = ((b % g.nby) * g.by + w % g.by) * g.wy + yy;
    z = ((b / g.nby) * g.bz + w / g.by) * g.wz + zz;
    x = s - (yy + zz);
    return y < g.ny && z < g.nz && x >= 0 && x < g.nx ? x + static_cast<long long>(g.nx) * (y + static_cast<long long>(g.ny) * z) : -1;
}

// Packs the operand stream from A's values on the factor's pattern.  The entries a_ji of the
// lower neighbours j are theirs at i: the first (x), the one after it (y) or the last (z) of
// their strict-upper parts.  Slots without a row hold a unit pivot.
static __global__ void line_factor_pack_kernel(LineGeom g, const int* __restrict__ rp, const int* __restrict__ diag,
                                               const double* __restrict__ a, const double* __restrict__ shift,
                                               double* __restrict__ dst) {
    const long long plane = static_cast<long long>(g.nx) * g.ny;
    const int az = g.ny > 1 ? 4 : 7;  // (2-D rows have three parts)
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < g.slots();
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long slot;
        int x, y, z;
        const long long r = line_factor_row(g, i, slot, x, y, z);
        double v[kLineFactorRow] = {1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (r >= 0) {
            int p = rp[r];
            if (z > 0) {
                v[1] = a[p++];
                (az == 4 ? v[4] : v[7]) = a[rp[r - plane + 1] - 1];
            }
            if (y > 0) {
                v[2] = a[p++];
                v[5] = a[diag[r - g.nx] + 1 + (x < g.nx - 1 ? 1 : 0)];
            }
            if (x > 0) {
                v[3] = a[p++];
                v[6] = a[diag[r - 1] + 1];
            }
            v[0] = shift != nullptr ? a[p] + shift[r] : a[p];
        }
#pragma unroll
        for (int e = 0; e < kLineFactorRow; e += 2)
            if (e != 4 || g.ny > 1) *reinterpret_cast<double2*>(dst + line_factor_at(slot, e)) = make_double2(v[e], v[e + 1]);
    }
}

// Takes the factorised rows from the stream to the CSR values (the strict-upper entries stay
// A's) and reports the pivots that are zero or not finite.
static __global__ void line_factor_unpack_kernel(LineGeom g, const int* __restrict__ rp, const double* __restrict__ src,
                                                 double* __restrict__ lu, int* status) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < g.slots();
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long slot;
        int x, y, z;
        const long long r = line_factor_row(g, i, slot, x, y, z);
        if (r < 0) continue;
        const double2 dz = *reinterpret_cast<const double2*>(src + line_factor_at(slot, 0));
        const double2 yx = *reinterpret_cast<const double2*>(src + line_factor_at(slot, 2));
        int p = rp[r];
        if (z > 0) lu[p++] = dz.y;
        if (y > 0) lu[p++] = yx.x;
        if (x > 0) lu[p++] = yx.y;
        lu[p] = dz.x;
        const unsigned dh = static_cast<unsigned>(__double2hiint(dz.x)) << 1;
        if (dh >= 0x7FFu << 21 || (dh | static_cast<unsigned>(__double2loint(dz.x))) == 0u) {
            atomicAdd(status + kStatusBreakdowns, 1);
            atomicMin(status + kStatusFirstBreakdown, static_cast<int>(r));
        }
    }
}

}  // namespace gb300
