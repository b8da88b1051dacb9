// Neighbour-list build and real-space pair forces on shared-memory tiles.
//
// One block per group of consecutive cells (nxm_hood.cuh): the block stages
// the group's neighbourhood once, then each warp takes pairs of the group's
// atoms, near ones, which share a list.
//
// Physics follows NonbondedForce::DirectForcesAndEnergy
// (core/baseline/src/Forces/NonbondedForce.cpp:530-585): sigma_ij =
// sigma_i/2 + sigma_j/2, eps_ij = (2 sqrt eps_i)(2 sqrt eps_j), no LJ shift,
// no dispersion correction.  The optional switching function is applied per
// pair (the reference never resets its switch state between pairs, :541;
// that order-dependent carry-over is not reproduced).  Pair membership is
// decided exactly as the reference's list does (NeighborList.cpp:106-116):
// FP64 single-shift minimum image (PeriodicBoundaryCondition.cpp:93-104),
// r^2 < cutoff^2.  The list holds a superset (cutoff + skin, FP32 test with
// a safety margin); in mixed mode the FP32 r^2 settles every pair except
// those within 1e-5 relative of the cutoff, which are re-tested in FP64.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "nxm_ewald64.cuh"
#include "nxm_hood.cuh"
#include "nxm_view.h"

namespace nxm {

// r^2 of the pair exactly as the reference forms it: d = p_j - p_i with one
// shift per component, then (dx*dx + dy*dy) + dz*dz with no fused multiply-add.
__device__ __forceinline__ double exact_r2(const DevView &v, const SysDev &S, int i, int j) {
    double dx = min_image(__dsub_rn(v.x[j], v.x[i]), S.L[0], S.halfL[0]);
    double dy = min_image(__dsub_rn(v.y[j], v.y[i]), S.L[1], S.halfL[1]);
    double dz = min_image(__dsub_rn(v.z[j], v.z[i]), S.L[2], S.halfL[2]);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ void offset_in_cell(const DevView &v, const SysDev &S, int s, int c3, float o[3]) {
    int c[3] = {c3 & 1023, (c3 >> 10) & 1023, (c3 >> 20) & 1023};
    double p[3] = {v.x[s], v.y[s], v.z[s]};
#pragma unroll
    for (int d = 0; d < 3; ++d) o[d] = (float)min_image(p[d] - (S.lb[d] + c[d] * S.cs[d]), S.L[d], S.halfL[d]);
}

// This system's cell-image displacements (v.dtab: code r * kRowCells +
// oz + 2 -> -(ox, oy, oz) * cell edge) copied into shared memory by the
// threads outside warp 0 while warp 0 enumerates the neighbourhood; read
// after the barrier that follows.
__device__ __forceinline__ void load_dtab(const DevView &v, int sys, float4 *s_dt) {
    const float4 *dt = v.dtab + sys * kDtabStride;
    for (int e = (int)threadIdx.x - 32; e < 25 * kRowCells; e += blockDim.x - 32)
        if (e >= 0) s_dt[e] = __ldg(dt + e);
}

// Stage the group's neighbourhood (spans already in shared memory):
// positions shifted into the group frame, .w = the scaled charge (pair
// kernel, mixed mode) or the original index's bits (build), and the LJ
// parameters (pair kernel).  Each atom's
// own-cell offset is shifted by its cell's displacement from the group's
// first cell (a span's cells are consecutive in z, so the code is the
// span's first code plus the z step).  In mixed mode each lane loads four
// atoms of its span before it stores any, so the loads of a span are in
// flight together.
template <bool BUILD, bool MIXED>
__device__ void stage(const DevView &v, const SysDev &S, float4 *s_q, float2 *s_lj, const HoodSpan *spans, int nsp,
                      const float4 *s_dt) {
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int sp = warp; sp < nsp; sp += nw) {
        HoodSpan h = spans[sp];
        if (MIXED) {
            constexpr int U = 4;
            for (int t0 = 0; t0 < h.count; t0 += 32 * U) {
                int cj[U], oj[U];
                float4 p[U];
                float2 l[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    int t = t0 + lane + 32 * u;
                    if (t < h.count) {
                        int j = h.start + t;
                        cj[u] = v.cell3[j];
                        p[u] = v.pf[j];
                        if (BUILD)
                            oj[u] = v.orig[j];
                        else
                            l[u] = v.ljf[j];
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    int t = t0 + lane + 32 * u;
                    if (t < h.count) {
                        int k = h.offset + t;
                        float4 D = s_dt[h.code0 + (((cj[u] >> 20) & 1023) - h.cz0)];
                        s_q[k] = make_float4(p[u].x - D.x, p[u].y - D.y, p[u].z - D.z,
                                             BUILD ? __int_as_float(oj[u]) : p[u].w);
                        if (!BUILD) s_lj[k] = l[u];
                    }
                }
            }
        } else {
            for (int t = lane; t < h.count; t += 32) {
                int j = h.start + t, k = h.offset + t;
                int cj = v.cell3[j];
                float4 D = s_dt[h.code0 + (((cj >> 20) & 1023) - h.cz0)];
                float o[3];
                offset_in_cell(v, S, j, cj, o);
                s_q[k] = make_float4(o[0] - D.x, o[1] - D.y, o[2] - D.z, BUILD ? __int_as_float(v.orig[j]) : 0.f);
            }
        }
    }
    __syncthreads();
}

// Lists.  One list serves two atoms of a cell, the pair that k_cellsort put
// together (near neighbours, most often bonded ones; pair_first and
// DevView::ipair): the union of their neighbours, of which 12% belong to one
// of them only.  A list's 256-entry chunks are stored transposed, entry p of
// a chunk at position 8 * (p mod 32) + p / 32, so that lane L of a warp
// fetches entries L, L+32, ..., L+224 with one 16-byte load.  An entry holds
// 8 times the tile index (the byte offset of the atom's LJ pair in the pair
// kernel's staged tile; tile indices stay below 8,192) and in its low bits
// which of the two atoms it is excluded from (1: the first, 2: the second;
// from both: no entry); such entries come last.  The list ends with entries
// of the tile's spare place (an atom beyond every cutoff) up to a multiple of
// 32, so that the walk needs no range check.
__device__ __forceinline__ int list_pos(int p) { return (p & ~255) | ((p & 31) << 3) | ((p >> 5) & 7); }
constexpr int kEntryShift = 3;
constexpr int kTileSpare = 32;  // places behind a staged tile's capacity, the first of them the spare one

// Shared memory by 32-bit addresses: base plus entry is an address as it is.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 lds128(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float2 lds64(unsigned a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
// The value in a register: not worked out again where it is used.
__device__ __forceinline__ unsigned held(unsigned a) {
    asm volatile("mov.u32 %0, %0;" : "+r"(a));
    return a;
}
__device__ __forceinline__ int lds32(unsigned a) {
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts32(unsigned a, int v) {
    asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(unsigned a, int v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((short)v) : "memory");
}

// The list of pair q in memory.
__device__ __forceinline__ uint16_t *pair_list(const DevView &v, int q) {
    return v.nl16 + (size_t)q * pair_stride(v.stride);
}

// ------------------------------------------------------------------ build

// Stores one 256-entry list chunk held in order in shared memory as the list
// layout wants it: lane l writes 16 bytes, entries l + 32 q for q = 0..7.
__device__ __forceinline__ void store_chunk(uint16_t *dst, const uint16_t *src, int lane) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = (uint32_t)src[lane + 64 * q] | ((uint32_t)src[lane + 64 * q + 32] << 16);
    reinterpret_cast<uint4 *>(dst)[lane] = make_uint4(w[0], w[1], w[2], w[3]);
}

// An atom of a pair, for the build: its tile position, original index and
// exclusion partners (the first 32 in shared memory at `list`).
struct BuildAtom {
    float x, y, z;
    int oi, e0, ne, lo;
    unsigned win, list;
    __device__ __forceinline__ void load(const DevView &v, float4 q, unsigned list_, int lane) {
        x = q.x;
        y = q.y;
        z = q.z;
        oi = __float_as_int(q.w);
        list = list_;
        e0 = v.excl_off[oi];
        ne = v.excl_off[oi + 1] - e0;
        if (lane < ne) sts32(list + 4 * lane, v.excl_lst[e0 + lane]);
        // Index window [lo, lo + win] of the atom itself and its exclusion
        // partners (rows ascending): a candidate outside it needs no
        // membership test.  The atom is left out by its index too, so every
        // image of it is (the far one lies beyond the list radius anyway).
        lo = ne ? min(v.excl_lst[e0], oi) : oi;
        win = (unsigned)((ne ? max(v.excl_lst[e0 + ne - 1], oi) : oi) - lo);
    }
    __device__ __forceinline__ bool excluded(const DevView &v, int oj) const {
        bool ex = oj == oi;
#pragma unroll 1
        for (int e = 0; e < min(ne, 32); ++e) ex |= lds32(list + 4 * e) == oj;
#pragma unroll 1
        for (int e = 32; e < ne; ++e) ex |= v.excl_lst[e0 + e] == oj;
        return ex;
    }
    __device__ __forceinline__ float r2(const float4 &q) const {
        const float dx = x - q.x, dy = y - q.y, dz = z - q.z;
        return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    }
};

// Each warp takes pairs of the group; every staged atom within the list
// radius of one of the two and not excluded from it is appended to the
// pair's list (ballot compaction: deterministic order).  A pair scans only
// the rows of the neighbourhood its list spheres reach, and in each row
// (z-sorted: k_cellsort orders every cell by z) only the atoms within the z
// extent the spheres have over that row, found by binary search (0.01 nm
// margin), in tile order: the list is the one a scan of the whole tile gives.
//
// Bound by instruction issue: a warp tests 32 candidates against both atoms
// with one load of each candidate and one compaction, so an atom costs about
// two thirds of what a list of its own does, and half the list traffic.
// 94,100 atoms: 312 us with a list per atom, 221 so (257 -> 167 M warp
// instructions).  Its loops are kept rolled: unrolled by the compiler they
// spend more on moving registers than the unrolling saves (241 -> 221 us).
//
// W warps per block: 16 (two blocks per SM) or, when two blocks' shared
// memory does not fit on an SM, 32 (one block per SM, the same 32 warps).
constexpr int kKeep = 64, kBuildWarpWords = 512 + kKeep + 128;  // 16-bit words
template <bool MIXED, int W>
__global__ void __launch_bounds__(W * 32, W == kHoodWarps ? 2 : 1) k_build(DevView v) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (!v.flags->rebuild) return;
    const unsigned full = 0xffffffffu;
    CellGroup G = v.groups[blockIdx.x];
    int a0 = v.cell_start[G.cell], a1 = v.cell_start[G.cell + G.ncell];
    if (a0 == a1) return;
    const int q0 = pair_first(a0, G.cell), q1 = pair_first(a1, G.cell + G.ncell);
    const SysDev &S = v.sys[G.sys];
    if (!S.nb_on) {
        for (int q = q0 + threadIdx.x; q < q1; q += blockDim.x) v.ncount[q] = make_int2(0, 0);
        return;
    }
    int cap = v.hood_cap;
    float4 *s_q = reinterpret_cast<float4 *>(smem);  // .w: the original index's bits
    // per warp: a list's two chunks in the making (512 entries), the entries
    // kept for its end (kKeep), the two atoms' exclusion partners (2 x 32)
    uint16_t *s_buf = reinterpret_cast<uint16_t *>(s_q + cap);
    int *s_bnd = reinterpret_cast<int *>(s_buf + W * kBuildWarpWords);
    HoodSpan *spans = reinterpret_cast<HoodSpan *>(s_bnd + 25 * (kRowCells + 1));
    int *s_n = reinterpret_cast<int *>(spans + kMaxSpans);
    __shared__ float4 s_dt[25 * kRowCells];
    load_dtab(v, G.sys, s_dt);
    int n = hood_setup(v, S, v.cell3[a0], G.ncell, spans, s_n, s_bnd);
    int nsp = s_n[1];
    // the group's own atoms are consecutive in the tile from here on
    const int kbase = s_bnd[12 * (kRowCells + 1) + 2] - a0;
    // the spans, for the pair kernel's steps until the next rebuild
    {
        const int *src = reinterpret_cast<const int *>(spans);
        int *dst = v.gspan + (size_t)blockIdx.x * kGroupSpanWords;
        for (int e = threadIdx.x; e < min(nsp, kMaxSpans) * kSpanWords; e += blockDim.x) dst[e] = src[e];
        if (threadIdx.x == 0) v.gspan_n[blockIdx.x] = make_int4(n, nsp, kbase, 0);
    }
    if (n > v.hood_cap || nsp > kMaxSpans) {
        if (threadIdx.x == 0) atomicOr(&v.flags->error, ERR_NLIST_OVERFLOW);
        return;
    }
    stage<true, MIXED>(v, S, s_q, nullptr, spans, nsp, s_dt);
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    float rl2 = S.rlist2f * 1.0001f + 1e-6f;
    const float margin = 0.01f;
    const float rlm = sqrtf(rl2) + margin;
    const float csx = (float)S.cs[0], csy = (float)S.cs[1], csz = (float)S.cs[2], icsz = 1.0f / csz;
    int g = G.ncell;
    uint16_t *buf = s_buf + warp * kBuildWarpWords, *keep = buf + 512;
    const unsigned keep_addr = smem_addr(keep), ex_addr = keep_addr + 2 * kKeep, lt = (1u << lane) - 1u;
    const unsigned tile_lane = held(smem_addr(s_q) + 16 * lane), buf_addr = held(smem_addr(buf));
    const int cap_entries = pair_stride(v.stride);
    for (int q = q0 + warp; q < q1; q += nw) {
        const int2 ab = v.ipair[q];
        if (ab.x < 0) continue;
        BuildAtom A, B;
        A.load(v, s_q[kbase + ab.x], ex_addr, lane);
        B.load(v, s_q[kbase + (ab.y < 0 ? ab.x : ab.y)], ex_addr + 128, lane);
        if (ab.y < 0) B.x = B.y = B.z = 1e15f;  // no second atom: beyond every list radius
        __syncwarp();
        int count = 0, kept = 0;
        unsigned flagged = 0;  // chunks with an entry that is excluded from one of the two
        uint16_t *out = pair_list(v, q);
        // lane r < 25: the tile range [kb, ke) of row r that a sphere reaches
        int kb = 0, ke = 0;
        if (lane < 25) {
            // z extent of the two spheres over the row: distance from each
            // atom to the row's cell column in x and y
            const float ox = (float)(lane / 5 - 2) * csx, oy = (float)(lane % 5 - 2) * csy;
            float zl = 1e30f, zh = -1e30f;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float px = m ? B.x : A.x, py = m ? B.y : A.y, pz = m ? B.z : A.z;
                const float ddx = fmaxf(fmaxf(ox - px, px - (ox + csx)), 0.0f);
                const float ddy = fmaxf(fmaxf(oy - py, py - (oy + csy)), 0.0f);
                const float rem = rlm * rlm - (ddx * ddx + ddy * ddy);
                if (rem >= 0.0f) {
                    const float h = sqrtf(rem) + margin;
                    zl = fminf(zl, pz - h);
                    zh = fmaxf(zh, pz + h);
                }
            }
            if (zl <= zh) {
                int zlo = max((int)floorf(zl * icsz), -2);
                int zhi = min((int)floorf(zh * icsz), g + 1);
                if (zlo <= zhi) {
                    const int *b = s_bnd + lane * (kRowCells + 1);
                    // the row is sorted by z (cells in z order, atoms in a
                    // cell by z): narrow to the atoms with z in [zl, zh].  The
                    // first such atom lies in cell zlo and the last in cell
                    // zhi, so each search covers one cell.
                    int l = b[zlo + 2], r = b[zlo + 3];
#pragma unroll 1
                    while (l < r) {
                        int mid = (l + r) >> 1;
                        if (s_q[mid].z < zl)
                            l = mid + 1;
                        else
                            r = mid;
                    }
                    kb = l;
                    l = max(b[zhi + 2], kb);
                    r = b[zhi + 3];
#pragma unroll 1
                    while (l < r) {
                        int mid = (l + r) >> 1;
                        if (s_q[mid].z <= zh)
                            l = mid + 1;
                        else
                            r = mid;
                    }
                    ke = l;
                }
            }
        }
        // The list is assembled per 256-entry chunk in two halves per warp
        // (entry p at p & 511), so an iteration that completes a chunk writes
        // on into the other half; a completed chunk is stored transposed as
        // in memory (lane l's 16 bytes hold entries l + 32 q, q = 0..7).
        // Every lane stores: a rejected candidate goes to count + 32 + lane,
        // past the entries of this iteration -- a slot that a later entry
        // overwrites or that lies beyond the list's count (never in the half
        // being stored: at most 32 entries come per iteration).
        auto append = [&](bool cand, int entry) {
            const unsigned m = __ballot_sync(full, cand);
            const int newc = count + __popc(m);
            const int at = (cand ? count + __popc(m & lt) : count + 32 + lane) & 511;
            sts16(buf_addr + 2 * at, entry);
            if ((newc ^ count) >> 8) {
                // chunk count >> 8 complete: one 16-byte store per lane
                __syncwarp();
                const int c = count >> 8;
                if ((c + 1) * 256 <= cap_entries) store_chunk(out + c * 256, buf + (c & 1) * 256, lane);
                __syncwarp();
            }
            count = newc;
        };
        unsigned rows = __ballot_sync(full, ke > kb);
#pragma unroll 1
        while (rows) {
            int r = __ffs(rows) - 1;
            rows &= rows - 1;
            const int rb = __shfl_sync(full, kb, r), re = __shfl_sync(full, ke, r);
            unsigned at = tile_lane + 16 * rb;
            int entry0 = (rb + lane) << kEntryShift;
#pragma unroll 1
            for (int left = re - rb; left > 0; left -= 32, at += 512, entry0 += 32 << kEntryShift) {
                // a place past the row's end reads a later row or the chunk
                // buffers behind the tile, inside the block's shared
                // memory; such a lane is no candidate
                const float4 c = lds128(at);
                const float reach = lane < left ? rl2 : -1.0f;
                const float2 dx = make_float2(A.x - c.x, B.x - c.x), dy = make_float2(A.y - c.y, B.y - c.y),
                             dz = make_float2(A.z - c.z, B.z - c.z);
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                bool inA = r2.x < reach, inB = r2.y < reach;
                const int oj = __float_as_int(c.w);
                int entry = entry0;
                bool cand = inA | inB;
                if (__any_sync(full, cand && ((unsigned)(oj - A.lo) <= A.win || (unsigned)(oj - B.lo) <= B.win))) {
                    const bool exA = A.excluded(v, oj), exB = B.excluded(v, oj);
                    inA &= !exA;
                    inB &= !exB;
                    cand = inA | inB;
                    entry |= (exA ? 1 : 0) | (exB ? 2 : 0);
                    // excluded from one of the two: kept for the list's end
                    // while there is room
                    const unsigned m = __ballot_sync(full, cand && (exA || exB));
                    if (kept + __popc(m) <= kKeep) {
                        if ((m >> lane) & 1) sts16(keep_addr + 2 * (kept + __popc(m & lt)), entry);
                        kept += __popc(m);
                        cand = cand && !((m >> lane) & 1);
                    } else {
                        // (an iteration's entries lie in the chunks of its
                        // first and its last possible place)
                        flagged |= 1u << (count >> 8) | 1u << min((count + 31) >> 8, 31);
                    }
                }
                // The FP64 kernel and the pair set take an entry's atom at its
                // nearest image; in a box of few cells the tile holds two
                // images of an atom, one for either atom of the pair, so
                // there an entry counts only for the atoms it is near
                // (marked in FP64 only: the mixed kernel takes the tile's image)
                if (!MIXED) entry |= (inA ? 0 : 1) | (inB ? 0 : 2);
                append(cand, entry);
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int t0 = 0; t0 < kept; t0 += 32) {
            flagged |= 1u << (count >> 8) | 1u << min((count + 31) >> 8, 31);
            append(t0 + lane < kept, keep[min(t0 + lane, kKeep - 1)]);
        }
        __syncwarp();
        if (((count + lane) ^ count) < 32 && (count & 31)) sts16(buf_addr + 2 * ((count + lane) & 511), cap << kEntryShift);
        __syncwarp();
        {
            const int c = count >> 8;
            if ((count & 255) && (c + 1) * 256 <= cap_entries) store_chunk(out + c * 256, buf + (c & 1) * 256, lane);
        }
        __syncwarp();
        bool over = false;
        if (count > v.stride) {
            // The capacity is an atom's: its own entries, whatever the
            // union's count.  Counted apart, as it is hardly ever asked.
            int nA = 0, nB = 0;
#pragma unroll 1
            for (unsigned left = __ballot_sync(full, ke > kb); left; left &= left - 1) {
                const int r = __ffs(left) - 1;
                const int rb = __shfl_sync(full, kb, r), re = __shfl_sync(full, ke, r);
#pragma unroll 1
                for (int k = rb + lane; k < re; k += 32) {
                    const float4 c = s_q[k];
                    const int oj = __float_as_int(c.w);
                    nA += A.r2(c) < rl2 && !A.excluded(v, oj);
                    nB += B.r2(c) < rl2 && !B.excluded(v, oj);
                }
            }
            over = max(__reduce_add_sync(full, nA), __reduce_add_sync(full, nB)) > v.stride;
        }
        if (lane == 0) {
            v.ncount[q] = make_int2(over ? 0 : count, (int)flagged);
            if (over) atomicOr(&v.flags->error, ERR_NLIST_OVERFLOW);
        }
    }
}

// ------------------------------------------------------------------ pairs

struct PairPrm {
    float ex2c, a04, k2a, sw, inv_w;  // SysDev::ex2c, a04, k2a, sw_distf, sw_invf
};

__device__ __forceinline__ float fast_ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }

// g(t) of erfc(x) = exp(-x^2) g(t), t = 1 / (1 + 0.4 x), x in [0, 4]: degree-6
// least-squares fit of the scaled complementary error function on Chebyshev
// nodes of t, max relative error 5e-7 in FP32 (derivation and error table:
// fit_erfcx.py next to this file).
__device__ __forceinline__ float2 erfcx_fit2(float2 t) {
    float2 g = dup2(-2.164941738e-01f);
    g = __ffma2_rn(g, t, dup2(7.803782561e-01f));
    g = __ffma2_rn(g, t, dup2(-4.985805536e-01f));
    g = __ffma2_rn(g, t, dup2(5.875147125e-01f));
    g = __ffma2_rn(g, t, dup2(1.009222009e-01f));
    g = __ffma2_rn(g, t, dup2(2.479314205e-01f));
    g = __ffma2_rn(g, t, dup2(-1.671998421e-03f));
    return g;
}

// The two atoms of a pair against one list entry: FP32 force (and energy) of
// both, NonbondedForce.cpp:559-581 in single precision, in the two halves of
// packed FP32x2 operations (one instruction for both; the reciprocal square
// root, exponential and reciprocal are scalar), added to the lane's sums
// where `in`.  Without branches: an entry outside the cutoff (or at a distance
// that is not a number) gives a value that a select drops.  The selects are on
// the results: a factor set to zero instead would still carry a NaN into the
// sums.
// exp(-(alpha r)^2) comes straight from r^2; erfc(alpha r) =
// exp(-(alpha r)^2) g(t), t = 1 / (1 + 0.4 alpha r).
struct PairSums {
    float2 fx, fy, fz, ec, ev;  // .x: the first atom, .y: the second
};

template <bool ENERGY, bool SW>
__device__ __forceinline__ void pair_mixed2(bool in0, bool in1, float2 dx, float2 dy, float2 dz, float2 r2, float2 qq,
                                            float2 sg, float2 eps, const PairPrm &P, PairSums &F) {
    auto only = [&](float2 a) { return make_float2(in0 ? a.x : 0.0f, in1 ? a.y : 0.0f); };
    const float2 rinv = make_float2(fast_rsqrt(r2.x), fast_rsqrt(r2.y));
    const float2 rinv2 = __fmul2_rn(rinv, rinv);
    const float2 r = __fmul2_rn(r2, rinv);
    const float2 ea = __fmul2_rn(r2, dup2(P.ex2c));
    const float2 ex = make_float2(fast_ex2(ea.x), fast_ex2(ea.y));
    const float2 tt = __ffma2_rn(dup2(P.a04), r, dup2(1.0f));
    const float2 erfcv = __fmul2_rn(ex, erfcx_fit2(make_float2(fast_rcp(tt.x), fast_rcp(tt.y))));
    const float2 qr = __fmul2_rn(qq, rinv);
    float2 dEdR = __fmul2_rn(__fmul2_rn(qr, rinv2), __ffma2_rn(__fmul2_rn(dup2(P.k2a), r), ex, erfcv));
    if (ENERGY) F.ec = __fadd2_rn(F.ec, only(__fmul2_rn(qr, erfcv)));
    const float2 s2 = __fmul2_rn(__fmul2_rn(sg, sg), rinv2);
    const float2 s6 = __fmul2_rn(__fmul2_rn(s2, s2), s2);
    const float2 es6 = __fmul2_rn(eps, s6);
    float2 lj = __fmul2_rn(es6, __ffma2_rn(dup2(12.0f), s6, dup2(-6.0f)));
    if (SW) {
        // t = 0 before the switching distance (and where the system has no
        // switch): the factor is 1 and its derivative 0; at most 1, so that an
        // entry beyond every cutoff stays finite
        const float2 u = __ffma2_rn(r, dup2(P.inv_w), dup2(-P.sw * P.inv_w));
        const float2 t = make_float2(__saturatef(u.x), __saturatef(u.y));
        const float2 t2 = __fmul2_rn(t, t);
        const float2 sw = __ffma2_rn(__fmul2_rn(t2, t), __ffma2_rn(t, __ffma2_rn(t, dup2(-6.0f), dup2(15.0f)), dup2(-10.0f)),
                                     dup2(1.0f));
        const float2 mdsw = __fmul2_rn(__fmul2_rn(t2, dup2(P.inv_w)),
                                       __ffma2_rn(t, __ffma2_rn(t, dup2(30.0f), dup2(-60.0f)), dup2(30.0f)));
        const float2 l = __ffma2_rn(es6, s6, make_float2(-es6.x, -es6.y));
        lj = __ffma2_rn(sw, lj, __fmul2_rn(__fmul2_rn(l, mdsw), r));
        if (ENERGY) F.ev = __fadd2_rn(F.ev, only(__fmul2_rn(l, sw)));
    } else if (ENERGY) {
        F.ev = __fadd2_rn(F.ev, only(__ffma2_rn(es6, s6, make_float2(-es6.x, -es6.y))));
    }
    dEdR = only(__ffma2_rn(lj, rinv2, dEdR));
    F.fx = __ffma2_rn(dx, dEdR, F.fx);
    F.fy = __ffma2_rn(dy, dEdR, F.fy);
    F.fz = __ffma2_rn(dz, dEdR, F.fz);
}

// Whether list entry w, at an FP32 r^2 from atom m of its pair (0 the first, 1
// the second), is too near the cutoff for FP32 to tell: within 1e-5, and not
// excluded.  Then exact_r2 decides as the reference does.
// (lo: S.cut2f_lo, which the walk holds in a register)
__device__ __forceinline__ bool at_cutoff(const SysDev &S, unsigned w, unsigned m, float r2, float lo) {
    return !(w & (1u << m)) && r2 >= lo && r2 < S.cut2f_hi;
}

// The entries of one chunk (c0) of pair q's list whose FP32 r^2 is within
// 1e-5 of the cutoff's, which the walk left out: decided in FP64 (at_cutoff) and
// added where they are within it.  One chunk in a hundred comes here.  The energies'
// kernel calls it when the pair is done, with its own atomics, so that its
// registers are not added to the walk's (179 -> 157 us at 94,100 atoms).
template <bool ENERGY, bool SW>
__device__ __forceinline__ void near_cutoff(const DevView &v, const SysDev &S, const HoodSpan *spans, int nsp, int kbase,
                                            int q, int c0, unsigned q_addr, unsigned lj_addr) {
    const int lane = threadIdx.x & 31;
    const int2 ab = v.ipair[q];
    const int cnt = min(v.ncount[q].x, c0 + 256);
    const uint16_t *list = pair_list(v, q);
    const PairPrm P{S.ex2c, S.a04, S.k2a, S.sw_distf, S.sw_invf};
    for (int k = c0 + lane; k < cnt; k += 32) {
        const unsigned w = list[list_pos(k)], e = w & 0xfff8u;
        const float4 p = lds128(q_addr + 2 * e);
        const float2 l = lds64(lj_addr + e);
        for (int m = 0; m < 2; ++m) {
            const int i = m ? ab.y : ab.x;
            if (i < 0) continue;
            const float4 pi = lds128(q_addr + 16 * (kbase + i));
            const float dx = pi.x - p.x, dy = pi.y - p.y, dz = pi.z - p.z;
            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            if (!at_cutoff(S, w, m, r2, S.cut2f_lo)) continue;
            if (!(exact_r2(v, S, i, hood_slot(spans, nsp, (int)(e >> kEntryShift))) < S.cut2)) continue;
            const float2 li = lds64(lj_addr + 8 * (kbase + i));
            PairSums F;
            F.fx = F.fy = F.fz = F.ec = F.ev = make_float2(0.f, 0.f);
            pair_mixed2<ENERGY, SW>(true, false, make_float2(dx, 0.f), make_float2(dy, 0.f), make_float2(dz, 0.f),
                                    make_float2(r2, r2), make_float2(pi.w * p.w, 0.f), make_float2(li.x + l.x, 0.f),
                                    make_float2(li.y * l.y, 0.f), P, F);
            acc_add(static_cast<long long *>(v.fx) + i, F.fx.x);
            acc_add(static_cast<long long *>(v.fy) + i, F.fy.x);
            acc_add(static_cast<long long *>(v.fz) + i, F.fz.x);
            if (ENERGY) {
                long long *E = v.E + (size_t)v.sys_of[i] * E_SLOTS;
                atomicAdd(reinterpret_cast<unsigned long long *>(E + E_COUL),
                          static_cast<unsigned long long>(energy_fixed(0.5f * F.ec.x)));
                atomicAdd(reinterpret_cast<unsigned long long *>(E + E_VDW),
                          static_cast<unsigned long long>(energy_fixed(0.5f * F.ev.x)));
            }
        }
    }
}

// Mixed precision: one warp per pair of atoms walks the pair's list; j comes
// from the staged tile, once for both.
//
// Bound by instruction issue and the FP32 pipe (a packed operation takes the
// pipe for two).  An entry costs one load of j, one decoding and one set of
// packed operations for two interactions, 12% of which the other atom's
// share of the list adds: 145 -> 132 us at 94,100 atoms against a list per
// atom, 189 -> 129 us with the switching function at 74,400, 101 -> 88 M warp
// instructions.  Of its walk 57% of the cycles issue; the rest is the staging
// before it and a block's last pairs.
// SW: some system of the batch uses the switching function; W: warps per block
// (pairs_warps).
template <bool ENERGY, bool SW, int W>
__global__ void __launch_bounds__(W * 32, W <= kHoodWarps ? 2 : 1) k_pairs_mixed(const __grid_constant__ DevView v) {
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned full = 0xffffffffu;
    CellGroup G = v.groups[blockIdx.x];
    int a0 = v.cell_start[G.cell], a1 = v.cell_start[G.cell + G.ncell];
    if (a0 == a1) return;
    const SysDev &S = v.sys[G.sys];
    if (!S.nb_on) return;
    const int cap = v.hood_cap;
    // tile: LJ pairs first (a list entry is the byte offset of its atom's
    // pair), then positions at twice that offset past them (cap is a
    // multiple of 32, so the positions stay 16-byte aligned)
    float2 *s_lj = reinterpret_cast<float2 *>(smem);
    float4 *s_q = reinterpret_cast<float4 *>(s_lj + cap + kTileSpare);
    HoodSpan *spans = reinterpret_cast<HoodSpan *>(s_q + cap + kTileSpare);
    __shared__ float4 s_dt[25 * kRowCells];
    __shared__ int4 s_nn;
    // the neighbourhood's spans as the list build enumerated them (the
    // cells have not changed since), and the displacement table
    {
        const int *src = v.gspan + (size_t)blockIdx.x * kGroupSpanWords;
        int *dst = reinterpret_cast<int *>(spans);
        for (int e = threadIdx.x; e < kGroupSpanWords; e += blockDim.x) dst[e] = src[e];
        if (threadIdx.x == 0) {
            s_nn = v.gspan_n[blockIdx.x];
            // the spare place: an atom beyond every cutoff, without charge
            // (the next: the second atom of a pair of one, as far the other way)
            s_q[cap] = make_float4(1e15f, 1e15f, 1e15f, 0.f);
            s_q[cap + 1] = make_float4(-1e15f, -1e15f, -1e15f, 0.f);
            s_lj[cap] = s_lj[cap + 1] = make_float2(0.f, 0.f);
        }
        const float4 *dt = v.dtab + G.sys * kDtabStride;
        for (int e = threadIdx.x; e < 25 * kRowCells; e += blockDim.x) s_dt[e] = __ldg(dt + e);
    }
    __syncthreads();
    const int n = s_nn.x, nsp = s_nn.y, kbase = s_nn.z;
    if (n > v.hood_cap || nsp > kMaxSpans) {
        if (threadIdx.x == 0) atomicOr(&v.flags->error, ERR_NLIST_OVERFLOW);
        return;
    }
    // the warp's first pair, its counts and the first chunk of its list (whose
    // place always exists: the load need not wait for the count) come in
    // beside the staging, each later one's beside the sums before it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q1 = pair_first(a1, G.cell + G.ncell);
    int2 ab, nc;
    uint4 cur;
    auto fetch = [&](int q) {
        if (q >= q1) return;
        ab = v.ipair[q];
        nc = v.ncount[q];
        cur = __ldg(reinterpret_cast<const uint4 *>(pair_list(v, q)) + lane);
    };
    int q = pair_first(a0, G.cell) + warp;
    fetch(q);
    stage<false, true>(v, S, s_q, s_lj, spans, nsp, s_dt);
    const unsigned q_addr = smem_addr(s_q), lj_addr = smem_addr(s_lj);
    const float lo = S.cut2f_lo, cut2 = S.cut2f;
    const PairPrm P{S.ex2c, S.a04, S.k2a, S.sw_distf, S.sw_invf};
    PairSums F;
    F.ec = F.ev = make_float2(0.f, 0.f);
    while (q < q1) {
        const uint4 *lst4 = reinterpret_cast<const uint4 *>(pair_list(v, q)) + lane;
        q += W;
        if (ab.x < 0) {
            fetch(q);
            continue;
        }
        const int cnt = nc.x;
        const int ka = kbase + ab.x, kb = ab.y < 0 ? cap + 1 : kbase + ab.y;
        const float4 pa = s_q[ka];
        const float4 pb = s_q[kb];
        const float2 la = s_lj[ka], lb = s_lj[kb];
        F.fx = F.fy = F.fz = make_float2(0.f, 0.f);
        unsigned near = 0;  // chunks with an entry at the cutoff (energies)
        for (int c0 = 0; c0 < cnt; c0 += 256) {
            float edge = 1e30f;  // the least distance of an FP32 r^2 from the cutoff's
            // this lane's entries c0 + lane + 32u, u = 0..7, and the next chunk in flight
            uint4 nxt = c0 + 256 < cnt ? __ldg(lst4 + (c0 + 256) / 8) : make_uint4(0, 0, 0, 0);
            // FLAGS: the entry may be excluded from one of the two atoms
            auto entry = [&](unsigned w, auto flags) {
                constexpr bool FLAGS = decltype(flags)::value;
                const unsigned e = FLAGS ? w & 0xfff8u : w;
                const float4 p = lds128(q_addr + 2 * e);
                const float2 l = lds64(lj_addr + e);
                const float2 dx = make_float2(pa.x - p.x, pb.x - p.x);
                const float2 dy = make_float2(pa.y - p.y, pb.y - p.y);
                const float2 dz = make_float2(pa.z - p.z, pb.z - p.z);
                float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                if (FLAGS) {
                    if (w & 1) r2.x = 1e30f;
                    if (w & 2) r2.y = 1e30f;
                }
                const float2 off = __fadd2_rn(r2, dup2(-cut2));
                edge = fminf(edge, fminf(fabsf(off.x), fabsf(off.y)));
                pair_mixed2<ENERGY, SW>(r2.x < lo, r2.y < lo, dx, dy, dz, r2, make_float2(pa.w * p.w, pb.w * p.w),
                                        make_float2(la.x + l.x, lb.x + l.x), make_float2(la.y * l.y, lb.y * l.y), P,
                                        F);
            };
            if (c0 + 256 <= cnt && !((nc.y >> (c0 >> 8)) & 1)) {
                const uint32_t wds[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    entry((u & 1) ? wds[u >> 1] >> 16 : wds[u >> 1] & 0xffffu, std::false_type{});
            } else {
                uint4 w = cur;
                for (int u0 = c0; u0 < min(cnt, c0 + 256); u0 += 32) {
                    entry(w.x & 0xffffu, std::true_type{});
                    w.x = __funnelshift_r(w.x, w.y, 16);
                    w.y = __funnelshift_r(w.y, w.z, 16);
                    w.z = __funnelshift_r(w.z, w.w, 16);
                    w.w >>= 16;
                }
            }
            if (__any_sync(full, edge < cut2 * 1.1e-5f)) {
                if constexpr (ENERGY) {
                    near |= 1u << (c0 >> 8);
                } else {
                    // at once, into the walk's sums
                    uint4 ws = cur;
                    for (int u0 = c0; u0 < min(cnt, c0 + 256); u0 += 32) {
                        const unsigned w = ws.x & 0xffffu, e = w & 0xfff8u;
                        ws.x = __funnelshift_r(ws.x, ws.y, 16);
                        ws.y = __funnelshift_r(ws.y, ws.z, 16);
                        ws.z = __funnelshift_r(ws.z, ws.w, 16);
                        ws.w >>= 16;
                        const float4 p = lds128(q_addr + 2 * e);
                        const float2 l = lds64(lj_addr + e);
                        const float2 dx = make_float2(pa.x - p.x, pb.x - p.x);
                        const float2 dy = make_float2(pa.y - p.y, pb.y - p.y);
                        const float2 dz = make_float2(pa.z - p.z, pb.z - p.z);
                        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                        bool in0 = at_cutoff(S, w, 0, r2.x, lo);
                        bool in1 = at_cutoff(S, w, 1, r2.y, lo);
                        if (!(in0 || in1)) continue;
                        const int j = hood_slot(spans, nsp, (int)(e >> kEntryShift));
                        in0 = in0 && exact_r2(v, S, ab.x, j) < S.cut2;
                        in1 = in1 && exact_r2(v, S, ab.y, j) < S.cut2;
                        pair_mixed2<ENERGY, SW>(in0, in1, dx, dy, dz, r2, make_float2(pa.w * p.w, pb.w * p.w),
                                                make_float2(la.x + l.x, lb.x + l.x),
                                                make_float2(la.y * l.y, lb.y * l.y), P, F);
                    }
                }
            }
            cur = nxt;
        }
        const int2 at = ab;
        fetch(q);
        // six sums over 32 lanes in eight steps: lanes take a share of the
        // sums at each of the first three (bit 4 of the lane: the atom; then
        // bit 3 x or y; bit 2 set: z)
        const bool up16 = lane & 16, up8 = lane & 8, up4 = lane & 4;
        float sx = (up16 ? F.fx.y : F.fx.x) + __shfl_xor_sync(full, up16 ? F.fx.x : F.fx.y, 16);
        float sy = (up16 ? F.fy.y : F.fy.x) + __shfl_xor_sync(full, up16 ? F.fy.x : F.fy.y, 16);
        float sz = (up16 ? F.fz.y : F.fz.x) + __shfl_xor_sync(full, up16 ? F.fz.x : F.fz.y, 16);
        sx = (up8 ? sy : sx) + __shfl_xor_sync(full, up8 ? sx : sy, 8);
        sz += __shfl_xor_sync(full, sz, 8);
        sx = (up4 ? sz : sx) + __shfl_xor_sync(full, up4 ? sx : sz, 4);
        sx += __shfl_xor_sync(full, sx, 2);
        sx += __shfl_xor_sync(full, sx, 1);
        const int i = up16 ? at.y : at.x;
        if ((lane & 3) == 0 && !(up4 && up8) && i >= 0)
            acc_add(static_cast<long long *>(up4 ? v.fz : (up8 ? v.fy : v.fx)) + i, sx);
        for (; near; near &= near - 1)
            near_cutoff<ENERGY, SW>(v, S, spans, nsp, kbase, q - W, (__ffs(near) - 1) << 8, q_addr, lj_addr);
    }
    if (ENERGY) {
        // each pair sits in both partners' lists
        energy_add_f(v.E, G.sys, E_COUL, 0.5f * (F.ec.x + F.ec.y));
        energy_add_f(v.E, G.sys, E_VDW, 0.5f * (F.ev.x + F.ev.y));
    }
}

// ---- FP64 form: the same list, every pair once, in double precision from the
// FP64 positions with the reference's minimum image (NonbondedForce.cpp:548-581).
//
// Bound by the FP64 pipe (two lanes per SM and clock on this GPU), so the
// work is arranged to give that pipe as few instructions as the sum needs:
//  * a filter on FP32 r^2 from the staged box fractions (integer and FP32
//    instructions only) drops the list entries beyond the cutoff, and takes
//    each pair from one of its two lists only (the other atom's force by
//    atomics, which the FP64 engine's force sums are anyway);
//  * what passes is compacted into a per-warp queue and evaluated 32 at a
//    time, so no lane of an FP64 instruction idles;
//  * comparisons and conversions, FP64 instructions too, are done on the
//    numbers' bits;
//  * 1/r by one step from the FP32 reciprocal root (the binomial series of
//    (1 - e)^(-1/2) to second order), and the Ewald terms from polynomials in
//    r^2 in a table that stays in L1 (nxm_ewald64.cuh): about 40 FP64
//    instructions per pair, where erfc, exp, sqrt and the divisions took
//    about 240 per list entry.  23,800 atoms: 5,390 -> 553 us, the FP64 pipe
//    busy 78% of the kernel's active cycles; 2,700 atoms: 727 -> 92 us.
// The pair set is decided on the exact r^2 of the reference's list.

constexpr int kWarps64 = 8;

__device__ __forceinline__ long long bits_of(double x) { return __double_as_longlong(x); }

// -x by its sign bit
__device__ __forceinline__ double negated(double x) {
    return __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x));
}

// min_image() with |d| > L/2 compared as integers (the order of non-negative
// doubles), and no FP64 addition issued for a warp none of whose lanes shifts
// (volatile: else both sums are formed ahead of the vote and one is selected,
// a fifth of the kernel's DADD by the opcode counters; 24k atoms 567 -> 554 us).
__device__ __forceinline__ double min_image_bits(double d, double L, double halfL) {
    const long long b = __double_as_longlong(d);
    const bool far = (b & 0x7fffffffffffffffLL) > __double_as_longlong(halfL);
    if (__any_sync(__activemask(), far)) {
        const double shift = far ? (b < 0 ? L : negated(L)) : 0.0;
        asm volatile("add.rn.f64 %0, %0, %1;" : "+d"(d) : "d"(shift));
    }
    return d;
}

template <bool ENERGY, bool SW>
struct Pairs64 {
    const DevView &v;
    const SysDev &S;
    const double L0, L1, L2, h0, h1, h2, cut2, alpha2, alpha3, sw_dist, sw_inv;
    const long long near_bits;  // r^2 from here on: too close to the cutoff for a fused r^2 to decide
    const float a2f;
    double fx = 0, fy = 0, fz = 0, ec = 0, ev = 0;
    int cur = -1;  // the atom the warp's sums fx, fy, fz belong to
    double *sums;  // DevView::fpair: the copy that this lane adds to

    __device__ Pairs64(const DevView &v_, const SysDev &S_)
        : v(v_), S(S_), L0(S_.L[0]), L1(S_.L[1]), L2(S_.L[2]), h0(S_.halfL[0]), h1(S_.halfL[1]), h2(S_.halfL[2]),
          cut2(S_.cut2), alpha2(S_.alpha2), alpha3(S_.alpha3), sw_dist(S_.sw_dist),
          sw_inv(SW ? 1.0 / (S_.cutoff - S_.sw_dist) : 0.0), near_bits(bits_of(S_.cut2 * (1.0 - 1e-14))),
          a2f((float)S_.alpha2), sums(v_.fpair + (size_t)4 * v_.N * (threadIdx.x & 1)) {}

    // the pair (i, j): j's force by atomics; i's into the warp's sums where i
    // is `cur`, by atomics otherwise
    __device__ __forceinline__ void pair(int i, int j) {
        // d = p_j - p_i; near the cutoff r^2 is formed again as the list
        // decides (exact_r2)
        const double dx = min_image_bits(__dsub_rn(v.x[j], v.x[i]), L0, h0);
        const double dy = min_image_bits(__dsub_rn(v.y[j], v.y[i]), L1, h1);
        const double dz = min_image_bits(__dsub_rn(v.z[j], v.z[i]), L2, h2);
        const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
        const long long rb = __double_as_longlong(r2);
        if (rb >= near_bits) {
            const double x2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            if (!(x2 < cut2)) return;
        }
        // r^2 to FP32 by its bits (truncated), 1/r from the FP32 estimate y
        // (e = 1 - r^2 y^2 below 2^-20): y (1 + e/2 + 3 e^2 / 8), error e^3
        const int hi = (int)(rb >> 32);
        float r2f = __int_as_float(((hi - 0x38000000) << 3) | (int)((unsigned)rb >> 29));
        double rinv;
        if (hi > 0x39000000 && hi < 0x46000000) {
            const unsigned yb = __float_as_uint(fast_rsqrt(r2f));
            const double y = __hiloint2double((int)((yb >> 3) + 0x38000000u), (int)(yb << 29));
            const double e = fma(-(r2 * y), y, 1.0);
            rinv = fma(y * e, fma(e, 0.375, 0.5), y);
        } else {
            rinv = 1.0 / sqrt(r2);  // outside FP32's range (coinciding atoms among them)
            r2f = (float)r2;
        }
        const double rinv2 = rinv * rinv;
        const double2 li = v.ljd[i], lj = v.ljd[j];
        const double qq = v.qs[i] * v.qs[j];
        const double sr = (li.x + lj.x) * rinv;
        const double s2 = sr * sr;
        const double s6 = s2 * s2 * s2;
        const double es6 = li.y * lj.y * s6;
        double vdw = es6 * fma(12.0, s6, -6.0);  // times 1/r^2 below
        double evdw = (ENERGY || SW) ? fma(es6, s6, -es6) : 0.0;
        if (SW && S.use_switch) {
            const double r = r2 * rinv;
            if (r > sw_dist) {
                const double t = (r - sw_dist) * sw_inv;
                const double sw = 1 + t * t * t * (-10 + t * (15 - t * 6));
                const double dsw = t * t * (-30 + t * (60 - t * 30)) * sw_inv;
                vdw = sw * vdw - evdw * dsw * r;
                evdw *= sw;
            }
        }
        // Ewald (nxm_ewald64.cuh); the rows reach past the cutoff, so the
        // table's end is only for what rounding or a wild r^2 may ask
        const int row = min(ewald_row(r2f * a2f), v.ewald_rows - 1);
        const double *c = v.ewald + kEwaldRow * row;
        const double coul = ewald_term(row, ewald_poly(c, r2, alpha2), alpha3, rinv * rinv2);
        double ecoul = 0.0;
        if (ENERGY) ecoul = ewald_term(row, ewald_poly(c + kEwaldRow * v.ewald_rows, r2, alpha2), S.alpha, rinv);
        const double dEdR = fma(qq, coul, vdw * rinv2);
        const double gx = dx * dEdR, gy = dy * dEdR, gz = dz * dEdR;  // on j
        double *fj = sums + 4 * (size_t)j;
        atomicAdd(fj, gx);
        atomicAdd(fj + 1, gy);
        atomicAdd(fj + 2, gz);
        if (i == cur) {
            fx += gx;
            fy += gy;
            fz += gz;
        } else {
            double *fi = sums + 4 * (size_t)i;
            atomicAdd(fi, negated(gx));
            atomicAdd(fi + 1, negated(gy));
            atomicAdd(fi + 2, negated(gz));
        }
        if (ENERGY) {
            ec = fma(qq, ecoul, ec);
            ev += evdw;
        }
    }

    // the warp's sums to atom `cur`: three sums over 32 lanes in six
    // additions (x and y share lanes from the first step, z from the second)
    __device__ __forceinline__ void flush(int lane) {
        const unsigned full = 0xffffffffu;
        const bool up16 = lane & 16, up8 = lane & 8;
        double a = up16 ? fy : fx;
        a += __shfl_xor_sync(full, up16 ? fx : fy, 16);  // x in lanes 0-15, y in 16-31
        double b = fz + __shfl_xor_sync(full, fz, 16);   // z, both halves alike
        double c = up8 ? b : a;
        c += __shfl_xor_sync(full, up8 ? a : b, 8);      // bit 3 clear: x or y; set: z
        c += __shfl_xor_sync(full, c, 4);
        c += __shfl_xor_sync(full, c, 2);
        c += __shfl_xor_sync(full, c, 1);
        if ((lane & 7) == 0 && lane != 24) atomicAdd(sums + 4 * (size_t)cur + (up8 ? 2 : (up16 ? 1 : 0)), negated(c));
        fx = fy = fz = 0.0;
    }
};

template <bool ENERGY, bool SW>
__global__ void __launch_bounds__(kWarps64 * 32, 2) k_pairs_fp64(DevView v) {
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned full = 0xffffffffu;
    CellGroup G = v.groups[blockIdx.x];
    const int a0 = v.cell_start[G.cell], a1 = v.cell_start[G.cell + G.ncell];
    if (a0 == a1) return;
    const SysDev &S = v.sys[G.sys];
    if (!S.nb_on) return;
    // tile: box fractions and the slot of each atom of the neighbourhood
    int4 *s_u = reinterpret_cast<int4 *>(smem);
    HoodSpan *spans = reinterpret_cast<HoodSpan *>(s_u + v.hood_cap);
    __shared__ int2 s_queue[kWarps64][64];
    __shared__ int4 s_nn;
    __shared__ int s_next;
    {
        const int *src = v.gspan + (size_t)blockIdx.x * kGroupSpanWords;
        int *dst = reinterpret_cast<int *>(spans);
        for (int e = threadIdx.x; e < kGroupSpanWords; e += blockDim.x) dst[e] = src[e];
        if (threadIdx.x == 0) {
            s_nn = v.gspan_n[blockIdx.x];
            s_next = 0;
        }
    }
    __syncthreads();
    const int n = s_nn.x, nsp = s_nn.y;
    if (n > v.hood_cap || nsp > kMaxSpans) {
        if (threadIdx.x == 0) atomicOr(&v.flags->error, ERR_NLIST_OVERFLOW);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = kWarps64;
    for (int sp = warp; sp < nsp; sp += nw) {
        const HoodSpan h = spans[sp];
        for (int t = lane; t < h.count; t += 32) {
            int4 u = v.uf[h.start + t];
            u.w = h.start + t;
            s_u[h.offset + t] = u;
        }
    }
    __syncthreads();
    Pairs64<ENERGY, SW> P(v, S);
    const float ux = S.u2nm[0], uy = S.u2nm[1], uz = S.u2nm[2], pre = S.cut2f_pre;
    int2 *queue = s_queue[warp];
    const unsigned lt = (1u << lane) - 1u;
    int head = 0, tail = 0;  // the queue holds entries head .. tail - 1 (at most 63), entry k at k & 63
    const int q0 = pair_first(a0, G.cell), q1 = pair_first(a1, G.cell + G.ncell);
    // a unit of work: the even or the odd chunks of a pair's list for one of
    // its atoms, taken by the next warp that is free
    for (;;) {
        int t = lane == 0 ? atomicAdd(&s_next, 1) : 0;
        t = __shfl_sync(full, t, 0) * gridDim.y + blockIdx.y;
        const int q = q0 + (t >> 2), second = (t >> 1) & 1;
        if (q >= q1) break;
        const int2 ab = v.ipair[q];
        const int i = second ? ab.y : ab.x;
        if (i < 0) continue;
        const int4 ui = v.uf[i];
        const int cnt = v.ncount[q].x;
        const uint4 *lst4 = reinterpret_cast<const uint4 *>(pair_list(v, q)) + lane;
        P.cur = i;
        for (int c0 = 256 * (t & 1); c0 < cnt; c0 += 512) {
            const uint4 w4 = __ldg(lst4 + c0 / 8);
            const uint32_t wds[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (c0 + 32 * u >= cnt) break;  // warp-uniform
                const unsigned e = (wds[u >> 1] >> (16 * (u & 1))) & 0xffffu;
                // not past the end, not excluded from this atom
                const bool valid = c0 + 32 * u + lane < cnt && !((e >> second) & 1);
                const int4 uj = s_u[valid ? e >> kEntryShift : 0];
                const float dx = (float)(uj.x - ui.x) * ux, dy = (float)(uj.y - ui.y) * uy,
                            dz = (float)(uj.z - ui.z) * uz;
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                const int j = uj.w;
                // each pair from one of its two lists, half of them either way
                const bool mine = (((i ^ j) & 1) != 0) == (i < j);
                const unsigned m = __ballot_sync(full, valid && mine && r2 < pre);
                if ((m >> lane) & 1u) queue[(tail + __popc(m & lt)) & 63] = make_int2(i, j);
                tail += __popc(m);
                if (tail - head >= 32) {
                    __syncwarp();
                    const int2 p = queue[(head + lane) & 63];
                    P.pair(p.x, p.y);
                    head += 32;
                    __syncwarp();
                }
            }
        }
        P.flush(lane);
    }
    P.cur = -1;
    __syncwarp();
    if (head + lane < tail) {
        const int2 p = queue[(head + lane) & 63];
        P.pair(p.x, p.y);
    }
    __syncwarp();
    if (ENERGY) {
        // one word per block and term: the words' rounding (2^-28 kJ/mol) is
        // most of these energies' error
        __shared__ double s_e[2][kWarps64];
        const double ec = warp_sum(P.ec), ev = warp_sum(P.ev);
        if (lane == 0) {
            s_e[0][warp] = ec;
            s_e[1][warp] = ev;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            double e = 0.0;
            for (int w = 0; w < kWarps64; ++w) e += s_e[threadIdx.x][w];
            if (e != 0.0) atomic_add_fixed(&v.E[G.sys * E_SLOTS + (threadIdx.x ? E_VDW : E_COUL)], e, kEnergyScale);
        }
    }
}

// Position of tile entry k in the group's frame, as stage() forms it.
__device__ __forceinline__ void tile_position(const DevView &v, const SysDev &S, const HoodSpan *spans, int nsp, int k,
                                              float p[3]) {
    const int j = hood_slot(spans, nsp, k);
    int sp = 0;
    while (sp + 1 < nsp && spans[sp + 1].offset <= k) ++sp;
    const int c3 = v.cell3[j];
    const float4 D = v.dtab[v.sys_of[j] * kDtabStride + spans[sp].code0 + (((c3 >> 20) & 1023) - spans[sp].cz0)];
    offset_in_cell(v, S, j, c3, p);
    p[0] -= D.x;
    p[1] -= D.y;
    p[2] -= D.z;
}

// ---- test support: the neighbour pair set within the cutoff, exactly as
// the reference decides it, as (larger, smaller) original indices.
__global__ void k_collect(DevView v, int sys_sel, int *out, long long cap, unsigned long long *n_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    CellGroup G = v.groups[blockIdx.x];
    if (G.sys != sys_sel) return;
    int a0 = v.cell_start[G.cell], a1 = v.cell_start[G.cell + G.ncell];
    if (a0 == a1) return;
    const SysDev &S = v.sys[G.sys];
    if (!S.nb_on) return;
    HoodSpan *spans = reinterpret_cast<HoodSpan *>(smem);
    int *s_n = reinterpret_cast<int *>(spans + kMaxSpans);
    hood_setup(v, S, v.cell3[a0], G.ncell, spans, s_n, nullptr);
    if (s_n[1] > kMaxSpans) return;
    int nsp = s_n[1];
    const int kbase = v.gspan_n[blockIdx.x].z;
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int q1 = pair_first(a1, G.cell + G.ncell);
    for (int q = pair_first(a0, G.cell) + warp; q < q1; q += nw) {
        const int2 ab = v.ipair[q];
        if (ab.x < 0) continue;
        const int cnt = v.ncount[q].x;
        for (int k = lane; k < cnt; k += 32) {
            const unsigned e = pair_list(v, q)[list_pos(k)];
            const int j = hood_slot(spans, nsp, (int)(e >> kEntryShift)), oj = v.orig[j];
            // the entry's image of j in the group's frame
            float tj[3];
            tile_position(v, S, spans, nsp, (int)(e >> kEntryShift), tj);
            for (int m = 0; m < 2; ++m) {
                const int i = m ? ab.y : ab.x;
                if (i < 0 || ((e >> m) & 1)) continue;
                const int oi = v.orig[i];
                if (oi <= oj) continue;
                float ti[3];
                tile_position(v, S, spans, nsp, kbase + i, ti);
                bool near = true;
                for (int d = 0; d < 3; ++d) near = near && fabsf(ti[d] - tj[d]) < S.halfLf[d];
                if (!near) continue;  // another image of j, listed for the pair's other atom
                if (!(exact_r2(v, S, i, j) < S.cut2)) continue;
                unsigned long long p = atomicAdd(n_out, 1ull);
                if ((long long)p < cap) {
                    out[2 * p] = oi - S.atom_off;
                    out[2 * p + 1] = oj - S.atom_off;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ launch

static size_t tail_bytes() { return kMaxSpans * sizeof(HoodSpan) + 4 * sizeof(int); }
static size_t smem_build(int cap, int warps) {
    return (size_t)cap * sizeof(float4) + (size_t)warps * kBuildWarpWords * sizeof(uint16_t) +
           25 * (kRowCells + 1) * sizeof(int) + tail_bytes();
}
static size_t smem_pairs(int cap) {
    return (size_t)(cap + kTileSpare) * (sizeof(float4) + sizeof(float2)) + tail_bytes();
}
static size_t smem_pairs64(int cap) { return (size_t)cap * sizeof(int4) + tail_bytes(); }
// static shared memory of the tile kernels (displacement table and counts)
constexpr size_t kTileStatic = 25 * kRowCells * sizeof(float4) + 16;

// Two blocks per SM when both blocks' shared memory fits (228 KB per SM, 1 KB
// reserved per block); otherwise one block of twice the warps, which keeps as
// many on the SM at the same registers per thread.  (Dense neighbourhoods --
// one-cell groups of large cells -- need the latter.)
static bool wide(size_t dynamic_smem) { return 2 * (dynamic_smem + kTileStatic + 1024) > 228 * 1024; }
static int build_warps(int cap) { return wide(smem_build(cap, kHoodWarps)) ? 2 * kHoodWarps : kHoodWarps; }

template <int W>
static void set_build_smem(int b) {
    cudaFuncSetAttribute(k_build<true, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    cudaFuncSetAttribute(k_build<false, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}

// Warps per block of the mixed pair kernel, two blocks per SM (or one of twice
// as many, `wide`): 16 at 64 registers per thread; 14 at 72 or 12 at 80 where
// what the kernel carries (the switch, the energies) would spill.  Measured
// with 16, 14 and 12: the switch at 74,400 atoms 142, 132, 129 us, steps with
// energies 262, 247, 242; without it at 94,100 atoms 133, 134, 133 us, steps
// with energies 0.268, 0.266, 0.269 ms; one block per SM, 32 systems 579, 570,
// 574 us, 473,400 atoms 914, 911, 930.
constexpr int pairs_warps(bool energy, bool sw, bool wide) {
    return sw ? (wide ? 24 : 12) : wide ? 28 : energy ? 14 : 16;
}

template <bool WIDE>
static void set_pairs_smem(int m) {
    auto set = [&](auto kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, m); };
    set(k_pairs_mixed<true, false, pairs_warps(true, false, WIDE)>);
    set(k_pairs_mixed<false, false, pairs_warps(false, false, WIDE)>);
    set(k_pairs_mixed<true, true, pairs_warps(true, true, WIDE)>);
    set(k_pairs_mixed<false, true, pairs_warps(false, true, WIDE)>);
}

// The dynamic shared-memory limit is a per-kernel attribute shared by every
// context of the process on a device: it is only ever raised, so a context
// with a smaller neighbourhood cannot lower it under another one.
void tiles_set_smem(int cap) {
    static std::mutex mu;
    static int seen_build[2][kMaxSmemDevices] = {}, seen_pairs[2][kMaxSmemDevices] = {},
               seen_pairs64[kMaxSmemDevices] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxSmemDevices) dev = 0;
    const int bw = build_warps(cap);
    const int b = (int)smem_build(cap, bw), m = (int)smem_pairs(cap), d = (int)smem_pairs64(cap);
    const int bi = bw == kHoodWarps ? 0 : 1, pi = wide(smem_pairs(cap)) ? 1 : 0;
    std::lock_guard<std::mutex> lock(mu);
    // launches up to 48 KB, static shared memory included, need no attribute
    constexpr int kFree = 48 * 1024 - (int)kTileStatic - 1024;
    if (b > kFree && b > seen_build[bi][dev]) {
        if (bi)
            set_build_smem<2 * kHoodWarps>(b);
        else
            set_build_smem<kHoodWarps>(b);
        seen_build[bi][dev] = b;
    }
    if (m > kFree && m > seen_pairs[pi][dev]) {
        if (pi)
            set_pairs_smem<true>(m);
        else
            set_pairs_smem<false>(m);
        seen_pairs[pi][dev] = m;
    }
    if (d > kFree && d > seen_pairs64[dev]) {
        cudaFuncSetAttribute(k_pairs_fp64<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, d);
        cudaFuncSetAttribute(k_pairs_fp64<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, d);
        cudaFuncSetAttribute(k_pairs_fp64<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, d);
        cudaFuncSetAttribute(k_pairs_fp64<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, d);
        seen_pairs64[dev] = d;
    }
}

template <int W>
static void launch_build_w(const DevView &v, cudaStream_t st) {
    const size_t sm = smem_build(v.hood_cap, W);
    if (v.mixed)
        k_build<true, W><<<v.ngroups, W * 32, sm, st>>>(v);
    else
        k_build<false, W><<<v.ngroups, W * 32, sm, st>>>(v);
}

void launch_build(const DevView &v, cudaStream_t st) {
    if (!v.ngroups) return;
    if (build_warps(v.hood_cap) == kHoodWarps)
        launch_build_w<kHoodWarps>(v, st);
    else
        launch_build_w<2 * kHoodWarps>(v, st);
}

template <bool ENERGY, bool SW, bool WIDE>
static void launch_pairs_variant(const DevView &v, cudaStream_t st) {
    constexpr int W = pairs_warps(ENERGY, SW, WIDE);
    k_pairs_mixed<ENERGY, SW, W><<<v.ngroups, W * 32, smem_pairs(v.hood_cap), st>>>(v);
}

template <bool WIDE>
static void launch_pairs_mixed(const DevView &v, int energy, cudaStream_t st) {
    if (v.any_switch)
        energy ? launch_pairs_variant<true, true, WIDE>(v, st) : launch_pairs_variant<false, true, WIDE>(v, st);
    else
        energy ? launch_pairs_variant<true, false, WIDE>(v, st) : launch_pairs_variant<false, false, WIDE>(v, st);
}

void launch_pairs(const DevView &v, int energy, cudaStream_t st) {
    if (v.N == 0 || v.ngroups == 0) return;
    if (v.mixed) {
        if (wide(smem_pairs(v.hood_cap)))
            launch_pairs_mixed<true>(v, energy, st);
        else
            launch_pairs_mixed<false>(v, energy, st);
        return;
    }
    // A group's atoms may be dealt to several blocks, each staging the
    // neighbourhood for itself: as many blocks as make the busiest SM's share
    // of the atoms least (the pipe that bounds the kernel belongs to the SM,
    // so its time is its atoms, however many blocks hold them).  23,800
    // atoms, 484 groups on 152 SMs: 652 us with one block per group, 567 so
    // (554 since, by fewer additions per pair).
    const int per = (v.N + v.ngroups - 1) / v.ngroups;
    int parts = 1, best = 1 << 30;
    for (int p = 1; p <= (per + kWarps64 - 1) / kWarps64; ++p) {
        const long long rounds = ((long long)v.ngroups * p + kSMs - 1) / kSMs;
        const int cost = (int)std::min<long long>(rounds * ((per + p - 1) / p), 1 << 29);
        if (cost <= best) {
            best = cost;
            parts = p;
        }
    }
    const dim3 g(v.ngroups, parts);
    const int t = kWarps64 * 32;
    const size_t sm = smem_pairs64(v.hood_cap);
    if (v.any_switch) {
        if (energy)
            k_pairs_fp64<true, true><<<g, t, sm, st>>>(v);
        else
            k_pairs_fp64<false, true><<<g, t, sm, st>>>(v);
    } else {
        if (energy)
            k_pairs_fp64<true, false><<<g, t, sm, st>>>(v);
        else
            k_pairs_fp64<false, false><<<g, t, sm, st>>>(v);
    }
}

long long launch_collect_pairs(const DevView &v, int sys, int *out_pairs, long long cap, cudaStream_t st) {
    unsigned long long *dn;
    cudaMallocAsync(&dn, sizeof(unsigned long long), st);
    cudaMemsetAsync(dn, 0, sizeof(unsigned long long), st);
    k_collect<<<v.ngroups, kHoodWarps * 32, tail_bytes(), st>>>(v, sys, out_pairs, cap, dn);
    unsigned long long n = 0;
    cudaMemcpyAsync(&n, dn, sizeof(n), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    cudaFreeAsync(dn, st);
    return (long long)n;
}

}  // namespace nxm
