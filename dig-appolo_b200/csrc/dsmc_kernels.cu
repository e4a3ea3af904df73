// The DSMC step kernels.
//
//   inject   preprocesseffquad (src/ProcessDSMC.cpp:2556-2570): per-cell
//            inflow counts with the reference's remainder carry, scan,
//            per-patch particle generation + trace for r*dt.
//   move     advection (src/ProcessDSMC.cpp:1946-2017): lanes trace
//            particles for dtime through the mesh, refilled from warp
//            chunks as their particles finish.
//   sort     cache2chain (src/ProcessDSMC.cpp:2030-2135): deterministic
//            counting sort. rank (warp per source cell: arrival slot and rank
//            from warp ballots; multi-hop and injected arrivals through
//            warp-aggregated atomics), scan, scatter of source indices, the
//            far arrivals put in source order, gather of the particles.
//   collide  collisionDSMC (src/ProcessDSMC.cpp:2621-2744): cells classed
//            by size; NTC candidate pairs in sequence per cell (claims keep
//            the reference's pair order), accepted pairs run together.
//   sample   statistic_macro (src/ProcessDSMC.cpp:2757-2861): the
//            18-moment sums of each cell in particle order.
#include <climits>
#include <cstddef>
#include <type_traits>

#include "dsmc_kernels.cuh"
#include "dsmc_macro.cuh"

namespace dsmc {

constexpr unsigned kFull = 0xffffffffu;


// Particle positions between HBM and the trace's FP64 registers: the FP64
// path stores absolute FP64; the mixed path stores FP32 offsets from the
// centre of the particle's cell (widened as centre + offset, stored as the
// FP32 rounding of position - centre).
template <typename Real, int kFaces = 0>
__device__ __forceinline__ void load_position(const DevMesh& M, const PBuf<Real>& B, int i, int cell, PRegs<Real>& p)
{
    if constexpr (sizeof(Real) == 8) {
        p.x[0] = B.x[0][i]; p.x[1] = B.x[1][i]; p.x[2] = B.x[2][i];
    } else {
        const double* cc = cell_centre<kFaces>(M, cell);
        p.x[0] = da(__ldg(cc), (double)B.x[0][i]);
        p.x[1] = da(__ldg(cc + 1), (double)B.x[1][i]);
        p.x[2] = da(__ldg(cc + 2), (double)B.x[2][i]);
    }
}

template <typename Real, int kFaces = 0>
__device__ __forceinline__ void store_position(const DevMesh& M, const PBuf<Real>& B, int i, int cell,
                                               const PRegs<Real>& p)
{
    if constexpr (sizeof(Real) == 8) {
        B.x[0][i] = p.x[0]; B.x[1][i] = p.x[1]; B.x[2][i] = p.x[2];
    } else {
        if (cell < 0 || cell >= M.ncell) return;   // removed: the slot is not read again
        const double* cc = cell_centre<kFaces>(M, cell);
        B.x[0][i] = (float)ds(p.x[0], __ldg(cc + 0));
        B.x[1][i] = (float)ds(p.x[1], __ldg(cc + 1));
        B.x[2][i] = (float)ds(p.x[2], __ldg(cc + 2));
    }
}

// The mesh's kind for the kernels that trace: the record stride when the exit
// search unrolls over it (tetrahedra 4, pyramids and wedges 5, hexahedra 6),
// else 0. Each kernel holds one kind's search only: with all of them in one
// kernel it ran slower than unrolling gained (372,500 tetrahedra: the
// tracing pass 960 -> 1146 us), its code no longer fitting the instruction
// cache.
inline int face_kind(const DevMesh& M) { return M.faceStride >= 4 && M.faceStride <= 6 ? M.faceStride : 0; }

// f(integral constant of the kind)
template <typename F>
inline void with_face_kind(const DevMesh& M, F&& f)
{
    switch (face_kind(M)) {
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        default: f(std::integral_constant<int, 0>{}); break;
    }
}

size_t geo_floats(const DevMesh& M)
{
    const int f = face_kind(M);
    return f == 0 ? 0 : f == 6 ? CellGeo<6>::kFloats : CellGeo<4>::kFloats;
}

template <int kFaces>
__global__ void pack_geo_kernel(DevMesh M, float4* geo)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < M.ncell; c += gridDim.x * blockDim.x) {
        float4* g = geo + (size_t)c * (CellGeo<kFaces>::kFloats / 4);
        for (int j = 0; j < kFaces; ++j) g[j] = M.planeF[(size_t)c * kFaces + j];
        double* cc = reinterpret_cast<double*>(g + kFaces);
        for (int d = 0; d < 3; ++d) cc[d] = M.cellCenter[(size_t)c * 3 + d];
        float* f = reinterpret_cast<float*>(g + kFaces);
        f[6] = M.recAux[(size_t)c * kFaces].y;
        for (int j = 0; j < kFaces; ++j) f[7 + j] = M.recAux[(size_t)c * kFaces + j].x;
    }
}

void launch_pack_geo(const DevMesh& M, float4* geo, cudaStream_t s)
{
    const int g = (M.ncell + 255) / 256;
    with_face_kind(M, [&](auto f) {
        constexpr int F = decltype(f)::value;
        if constexpr (F > 0) pack_geo_kernel<F><<<g < 2048 ? g : 2048, 256, 0, s>>>(M, geo);
    });
}

// ===========================================================================
// inject
// ===========================================================================
__global__ void inject_count_kernel(DevPatches P, double* remInj)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < P.ngroup; g += gridDim.x * blockDim.x) {
        const int b = P.groupStart[g];
        const int e = P.groupStart[g + 1];
        const int cell = P.cell[b];
        double rem = remInj[cell];
        // computeBoundaryInsertCount, src/ProcessDSMC.cpp:2398-2402
        for (int p = b; p < e; ++p) {
            const double addNum = da(P.addBase[p], rem);
            const double fl = floor(addNum);
            const int n = (int)fl;
            rem = ds(addNum, (double)n);
            P.count[p] = n;
        }
        remInj[cell] = rem;
    }
}

__global__ void __launch_bounds__(1024) inject_scan_kernel(DevPatches P, StepCtl* ctl, unsigned long long* counters)
{
    __shared__ int warpSum[32];
    __shared__ int carry;
    const int tid = threadIdx.x;
    const int lane = tid & 31, wid = tid >> 5;
    const int room = ctl->capacity - ctl->nLive;
    if (tid == 0) carry = 0;
    long long over = 0;
    __syncthreads();
    for (int base = 0; base < P.npatch; base += blockDim.x) {
        const int i = base + tid;
        const int v = (i < P.npatch) ? P.count[i] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warpSum[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int w = (lane < (int)(blockDim.x >> 5)) ? warpSum[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, w, o);
                if (lane >= o) w += y;
            }
            warpSum[lane] = w;
        }
        __syncthreads();
        const int incl = x + (wid > 0 ? warpSum[wid - 1] : 0);
        const int start = carry + incl - v;
        if (i < P.npatch) {
            P.start[i] = start;
            int allowed = room - start;
            allowed = allowed < 0 ? 0 : (allowed > v ? v : allowed);
            if (allowed < v) {
                over += v - allowed;
                P.count[i] = allowed;
            }
        }
        __syncthreads();
        if (tid == blockDim.x - 1) carry += incl;
        __syncthreads();
    }
    if (over) atomicAdd(counters + C_OVERFLOW, (unsigned long long)over);
    __syncthreads();
    if (tid == 0) {
        const int m = carry < room ? carry : (room > 0 ? room : 0);
        ctl->nInj = m;
        atomicAdd(counters + C_INJECTED, (unsigned long long)m);
    }
}

// sampleBoundaryParticle, src/ProcessDSMC.cpp:2416-2458: normal speed by
// acceptance-rejection against the fs1/fs2 envelope, tangential components by
// Box-Muller, rotational energy -ln(r) T / 2, all in the patch frame.
__device__ __forceinline__ void sample_inflow_velocity(const double* gas, const double* R, Stream& rs,
                                                       double v[3], double& ir, int* errorWord)
{
    const double snp = gas[0], fs1 = gas[1], fs2 = gas[2], stp1 = gas[3], stp2 = gas[4];
    const double tN = gas[5], sq = gas[6], QA = gas[7];
    double vzr = 0.0, vza = 0.0;
    for (int outer = 0;; ++outer) {
        for (int inner = 0;; ++inner) {
            const double r = rs.uniform64();
            vzr = (-QA + 2.0 * QA * r) * sq;
            vza = vzr / sq + snp;
            if (vza > 0) break;
            if (inner > (1 << 20)) { atomicOr(errorWord, kErrRejectLoop); vza = 1e-3; break; }
        }
        const double vzn = vzr / sq;
        const double pp = (2.0 * vza / fs1) * exp(fs2 - vzn * vzn);
        if (rs.uniform64() < pp) break;
        if (outer > (1 << 20)) { atomicOr(errorWord, kErrRejectLoop); break; }
    }
    const double r = rs.uniform64();
    const double th = rs.uniform64();
    double s, c;
    sincospi(2.0 * th, &s, &c);
    const double a = sqrt(-log(r));
    const double vxa = (a * s + stp1) * sq;
    const double vya = (a * c + stp2) * sq;
    vza *= sq;
    v[0] = R[0] * vxa + R[1] * vya + R[2] * vza;
    v[1] = R[3] * vxa + R[4] * vya + R[5] * vza;
    v[2] = R[6] * vxa + R[7] * vya + R[8] * vza;
    ir = -log(rs.uniform64()) * tN * 0.5;
}

// One thread per injected particle; its patch is found by binary search in
// the exclusive scan of the per-patch counts (slots of one patch are
// consecutive, so a warp mostly works on one patch).
template <typename Real, int kFaces>
__global__ void __launch_bounds__(128) inject_gen_kernel(StepArgs<Real> a)
{
    __shared__ ExitHit scanned[128];
    const int istep = a.ctl->istep;
    const int nLive = a.ctl->nLive;
    const int m = a.ctl->nInj;
    const int np = a.P.npatch;
    TraceCounts cnt{};
    const int lane = threadIdx.x & 31;
    // whole warps, the lanes past the end with a copy of the last particle
    // that is not stored (they take part in the warp's traces)
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < m; base += gridDim.x * blockDim.x) {
        const bool mine = base + lane < m;
        const int slot = min(base + lane, m - 1);
        int lo = 0, hi = np - 1;          // last patch with start <= slot
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.P.start[mid] <= slot) lo = mid; else hi = mid - 1;
        }
        const int p = lo;
        const int pcell = a.P.cell[p];
        const int pedge = a.P.edge[p];
        const int ptag = a.P.triTag[p];
        const double* G = a.P.geom + (size_t)p * 9;
        const double* R = a.P.rot + (size_t)p * 9;
        const double* gas = a.P.gas + (size_t)p * 8;
        const int gi = nLive + slot;
        Stream rs;
        rs.init((uint32_t)gi, (uint32_t)istep, kPurposeInject, a.C.seedLo, a.C.seedHi);
        double u = rs.uniform64(), w = rs.uniform64();
        if (u + w > 1.0) { u = 1.0 - u; w = 1.0 - w; }
        double pos[3];
        // p0 + u e10 + v e20 (src/ProcessDSMC.cpp:2524-2526), unfused
        for (int d = 0; d < 3; ++d) pos[d] = da(da(G[d], dm(u, G[3 + d])), dm(w, G[6 + d]));
        double vel[3], irv;
        sample_inflow_velocity(gas, R, rs, vel, irv, a.errorWord);
        double dtleft = rs.uniform64() * a.C.dtime;
        PRegs<Real> pr;
        int cell = pcell;
        for (int d = 0; d < 3; ++d) pr.x[d] = pos[d];
        for (int d = 0; d < 3; ++d) pr.v[d] = (Real)vel[d];
        pr.ir = (Real)irv;
        const int out = trace_particle_warp<Real, kFaces>(mine, a.M, a.C, pr, cell, pedge, ptag, dtleft, rs, istep,
                                                          a.wallTally, cnt, &scanned[threadIdx.x]);
        if (!mine) continue;
        store_position<Real, kFaces>(a.M, a.A, gi, cell, pr);
        a.A.v[0][gi] = pr.v[0]; a.A.v[1][gi] = pr.v[1]; a.A.v[2][gi] = pr.v[2];
        a.A.ir[gi] = pr.ir;
        a.A.cell[gi] = (out >= 0) ? cell : -1;
    }
    flush_counts(a.counters, cnt);
}

template <typename Real>
void launch_inject(const StepArgs<Real>& a, const LaunchShape& L, cudaStream_t s)
{
    if (a.P.npatch == 0) {
        cudaMemsetAsync(&a.ctl->nInj, 0, sizeof(int), s);
        return;
    }
    const int gCount = (a.P.ngroup + 127) / 128;
    inject_count_kernel<<<gCount > 0 ? gCount : 1, 128, 0, s>>>(a.P, a.remInj);
    inject_scan_kernel<<<1, 1024, 0, s>>>(a.P, a.ctl, a.counters);
    // one particle a thread at the expected count (a remainder can add one per patch)
    const int gGen = max(1, min(L.smCount * 8, (a.P.expected + 127) / 128));
    with_face_kind(a.M, [&](auto f) { inject_gen_kernel<Real, decltype(f)::value><<<gGen, 128, 0, s>>>(a); });
}

// ===========================================================================
// move
// ===========================================================================
// Two passes over the particles of the step.
//
// Stay pass (move_stay_kernel): one thread per particle, in slot order
// (coalesced loads, the particles of a cell next to each other, so a warp
// reads few cells' face records). Most particles stay in their cell for the
// whole step; where the first exit search settles that (stays_for_the_step)
// the particle is advanced and stored right there. The others are appended
// to a work list (in the sort's rank array, which is free until the sort),
// with their state copied to the same positions of the other particle buffer
// (free until the sort too): the tracing pass then reads its particles in list
// order instead of gathering them from sparse slots. A block takes its share
// of the list with one atomic for up to 1,024 particles: with one per warp
// and 32 particles, the million atomics on one address were the pass (37M
// particles: 974 us, 634 with one per block). It then waits for the cells'
// geometry.
//
// Tracing pass (move_kernel): the listed particles, traced from their start
// by trace_step. Warps claim chunks of 128 list entries from a cursor in
// the step control block (one atomic per chunk), and a lane whose particle
// has finished writes it back and takes the next particle of the chunk, so
// the lanes keep doing exit searches instead of waiting for the warp's
// longest trace. A list too short for that gives every warp an equal share
// instead, down to 8 entries: a warp that refilled its lanes while others had
// none would only add its rounds to the pass's latency (19,700 particles: 69
// -> 27 us). Three resident 256-thread blocks per SM (registers capped at 85):
// the trace is bound by dependent loads, so occupancy pays more than the few
// registers it spills to L1.
//
// Each particle runs the same code with its own random stream (particle
// index, step), and the stay pass takes exactly the decision the trace's
// first search takes, so results do not depend on the split, the list
// order, or which lane or warp traces a particle.
constexpr int kMoveChunk = 128;
constexpr int kMoveChunkMin = 8;

// K particles per thread (K x 256 consecutive slots per block and round):
// the loads of all K are issued before the first decision.
template <typename Real, int K, int kFaces>
__global__ void __launch_bounds__(256) move_stay_kernel(StepArgs<Real> a)
{
    __shared__ int sCount[2], sBase;
    const int n = a.ctl->nLive;
    const double dt = a.C.dtime;
    const int lane = threadIdx.x & 31;
    int parity = 0;
    if (threadIdx.x < 2) sCount[threadIdx.x] = 0;
    __syncthreads();
    // a step with fewer slots than K a thread takes as many as give every
    // thread its share, rather than K on few of them
    const int per = min(K, (n + (int)(gridDim.x * blockDim.x) - 1) / (int)(gridDim.x * blockDim.x));
    const int tile = per * (int)blockDim.x;
    for (int base = blockIdx.x * tile; base < n; base += gridDim.x * tile) {
        int cell[K];
        Real xs[K][3];
        PRegs<Real> p[K];
        // the slot's own loads first, all of them independent of each other
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = base + k * (int)blockDim.x + (int)threadIdx.x;
            if (i < n && k < per) {
                cell[k] = a.A.cell[i];
                xs[k][0] = a.A.x[0][i]; xs[k][1] = a.A.x[1][i]; xs[k][2] = a.A.x[2][i];
                p[k].v[0] = a.A.v[0][i]; p[k].v[1] = a.A.v[1][i]; p[k].v[2] = a.A.v[2][i];
            } else {
                cell[k] = -1;
            }
        }
        // the decisions: stayers advanced and stored, the others counted
        unsigned defer = 0u;
        int before[K], mine = 0;   // the warp's deferred ones before this lane's of set k
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = base + k * (int)blockDim.x + (int)threadIdx.x;
            bool d = false;
            if (cell[k] >= 0) {
                // the position as load_position widens it
                if constexpr (sizeof(Real) == 8) {
                    p[k].x[0] = xs[k][0]; p[k].x[1] = xs[k][1]; p[k].x[2] = xs[k][2];
                } else {
                    const double* cc = cell_centre<kFaces>(a.M, cell[k]);
                    p[k].x[0] = da(__ldg(cc + 0), (double)xs[k][0]);
                    p[k].x[1] = da(__ldg(cc + 1), (double)xs[k][1]);
                    p[k].x[2] = da(__ldg(cc + 2), (double)xs[k][2]);
                }
                if (stays_for_the_step<Real, kFaces>(a.M, cell[k], xs[k], p[k], dt)) {
                    advance(p[k], dt);
                    store_position<Real, kFaces>(a.M, a.A, i, cell[k], p[k]);
                } else {
                    d = true;
                }
            }
            const unsigned m = __ballot_sync(kFull, d);
            before[k] = mine + __popc(m & ((1u << lane) - 1u));
            mine += __popc(m);
            if (d) defer |= 1u << k;
        }
        // the block's share of the list: one atomic for all of its warps
        int at = 0;
        if (lane == 0 && mine) at = atomicAdd(&sCount[parity], mine);
        __syncthreads();
        if (threadIdx.x == 0) {
            const int c = sCount[parity];
            sBase = c ? atomicAdd(&a.ctl->moveList, c) : 0;
            sCount[parity ^ 1] = 0;
        }
        __syncthreads();
        at = sBase + __shfl_sync(kFull, at, 0);
        parity ^= 1;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((defer >> k) & 1u)) continue;
            // the entry: the slot, and the particle's state in the other
            // buffer (free until the sort) at the same position, so the
            // tracing pass reads it in list order
            const int i = base + k * (int)blockDim.x + (int)threadIdx.x;
            const int j = at + before[k];
            a.rank[j] = i;
            a.B.cell[j] = cell[k];
            a.B.x[0][j] = xs[k][0]; a.B.x[1][j] = xs[k][1]; a.B.x[2][j] = xs[k][2];
            a.B.v[0][j] = p[k].v[0]; a.B.v[1][j] = p[k].v[1]; a.B.v[2][j] = p[k].v[2];
            a.B.ir[j] = a.A.ir[i];
        }
    }
}

template <typename Real, int kFaces>
__global__ void __launch_bounds__(256, 3) move_kernel(StepArgs<Real> a)
{
    const int istep = a.ctl->istep;
    const int n = a.ctl->moveList;
    const int* __restrict__ list = a.rank;
    const int lane = threadIdx.x & 31;
    const unsigned lower = (1u << lane) - 1u;
    TraceCounts cnt{};
    const double dt0 = a.C.dtime;
    const int warps = (int)(gridDim.x * blockDim.x) >> 5;
    const int chunk = max(kMoveChunkMin, min(kMoveChunk, (n + warps - 1) / warps));
    int chunkNext = 0, chunkEnd = 0;   // this warp's chunk (warp-uniform)
    bool exhausted = false;            // warp-uniform
    int i = -1;                        // this lane's particle
    PRegs<Real> p;
    int cell = 0;
    double dtleft = 0;
    TraceState st;
    // the particle's wall draws; the mixed path's in one register (drawn a
    // re-emission at a time, from block 0)
    using Rng = typename std::conditional<sizeof(Real) == 4, BlockStream, Stream>::type;
    Rng rs;
    uint32_t wallBefore = 0;
    for (;;) {
        unsigned want = __ballot_sync(kFull, i < 0);
        while (want && !exhausted) {
            if (chunkNext >= chunkEnd) {
                int base = 0;
                if (lane == 0) base = atomicAdd(&a.ctl->moveCursor, chunk);
                base = __shfl_sync(kFull, base, 0);
                if (base >= n) {
                    exhausted = true;
                    break;
                }
                chunkNext = base;
                chunkEnd = min(base + chunk, n);
            }
            const int take = min(chunkEnd - chunkNext, __popc(want));
            const bool mine = ((want >> lane) & 1u) && __popc(want & lower) < take;
            if (mine) {
                // the entry's slot and state, as the stay pass wrote them
                const int j = chunkNext + __popc(want & lower);
                i = list[j];
                cell = a.B.cell[j];
                load_position<Real, kFaces>(a.M, a.B, j, cell, p);
                p.v[0] = a.B.v[0][j]; p.v[1] = a.B.v[1][j]; p.v[2] = a.B.v[2][j];
                p.ir = a.B.ir[j];
                if constexpr (sizeof(Real) == 4) rs.init((uint32_t)i, (uint32_t)istep, kPurposeWall);
                else rs.init((uint32_t)i, (uint32_t)istep, kPurposeWall, a.C.seedLo, a.C.seedHi);
                dtleft = dt0;
                st.begin(-1, -1);
                wallBefore = cnt.wall;
            }
            chunkNext += take;
            want &= ~__ballot_sync(kFull, mine);
        }
        const bool active = i >= 0;
        if (!__any_sync(kFull, active)) break;
        if (active && trace_step<Real, Rng, kFaces, false>(a.M, a.C, p, cell, dtleft, st, rs, istep, a.wallTally, cnt,
                                                           false, nullptr)) {
            if (st.ifout >= 0) {
                store_position<Real, kFaces>(a.M, a.A, i, cell, p);
                if (cnt.wall != wallBefore) {
                    a.A.v[0][i] = p.v[0]; a.A.v[1][i] = p.v[1]; a.A.v[2][i] = p.v[2];
                    a.A.ir[i] = p.ir;
                }
                a.A.cell[i] = cell;
            } else {
                a.A.cell[i] = -1;
            }
            i = -1;
        }
    }
    flush_counts(a.counters, cnt);
}

// resident blocks per SM of the stay pass (1, 2, 4 particles per thread) by
// kind, set by prepare_kernels
template <typename Real>
struct StayOcc {
    static int blocks[7][3];
};
template <typename Real>
int StayOcc<Real>::blocks[7][3];

template <typename Real>
cudaError_t prepare_move()
{
    cudaError_t e = cudaSuccess;
    auto blocks = [&](const void* k, int threads, int& out) {
        int nb = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, threads, 0);
        out = nb > 0 ? nb : 1;
    };
    auto kind = [&](auto f) {
        constexpr int F = decltype(f)::value;
        blocks((const void*)move_stay_kernel<Real, 1, F>, 256, StayOcc<Real>::blocks[F][0]);
        blocks((const void*)move_stay_kernel<Real, 2, F>, 256, StayOcc<Real>::blocks[F][1]);
        blocks((const void*)move_stay_kernel<Real, 4, F>, 256, StayOcc<Real>::blocks[F][2]);
    };
    kind(std::integral_constant<int, 0>{});
    kind(std::integral_constant<int, 4>{});
    kind(std::integral_constant<int, 5>{});
    kind(std::integral_constant<int, 6>{});
    return e;
}

template <typename Real>
void launch_move(const StepArgs<Real>& a, const LaunchShape& L, cudaStream_t s)
{
    static_assert(offsetof(StepCtl, moveList) == offsetof(StepCtl, moveCursor) + sizeof(int),
                  "the move's cursor and list count are reset together");
    cudaMemsetAsync(&a.ctl->moveCursor, 0, 2 * sizeof(int), s);
    with_face_kind(a.M, [&](auto f) {
        constexpr int F = decltype(f)::value;
        // one wave: every block resident (the blocks split the slots evenly,
        // so a second, partial wave would run at a fraction of the occupancy)
        const int* occ = StayOcc<Real>::blocks[F];
        if (L.stayPerThread == 4) move_stay_kernel<Real, 4, F><<<L.smCount * occ[2], 256, 0, s>>>(a);
        else if (L.stayPerThread == 2) move_stay_kernel<Real, 2, F><<<L.smCount * occ[1], 256, 0, s>>>(a);
        else move_stay_kernel<Real, 1, F><<<L.smCount * occ[0], 256, 0, s>>>(a);
        move_kernel<Real, F><<<L.smCount * L.moveBlocksPerSm, L.moveThreads, 0, s>>>(a);
    });
}

// advance the step counter on the device (batched steps, where the graph
// carries no host-written step number)
__global__ void bump_istep_kernel(StepCtl* ctl) { ctl->istep += 1; }

void launch_bump_istep(StepCtl* ctl, cudaStream_t s) { bump_istep_kernel<<<1, 1, 0, s>>>(ctl); }

// ===========================================================================
// sort: rank, scan, scatter
// ===========================================================================
// rank_kernel, a warp per cell: where each particle of the cell goes (the cell
// itself, a neighbour by its face, or further) and its place among those of
// the cell that go there. Bound by instruction issue in a large mesh and by the
// latency of a cell's slots and ids in a small one. The destination is a
// number of three bits: three ballots give every lane its fellows, and lane q
// holds destination q's count (a ballot per destination, and the counts in
// every lane, took twice the instructions). One wave of resident blocks, each
// warp reading the next cell's slots and neighbours ahead. 37M particles:
// 248 -> 207 us; 6,080 cells at 85: 15.6 -> 12.6 (16 blocks an SM: 212, 12.3).
constexpr int kRankPerSm = 5;
template <typename Real>
__global__ void __launch_bounds__(256, kRankPerSm) rank_kernel(StepArgs<Real> a)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int ncell = a.M.ncell;
    const unsigned lt = (1u << lane) - 1u;
    // the lanes whose destination is this lane's: the three ballots of the
    // destinations' bits, each complemented where this lane's bit is 0
    const unsigned l0 = (lane & 1) ? 0u : kFull, l1 = (lane & 2) ? 0u : kFull, l2 = (lane & 4) ? 0u : kFull;
    // a cell's slots and neighbours, read one cell ahead
    int bN = 0, eN = 0, nbN = -1, rvN = -1;
    auto ahead = [&](int s) {
        if (s >= ncell) return;
        bN = a.startA[s];
        eN = a.startA[s + 1];
        if (lane < 6) {
            nbN = a.M.cell2cell[(size_t)s * 6 + lane];
            rvN = (int)a.M.revSlot[(size_t)s * 6 + lane];
        }
    };
    ahead(warp);
    for (int s = warp; s < ncell; s += nwarps) {
        const int b = bN, e = eN, nbL = nbN, rvL = rvN;
        ahead(s + nwarps);
        const int nbPrev = __shfl_up_sync(kFull, nbL, 1);
        const int rvPrev = __shfl_up_sync(kFull, rvL, 1);
        int nbr[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) nbr[j] = __shfl_sync(kFull, nbL, j);
        // lane q <= 6: destination q's slot, and below it how many went there
        int run = lane >= 1 && lane <= 6 ? (rvPrev + 1) << 24 : 0;
        // the cell ids of up to 128 particles loaded first, then ranked 32 at
        // a time
        for (int base4 = b; base4 < e; base4 += 128) {
            int dq[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = base4 + 32 * u + lane;
                dq[u] = i < e ? a.A.cell[i] : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int base = base4 + 32 * u;
                if (base >= e) break;
                const int i = base + lane;
                const int d = dq[u];
                // destination: 0 the cell itself, 1..6 a neighbour, 7 another
                // cell, or removed
                int q = 7;
                if (d >= 0) {
#pragma unroll
                    for (int j = 5; j >= 0; --j)
                        if (d == nbr[j]) q = j + 1;
                    if (d == s) q = 0;
                }
                const unsigned b0 = __ballot_sync(kFull, q & 1), b1 = __ballot_sync(kFull, q & 2),
                               b2 = __ballot_sync(kFull, q & 4);
                const unsigned same = ((q & 1) ? b0 : ~b0) & ((q & 2) ? b1 : ~b1) & ((q & 4) ? b2 : ~b2);
                int packed = __shfl_sync(kFull, run, q) + __popc(same & lt);
                run += __popc((b0 ^ l0) & (b1 ^ l1) & (b2 ^ l2));
                if (q == 7) {
                    // multi-cell hops (a few percent): a slot each; their order
                    // is made canonical after the scatter
                    packed = -1;
                    if (d >= 0) packed = (kFarSlot << 24) | atomicAdd(a.countSlot + (size_t)d * kSlots + kFarSlot, 1);
                }
                if (i < e) a.rank[i] = packed;
            }
        }
        const int myRun = run & 0xFFFFFF;
        if (lane == 0) {
            a.countSlot[(size_t)s * kSlots] = myRun;
        } else if (lane <= 6) {
            if (nbPrev >= 0 && nbPrev < ncell && rvPrev >= 0) a.countSlot[(size_t)nbPrev * kSlots + rvPrev + 1] = myRun;
        }
    }
    // injected particles: all arrive through the far slot
    const int nLive = a.ctl->nLive;
    const int nTot = nLive + a.ctl->nInj;
    for (int base = nLive + warp * 32; base < nTot; base += nwarps * 32) {
        const int i = base + lane;
        const int d = (i < nTot) ? a.A.cell[i] : -1;
        const int key = d >= 0 ? d * kSlots + kFarSlot : -1;
        const int r = warp_claim(a.countSlot, key);
        if (i < nTot && d >= 0) a.rank[i] = (kFarSlot << 24) | r;
    }
}

__device__ __forceinline__ int row_total(const int* countSlot, int c)
{
    const int4 lo = *reinterpret_cast<const int4*>(countSlot + (size_t)c * kSlots);
    const int4 hi = *reinterpret_cast<const int4*>(countSlot + (size_t)c * kSlots + 4);
    return lo.x + lo.y + lo.z + lo.w + hi.x + hi.y + hi.z + hi.w;
}

__device__ __forceinline__ int block_sum(int v, int* sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    int t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    __syncthreads();
    if (threadIdx.x == 0) sh[0] = t;
    __syncthreads();
    const int r = sh[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(256) scan_partial_kernel(const int* countSlot, int ncell, int* partial)
{
    __shared__ int sh[32];
    const int chunk = (ncell + gridDim.x - 1) / gridDim.x;
    const int b = blockIdx.x * chunk;
    const int e = min(ncell, b + chunk);
    int s = 0;
    for (int c = b + threadIdx.x; c < e; c += blockDim.x) s += row_total(countSlot, c);
    s = block_sum(s, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) scan_final_kernel(const int* countSlot, int ncell, const int* partial,
                                                         int* start, StepCtl* ctl)
{
    __shared__ int sh[32];
    __shared__ int warpSum[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int pre = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) pre += partial[k];
    int carry = block_sum(pre, sh);
    const int chunk = (ncell + gridDim.x - 1) / gridDim.x;
    const int b = blockIdx.x * chunk;
    const int e = min(ncell, b + chunk);
    for (int base = b; base < e; base += blockDim.x) {
        const int c = base + threadIdx.x;
        const int v = (c < e) ? row_total(countSlot, c) : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warpSum[wid] = x;
        __syncthreads();
        int off = 0;
        for (int w = 0; w < wid; ++w) off += warpSum[w];
        int tileTotal = 0;
        for (int w = 0; w < 8; ++w) tileTotal += warpSum[w];
        if (c < e) start[c] = carry + off + x - v;
        __syncthreads();
        carry += tileTotal;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        start[ncell] = carry;
        ctl->nNext = carry;
    }
}

template <typename Real>
__global__ void __launch_bounds__(256) scatter_kernel(StepArgs<Real> a)
{
    // four particles per thread, their loads issued before their stores
    constexpr int U = 4;
    const int nTot = a.ctl->nLive + a.ctl->nInj;
    const int stride = gridDim.x * blockDim.x;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < nTot; i0 += U * stride) {
        int d[U], packed[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * stride;
            d[u] = i < nTot ? a.A.cell[i] : -1;
            packed[u] = i < nTot ? a.rank[i] : 0;
        }
        int4 lo[U], hi[U];
        int s0[U], s1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (d[u] < 0) continue;
            lo[u] = *reinterpret_cast<const int4*>(a.countSlot + (size_t)d[u] * kSlots);
            hi[u] = *reinterpret_cast<const int4*>(a.countSlot + (size_t)d[u] * kSlots + 4);
            s0[u] = a.startB[d[u]];
            s1[u] = a.startB[d[u] + 1];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (d[u] < 0) continue;
            const int slot = packed[u] >> 24;
            int base = s0[u] + (packed[u] & 0xFFFFFF);
            if (slot > 0) base += lo[u].x;
            if (slot > 1) base += lo[u].y;
            if (slot > 2) base += lo[u].z;
            if (slot > 3) base += lo[u].w;
            if (slot > 4) base += hi[u].x;
            if (slot > 5) base += hi[u].y;
            if (slot > 6) base += hi[u].z;
            if (base < s0[u] || base >= s1[u]) {   // self-check: slot counts inconsistent
                atomicOr(a.errorWord, kErrSortIndex);
                continue;
            }
            a.idx[base] = i0 + u * stride;
            a.B.cell[base] = d[u];
        }
    }
}

// Ascending bitonic sort of 32*K keys held K per lane (element e of lane l is
// position e*32 + l). Unused slots hold 0xffffffff.
template <int K>
__device__ __forceinline__ void warp_bitonic(uint32_t (&a)[K])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * K; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int je = j >> 5;
#pragma unroll
                for (int e = 0; e < K; ++e) {
                    const int e2 = e ^ je;
                    if (e2 > e) {
                        const bool asc = (((e << 5) | lane) & k) == 0;
                        const uint32_t lo = min(a[e], a[e2]), hi = max(a[e], a[e2]);
                        a[e] = asc ? lo : hi;
                        a[e2] = asc ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < K; ++e) {
                    const uint32_t o = __shfl_xor_sync(kFull, a[e], j);
                    const bool asc = (((e << 5) | lane) & k) == 0;
                    const bool lower = (lane & j) == 0;
                    a[e] = (lower == asc) ? min(a[e], o) : max(a[e], o);
                }
            }
        }
    }
}

template <int K>
__device__ __forceinline__ void sort_far_warp(int* seg, int m)
{
    const int lane = threadIdx.x & 31;
    uint32_t v[K];
#pragma unroll
    for (int e = 0; e < K; ++e) {
        const int p = e * 32 + lane;
        v[e] = (p < m) ? (uint32_t)seg[p] : 0xffffffffu;
    }
    warp_bitonic<K>(v);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < K; ++e) {
        const int p = e * 32 + lane;
        if (p < m) seg[p] = (int)v[e];
    }
    __syncwarp();
}

// Canonical order of a cell's far-slot arrivals: ascending source index.
// tmp is a scratch range of the same length (the output buffer's cell ids
// at those positions, written later by the gather).
__device__ void sort_far(int* seg, int m, int* tmp)
{
    const int lane = threadIdx.x & 31;
    if (m <= 32) sort_far_warp<1>(seg, m);
    else if (m <= 64) sort_far_warp<2>(seg, m);
    else if (m <= 128) sort_far_warp<4>(seg, m);
    else if (m <= 256) sort_far_warp<8>(seg, m);
    else if (m <= 512) sort_far_warp<16>(seg, m);
    else {
        // rank counting: O(m^2 / 32), for the rare very large far segments
        for (int e = lane; e < m; e += 32) tmp[e] = seg[e];
        __syncwarp();
        for (int e = lane; e < m; e += 32) {
            const int v = tmp[e];
            int r = 0;
            for (int f = 0; f < m; ++f) r += tmp[f] < v;
            seg[r] = v;
        }
        __syncwarp();
    }
}

// Canonical order of every cell's far-slot arrivals: ascending source
// index; the far counts are cleared for the next step's rank pass. Each
// lane takes one cell: a segment of up to kLaneSort arrivals (the common
// case, multi-cell hops) is insertion-sorted in the lane's own shared-memory
// row; longer ones (the cells behind an inlet, up to hundreds a step) by the
// whole warp, whose output cell ids serve as scratch for very long ones and
// are restored. A warp's 32 cells lie a grid apart: the inlet's cells are
// neighbours in the numbering, and in consecutive order one warp had 32 of
// them to sort one after another (6,080 hexahedra at 96 a cell: 116
// us; 6 as it is, each with a sort of the segment's own size instead
// of 512).
constexpr int kLaneSort = 12;
constexpr int kFarsortThreads = 256;

__global__ void __launch_bounds__(kFarsortThreads) farsort_kernel(int* countSlot, const int* startB, int* idx,
                                                                  int* cellB, int ncell)
{
    __shared__ int rows[kFarsortThreads][kLaneSort + 1];
    int* row = rows[threadIdx.x];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (long long first = warp; first < ncell; first += 32ll * nwarps) {
        const long long at = first + (long long)lane * nwarps;
        const int c = at < ncell ? (int)at : ncell;
        int far = 0, end = 0;
        if (c < ncell) {
            far = countSlot[(size_t)c * kSlots + kFarSlot];
            if (far) {
                countSlot[(size_t)c * kSlots + kFarSlot] = 0;
                end = startB[c + 1];
            }
        }
        if (far >= 2 && far <= kLaneSort) {
            int* seg = idx + end - far;
            for (int k = 0; k < far; ++k) row[k] = seg[k];
            for (int k = 1; k < far; ++k) {
                const int v = row[k];
                int j = k - 1;
                while (j >= 0 && row[j] > v) {
                    row[j + 1] = row[j];
                    --j;
                }
                row[j + 1] = v;
            }
            for (int k = 0; k < far; ++k) seg[k] = row[k];
        }
        for (unsigned m = __ballot_sync(kFull, far > kLaneSort); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const int cl = __shfl_sync(kFull, c, l);
            const int f = __shfl_sync(kFull, far, l);
            const int e = __shfl_sync(kFull, end, l);
            sort_far(idx + e - f, f, cellB + e - f);
            if (f > 512) {
                for (int k = lane; k < f; k += 32) cellB[e - f + k] = cl;
                __syncwarp();
            }
        }
    }
}

// cache2chain's data move (src/ProcessDSMC.cpp:2030-2135): output slot o
// takes source particle idx[o]. Coalesced writes; the reads follow the
// source order of each arrival group.
template <typename Real>
__global__ void __launch_bounds__(256) gather_kernel(StepArgs<Real> a)
{
    // four output slots per thread, their loads issued before their stores
    constexpr int U = 4;
    const int n = a.ctl->nNext;
    const unsigned nSrc = (unsigned)(a.ctl->nLive + a.ctl->nInj);
    const int stride = gridDim.x * blockDim.x;
    for (int o0 = blockIdx.x * blockDim.x + threadIdx.x; o0 < n; o0 += U * stride) {
        int src[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * stride;
            src[u] = o < n ? a.idx[o] : -1;
        }
        Real x[U], y[U], z[U], vx[U], vy[U], vz[U], ir[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * stride;
            if (o < n && (unsigned)src[u] < nSrc) {
                const int i = src[u];
                x[u] = a.A.x[0][i]; y[u] = a.A.x[1][i]; z[u] = a.A.x[2][i];
                vx[u] = a.A.v[0][i]; vy[u] = a.A.v[1][i]; vz[u] = a.A.v[2][i];
                ir[u] = a.A.ir[i];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int o = o0 + u * stride;
            if (o >= n) continue;
            if ((unsigned)src[u] >= nSrc) {   // self-check: never index outside the source
                atomicOr(a.errorWord, kErrSortIndex);
                continue;
            }
            a.B.x[0][o] = x[u]; a.B.x[1][o] = y[u]; a.B.x[2][o] = z[u];
            a.B.v[0][o] = vx[u]; a.B.v[1][o] = vy[u]; a.B.v[2][o] = vz[u];
            a.B.ir[o] = ir[u];
        }
    }
}

template <typename Real>
void launch_sort(const StepArgs<Real>& a, const LaunchShape& L, cudaStream_t s)
{
    const int g = L.smCount * L.sortBlocksPerSm;
    rank_kernel<Real><<<L.smCount * min(L.sortBlocksPerSm, kRankPerSm), 256, 0, s>>>(a);
    scan_partial_kernel<<<kScanBlocks, 256, 0, s>>>(a.countSlot, a.M.ncell, a.scanPartial);
    scan_final_kernel<<<kScanBlocks, 256, 0, s>>>(a.countSlot, a.M.ncell, a.scanPartial, a.startB, a.ctl);
    scatter_kernel<Real><<<g, 256, 0, s>>>(a);
    farsort_kernel<<<L.smCount * 4, kFarsortThreads, 0, s>>>(a.countSlot, a.startB, a.idx, a.B.cell, a.M.ncell);
    gather_kernel<Real><<<g, 256, 0, s>>>(a);
}

// ===========================================================================
// collisions
// ===========================================================================

// collision_diameter, src/ProcessDSMC.cpp:2603-2608 (each operation rounded
// on its own, as the oracle and the reference's x86-64 build evaluate it)
__device__ __forceinline__ double collision_diameter(double cr, double prefactor, double eta)
{
    const double cr2 = dm(cr, cr);
    return dm(dm(cr, prefactor), pow(dd(1.0, cr2), eta));
}

// The random words of candidate pair j of cell c at step istep: Philox
// blocks n = 0, 1, ... of counter (c, istep, kPurposeCollide | j << 4),
// read in order as one stream. Block 0 is drawn when the pair is handed out
// (words 0, 1: the two particles; word 2 and in FP64 word 3: the acceptance
// variate); the rest only for accepted pairs, always at the same positions,
// so the lanes of a warp draw their blocks together.
// FP64 (the oracle's layout): block 1 = relaxation test and energy fraction
// of the first particle, block 2 the same for the second, block 3 = the
// deflection and azimuth variates, 53-bit uniforms from word pairs.
// FP32: word 3 of block 0 and word 0 of block 1 are the two relaxation
// tests, words 1 and 2 of block 1 the deflection and azimuth variates; a
// particle that relaxes (u <= P) takes u / P as its energy fraction, which
// given u <= P is again uniform on (0, 1], so one block less is drawn.
struct PairDraw {
    U4 b0;
    uint32_t c, istep, purpose;
    __device__ __forceinline__ U4 block(uint32_t n, const DevConsts& C) const
    {
        return philox4x32_10(U4{c, istep, purpose, n}, C.seedLo, C.seedHi);
    }
};

__device__ __forceinline__ PairDraw pair_draw(int c, int istep, int j, int n, const DevConsts& C, int& k1, int& k2)
{
    PairDraw d;
    d.c = (uint32_t)c; d.istep = (uint32_t)istep; d.purpose = kPurposeCollide | ((uint32_t)j << 4);
    d.b0 = d.block(0, C);
    k1 = (int)__umulhi(d.b0.x, (uint32_t)n);
    k2 = k1 + 1 + (int)__umulhi(d.b0.y, (uint32_t)(n - 1));
    if (k2 >= n) k2 -= n;
    return d;
}

// Square root: IEEE in FP64; in the FP32 path from the hardware reciprocal
// square root (a few ulp; the argument is a sum of squares, >= 0).
__device__ __forceinline__ double psqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float psqrt(float x) { return x > 0.0f ? x * rsqrtf(x) : 0.0f; }

// A particle's collision state: velocity and internal energy.
template <typename Real>
struct PState {
    Real x, y, z, i;
};

// collisionVelocity, src/ProcessDSMC.cpp:2679-2744, on one candidate pair,
// in two halves: the acceptance test (pair_accept) and, for an accepted
// pair, the post-collision state (pair_execute). pair_execute recomputes the
// relative velocity from the same stored velocities, so the halves give the
// bits of the one-piece test-and-collide. w2, w3: words 2 and 3 of the
// pair's block 0; speed: for the cell's crmax, the relative speed in FP32 and
// its square in FP64 (largest_speed takes the root of the largest). The FP64
// branch rounds each operation on its own in the reference's evaluation
// order; the FP32 branch lets the compiler fuse.
template <typename Real>
__device__ __forceinline__ bool pair_accept(const PState<Real>& p, const PState<Real>& q, uint32_t w2, uint32_t w3,
                                            const DevConsts& C, double consCrm, Real crm0, bool splitSum, Real& speed)
{
    if constexpr (sizeof(Real) == 8) {
        const double vr0 = ds(p.x, q.x), vr1 = ds(p.y, q.y), vr2 = ds(p.z, q.z);
        const double cr2 = da(da(dm(vr0, vr0), dm(vr1, vr1)), dm(vr2, vr2));
        speed = cr2;
        const double u = unit64(w2, w3);
        // The acceptance is (cr / crmax)^e with e = 1 - 2 eta. In FP32, for a
        // squared ratio r of 2^-60 to 2^60, its exponent (e / 2) log2 r is off
        // by |e| / 2 times the errors of log2 r, 2^-17 (2 ulp, its documented
        // bound there) and 2^-20.5 (the roundings of cr2, c0, c0^2 and the
        // quotient's 2 ulp, times log2(e)), and by |e| 2^-18 (the roundings of e
        // and of the product): 8e-6 |e|, and the acceptance with exp2f's 2 ulp
        // by 6e-6 |e| + 3e-7 of itself. At |e| <= kVhsSettled that is 5e-5, under
        // half of 2^-13: a variate further than 2^-13 of the estimate away is
        // settled, and only the others (1 in 10^4) need the square root, the
        // power and the division of the FP64 test. Beyond it (vhsHalfF is NaN)
        // nothing is settled here. Squares that leave the normal range are
        // flushed to 0 or are infinite, and r is then out of its range.
        const float c0 = (float)crm0;
        const float r = __fdividef((float)cr2, c0 * c0);
        if (r > 0x1p-60f && r < 0x1p60f) {
            const float est = exp2f(C.vhsHalfF * __log2f(r)), uf = (float)u;
            if (uf < est * (1.0f - 0x1p-13f)) return true;
            if (uf > est * (1.0f + 0x1p-13f)) return false;
        }
        const double accept = dd(collision_diameter(dm(sqrt(cr2), C.vrms), C.cdPrefactor, C.eta), consCrm);
        return u < accept;
    } else {
        const float vr0 = p.x - q.x, vr1 = p.y - q.y, vr2 = p.z - q.z;
        // the squares added in one rounding each; in cells of up to kSmallMax
        // or more than kStagedSum particles (splitSum) the last one is rounded on
        // its own. Neither is the better one: mixed runs have always summed
        // so (by one lane and in place the one way, staged the other), and one
        // rounding changed changes every later pair of the run, so which it is
        // goes by the particle count and not by who runs the cell.
        const float xy = fmaf(vr0, vr0, __fmul_rn(vr1, vr1));
        const float cr = psqrt(splitSum ? __fadd_rn(xy, __fmul_rn(vr2, vr2)) : fmaf(vr2, vr2, xy));
        speed = cr;
        // ratio of the VHS sigma*c at cr and at crmax: (cr/crmax)^(1-2 eta)
        const float accept = exp2f(C.vhsExpF * __log2f(__fdividef(cr, crm0)));
        return unit32(w2) < accept;
    }
}

__device__ __forceinline__ void pair_execute_fp64(PState<double>& p, PState<double>& q, const PairDraw& d,
                                                  const DevConsts& C)
{
    const double vr0 = ds(p.x, q.x), vr1 = ds(p.y, q.y), vr2 = ds(p.z, q.z);
    const double cr2 = da(da(dm(vr0, vr0), dm(vr1, vr1)), dm(vr2, vr2));
    const double cr = sqrt(cr2);
    double preErt = dm(0.25, cr2);
    const U4 b1 = d.block(1, C), b2 = d.block(2, C), b3 = d.block(3, C);
    const double uRel[2] = {unit64(b1.x, b1.y), unit64(b2.x, b2.y)};
    const double rRel[2] = {unit64(b1.z, b1.w), unit64(b2.z, b2.w)};
    const double rChi = unit64(b3.x, b3.y), th = unit64(b3.z, b3.w);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        double& irp = (h == 0) ? p.i : q.i;
        if (uRel[h] <= C.prelax) {
            const double preEr = irp;
            const double postEr = dm(da(preErt, preEr), ds(1.0, pow(rRel[h], C.expLB)));
            irp = postEr;
            preErt = ds(da(preErt, preEr), postEr);
        }
    }
    const double postVr = sqrt(dd(dm(2.0, preErt), 0.5));
    const double vc0 = dm(0.5, da(p.x, q.x)), vc1 = dm(0.5, da(p.y, q.y)), vc2 = dm(0.5, da(p.z, q.z));
    const double cosChi = ds(dm(2.0, pow(rChi, C.invAlpha)), 1.0);
    const double sinChi = sqrt(ds(1.0, dm(cosChi, cosChi)));
    const double ang = dm(6.283185307179586, th);   // 2 pi th
    double sth, cth;
    sincos(ang, &sth, &cth);
    const double vrp = sqrt(da(dm(vr1, vr1), dm(vr2, vr2)));
    const double scale = dd(postVr, cr > 1.0e-300 ? cr : 1.0e-300);
    const double vrpc = vrp > 1.0e-300 ? vrp : 1.0e-300;
    double r1, r2, r3;
    if (vrp < 1e-6) {
        r1 = dm(dm(scale, cosChi), vr0);
        r2 = dm(dm(dm(scale, sinChi), vr0), cth);
        r3 = dm(dm(dm(scale, sinChi), vr0), sth);
    } else {
        r1 = dm(scale, da(dm(cosChi, vr0), dm(dm(sinChi, sth), vrp)));
        r2 = dm(scale, da(dm(cosChi, vr1), dd(dm(sinChi, ds(dm(dm(cr, vr2), cth), dm(dm(vr0, vr1), sth))), vrpc)));
        r3 = dm(scale, ds(dm(cosChi, vr2), dd(dm(sinChi, da(dm(dm(cr, vr1), cth), dm(dm(vr0, vr2), sth))), vrpc)));
    }
    p.x = da(vc0, dm(0.5, r1)); p.y = da(vc1, dm(0.5, r2)); p.z = da(vc2, dm(0.5, r3));
    q.x = ds(vc0, dm(0.5, r1)); q.y = ds(vc1, dm(0.5, r2)); q.z = ds(vc2, dm(0.5, r3));
}

__device__ __forceinline__ void pair_execute_fp32(PState<float>& p, PState<float>& q, const U4& b1, uint32_t w3,
                                                  const DevConsts& C)
{
    const float vr0 = p.x - q.x, vr1 = p.y - q.y, vr2 = p.z - q.z;
    const float cr2 = vr0 * vr0 + vr1 * vr1 + vr2 * vr2;
    const float cr = psqrt(cr2);
    float preErt = 0.25f * cr2;
    const float uRel[2] = {unit32(w3), unit32(b1.x)};
    const float rChi = unit32(b1.y), th = unit32(b1.z);
    const float expLB = (float)C.expLB;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float& irp = (h == 0) ? p.i : q.i;
        if (uRel[h] <= C.prelaxF) {
            const float r = fminf(uRel[h] * C.invPrelaxF, 1.0f);
            const float preEr = irp;
            const float postEr = (preErt + preEr) * (1.0f - exp2f(expLB * __log2f(r)));
            irp = postEr;
            preErt = preErt + preEr - postEr;
        }
    }
    const float postVr = 2.0f * psqrt(preErt);
    const float vc0 = 0.5f * (p.x + q.x), vc1 = 0.5f * (p.y + q.y), vc2 = 0.5f * (p.z + q.z);
    const float cosChi =
        (C.alpha == 1.0) ? 2.0f * rChi - 1.0f : 2.0f * exp2f((float)C.invAlpha * __log2f(rChi)) - 1.0f;
    const float sinChi = psqrt(1.0f - cosChi * cosChi);
    // azimuth 2 pi th: sin and cos of 2 pi (th - 1/2) in [-pi, pi), negated
    const float ang = 6.283185307179586f * (th - 0.5f);
    const float sth = -__sinf(ang), cth = -__cosf(ang);
    const float vrp = psqrt(vr1 * vr1 + vr2 * vr2);
    const float scale = __fdividef(postVr, cr > 1.0e-30f ? cr : 1.0e-30f);
    const float vrpc = vrp > 1.0e-30f ? vrp : 1.0e-30f;
    float r1, r2, r3;
    if (vrp < 1e-6f) {
        r1 = scale * cosChi * vr0;
        r2 = scale * sinChi * vr0 * cth;
        r3 = scale * sinChi * vr0 * sth;
    } else {
        r1 = scale * (cosChi * vr0 + sinChi * sth * vrp);
        r2 = scale * (cosChi * vr1 + __fdividef(sinChi * (cr * vr2 * cth - vr0 * vr1 * sth), vrpc));
        r3 = scale * (cosChi * vr2 - __fdividef(sinChi * (cr * vr1 * cth + vr0 * vr2 * sth), vrpc));
    }
    p.x = vc0 + 0.5f * r1; p.y = vc1 + 0.5f * r2; p.z = vc2 + 0.5f * r3;
    q.x = vc0 - 0.5f * r1; q.y = vc1 - 0.5f * r2; q.z = vc2 - 0.5f * r3;
}

// One candidate pair (j of cell c) on the two particles' states: tested and,
// when accepted, carried out. Returns whether it was accepted; crmLocal takes
// pair_accept's speed if it is larger.
template <typename Real>
__device__ __forceinline__ bool pair_collide(PState<Real>& p, PState<Real>& q, int c, int istep, int j, uint32_t w2,
                                             uint32_t w3, const DevConsts& C, double consCrm, Real crm0, bool splitSum,
                                             Real& crmLocal)
{
    Real speed;
    const bool acc = pair_accept<Real>(p, q, w2, w3, C, consCrm, crm0, splitSum, speed);
    if (speed > crmLocal) crmLocal = speed;
    if (acc) {
        PairDraw d;
        d.c = (uint32_t)c; d.istep = (uint32_t)istep; d.purpose = kPurposeCollide | ((uint32_t)j << 4);
        if constexpr (sizeof(Real) == 8) pair_execute_fp64(p, q, d, C);
        else pair_execute_fp32(p, q, d.block(1, C), w3, C);
    }
    return acc;
}

// The largest relative speed from the largest value pair_accept gave (the
// square root, rounded as it is, keeps the order).
__device__ __forceinline__ double largest_speed(double m) { return sqrt(m); }
__device__ __forceinline__ double largest_speed(float m) { return (double)m; }

// Candidate pair count of a cell from the majorant, with the carried
// remainder (collisionDSMC, src/ProcessDSMC.cpp:2631-2645), in the
// reference's evaluation order.
template <typename Real>
__device__ __forceinline__ int pair_count(const StepArgs<Real>& a, int c, int n, double& consCrm, double& crm0)
{
    crm0 = a.crmax[c];
    const double S = a.M.cellVolume[c];
    consCrm = collision_diameter(dm(crm0, a.C.vrms), a.C.cdPrefactor, a.C.eta);
    double t = dm(0.5, (double)n);
    t = dm(t, (double)(n - 1));
    t = dm(t, a.C.neff);
    t = dm(t, consCrm);
    t = dm(t, a.C.dtime);
    t = dm(t, a.C.dtref);
    const double pairs = da(dd(t, S), a.remColl[c]);
    const int npairs = (int)floor(pairs);
    a.remColl[c] = ds(pairs, (double)npairs);
    return npairs;
}

// NTC collisions of one small cell by one thread: the candidate pairs one
// after another, component q of particle k at v[q][k * stride].
template <typename Real>
__device__ void collide_cell_serial(Real* const (&v)[4], int stride, int n, int c, const StepArgs<Real>& a, int istep,
                                    uint32_t& collOut)
{
    const int npairs = a.cellPairs[c];
    const double consCrm = a.cellCons[c], crm0 = a.crmax[c];
    if (!(consCrm > 0.0) || npairs <= 0) return;
    Real crmLocal = (Real)0;
    const Real crm0r = (Real)crm0;
    auto load = [&](int k) { return PState<Real>{v[0][k * stride], v[1][k * stride], v[2][k * stride], v[3][k * stride]}; };
    auto store = [&](int k, const PState<Real>& p) {
        v[0][k * stride] = p.x; v[1][k * stride] = p.y; v[2][k * stride] = p.z; v[3][k * stride] = p.i;
    };
    for (int j = 0; j < npairs; ++j) {
        int k1, k2;
        const PairDraw d = pair_draw(c, istep, j, n, a.C, k1, k2);
        PState<Real> p = load(k1), q = load(k2);
        if (pair_collide<Real>(p, q, c, istep, j, d.b0.z, d.b0.w, a.C, consCrm, crm0r, true, crmLocal)) {
            store(k1, p);
            store(k2, q);
            ++collOut;
        }
    }
    const double crm = largest_speed(crmLocal);
    if (crm > crm0) a.crmax[c] = crm;
}

// the largest of a warp's values
template <typename Real>
__device__ __forceinline__ Real warp_max(Real m)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const Real y = __shfl_xor_sync(kFull, m, o);
        m = y > m ? y : m;
    }
    return m;
}

// The collision pass over the sorted buffer (collisionDSMC,
// src/ProcessDSMC.cpp:2621-2665). Cells are classed first (classify_kernel):
// - small cells (at most CellShape::small particles and kSmallPairs pairs): 32
//   at a time per warp, lane l owning one cell and running its pairs alone, with
//   the particles' velocities and internal energies in shared memory at slot
//   k * 32 + l (lane l's slots sit in bank l, so the lanes never conflict); when
//   all cells together are few enough for half a warp each, as large cells;
// - large cells: two at a time per warp, staged in shared memory
//   (collide_kernel), those of the most rounds first;
// - middle cells (more than kMiddlePairs pairs): as big cells when every one
//   of them finds a free block, as large cells otherwise;
// - big cells (more particles than a warp's arena, or more pairs than
//   kBigPairs) and giants (more pairs than kGiantPairs, handed out first):
//   one at a time by a block of 256 threads (collide_big_kernel), beside the
//   other kernel on the side stream.
// A cell's result depends on nothing but the cell, so neither the warp or
// block that takes it nor the order matters.
//
// What bounds it: a cell's pairs depend on each other through its particles,
// so a cell is a chain of rounds. Where cells are few, the pass is as long as
// its longest chain; where they are many, it is bound by instruction issue
// (of 32 lanes some 12 work) and by the warps that fit an SM.
// - With every cell run by one warp, 32 pairs a round at most, the few
//   compressed cells of a capsule (2,000 particles, 30,000-60,000 pairs) were
//   the whole pass. A block runs up to 256 pairs a round, in a fifth of the
//   rounds. Two blocks of 256 threads an SM, not one of 512: one's barriers are
//   covered by the other (FP64 capsule of 63,500 cells, the step: 2,990 us
//   with 512 threads, 2,750 with 2 x 256).
// - A warp outdoes a block in throughput, so in a full device the blocks only
//   get chains that would outlast the pass: with kBigPairs at 512 that
//   capsule's step took 4,380 us, at 2,048 2,840. Where the blocks are free,
//   they shorten the pass (6,080 cells: 52 -> 32 us).
// - Cells of up to 16 particles can have 900 pairs, one lane running one after
//   another. In a full device lanes still do best for those of up to 32 pairs
//   (372,500 cells, the step: 4,280 us; with warps for those of more than 4
//   particles 4,420); in an empty one they are the longest chain (760 cells:
//   19.5 us, 9.1 by half warps).
// - FP64 needs 36 bytes a particle: arenas of 376 let eight blocks (16 warps)
//   into an SM, of 512 six (48,640 cells: 113 us with six, 91 with eight).
// Arenas (FP32 20 KB, FP64 26 KB per block, plus the 1 KB the runtime reserves)
// fill an SM's 228 KB.
constexpr int kCellWarps = 2;                 // warps per block of collide_kernel
constexpr int kSmallMax = 16;
constexpr int kBigThreads = 256;
constexpr int kBigPerSm = 2;                  // resident blocks of collide_big_kernel per SM
constexpr int kBigPairs = 1024, kMiddlePairs = 512;
constexpr int kBigLeast = 128;                // fewer particles give a block no more pairs a round than a warp
template <typename Real>
struct CellShape;
template <>
struct CellShape<float> {
    static constexpr int arena = 512;         // staged particles per warp
    static constexpr int blocks = 10;         // resident blocks of collide_kernel per SM
    static constexpr int small = kSmallMax;   // particles of a small cell
    static constexpr int big = 4096;          // staged particles per block of collide_big_kernel
};
template <>
struct CellShape<double> {
    static constexpr int arena = 376;
    static constexpr int blocks = 8;
    static constexpr int small = 12;
    static constexpr int big = 3072;
};
constexpr int kSmallPairs = 32;
constexpr int kGiantPairs = 8192;
constexpr int kStagedSum = 512;               // see pair_accept: FP32 cells beyond it add the squares in two roundings

// shared memory of `slots` staged particles: their states and claims
template <typename Real>
__host__ __device__ constexpr size_t arena_bytes(int slots)
{
    return (size_t)slots * (4 * sizeof(Real) + sizeof(int));
}
static_assert(32 * CellShape<float>::small * 4 * sizeof(float) <= arena_bytes<float>(CellShape<float>::arena) &&
                  32 * CellShape<double>::small * 4 * sizeof(double) <= arena_bytes<double>(CellShape<double>::arena),
              "small-cell slots must fit in the arena");

// particle states in shared memory, 16 bytes a load
template <typename Real>
struct Arena;
template <>
struct Arena<float> {
    float4* v;
    int* claim;
    __device__ __forceinline__ Arena(unsigned char* p, int slots)
        : v(reinterpret_cast<float4*>(p)), claim(reinterpret_cast<int*>(v + slots))
    {
    }
    __device__ __forceinline__ PState<float> get(int k) const
    {
        const float4 t = v[k];
        return {t.x, t.y, t.z, t.w};
    }
    __device__ __forceinline__ void put(int k, const PState<float>& p) const { v[k] = make_float4(p.x, p.y, p.z, p.i); }
};
template <>
struct Arena<double> {
    double2 *lo, *hi;
    int* claim;
    __device__ __forceinline__ Arena(unsigned char* p, int slots)
        : lo(reinterpret_cast<double2*>(p)), hi(lo + slots), claim(reinterpret_cast<int*>(hi + slots))
    {
    }
    __device__ __forceinline__ PState<double> get(int k) const
    {
        const double2 s = lo[k], t = hi[k];
        return {s.x, s.y, t.x, t.y};
    }
    __device__ __forceinline__ void put(int k, const PState<double>& p) const
    {
        lo[k] = make_double2(p.x, p.y);
        hi[k] = make_double2(p.z, p.i);
    }
};

// the states and claims of a cell run in place in the particle buffer
template <typename Real>
struct InPlace {
    Real* v[4];
    int* claim;
    __device__ __forceinline__ PState<Real> get(int k) const { return {v[0][k], v[1][k], v[2][k], v[3][k]}; }
    __device__ __forceinline__ void put(int k, const PState<Real>& p) const
    {
        v[0][k] = p.x; v[1][k] = p.y; v[2][k] = p.z; v[3][k] = p.i;
    }
};

// Stage a cell (n particles from s0) at arena slots base.., by T threads of
// which this is thread t: the loads of four particles a thread are issued
// before their stores. unstage writes it back.
template <typename Real>
__device__ __forceinline__ void stage_cell(const PBuf<Real>& buf, const Arena<Real>& A, int s0, int n, int base, int t,
                                           int T)
{
    for (int k0 = t; k0 < n; k0 += 4 * T) {
        PState<Real> p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * T;
            if (k < n) p[u] = {buf.v[0][s0 + k], buf.v[1][s0 + k], buf.v[2][s0 + k], buf.ir[s0 + k]};
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * T;
            if (k < n) {
                A.put(base + k, p[u]);
                A.claim[base + k] = INT_MAX;
            }
        }
    }
}
template <typename Real>
__device__ __forceinline__ void unstage_cell(const PBuf<Real>& buf, const Arena<Real>& A, int s0, int n, int base, int t,
                                             int T)
{
    for (int k = t; k < n; k += T) {
        const PState<Real> p = A.get(base + k);
        buf.v[0][s0 + k] = p.x; buf.v[1][s0 + k] = p.y; buf.v[2][s0 + k] = p.z;
        buf.ir[s0 + k] = p.i;
    }
}

// cellWork: [0..2] large counts by their rounds (more than kManyRounds, more
//           than kSomeRounds, the rest), [3] small count, [4] big count, [5] giant
//           count, [6] next large item, [7] next small, [8] next giant or big,
//           [9] middle count
// cellList: small cells from the front of [0, ncell), big cells from its
//           back, giants from the front of [ncell, 2 ncell)
// cellItem: large cells, of many rounds from the front of [0, ncell), of some
//           from its back, the rest from the front of [ncell, 2 ncell), middle
//           cells from its back; handed out middle, many, some, rest, so that
//           the longest chains start first
constexpr int kWorkWords = 16;
constexpr int kManyRounds = 40, kSomeRounds = 12;
struct LargeLists {
    int middle, many, some, all;   // counts; all: of the three and the rest
    int small;                     // small cells that follow them, one item each
    __device__ __forceinline__ int slot(int it, int ncell) const
    {
        if (it < middle) return 2 * ncell - 1 - it;
        it -= middle;
        return it < many ? it : it < many + some ? ncell - 1 - (it - many) : ncell + (it - many - some);
    }
};
// Middle cells go to the blocks when every one of them finds a free block at
// once, and to the warps otherwise.
__device__ __forceinline__ bool middle_by_blocks(const int* work, int bigBlocks)
{
    return work[4] + work[5] + work[9] <= bigBlocks;
}
template <typename Real>
__global__ void classify_kernel(StepArgs<Real> a)
{
    const int lane = threadIdx.x & 31;
    const int* start = a.startA;
    const int ncell = a.M.ncell;
    int* work = a.cellWork;
    uint32_t pairs = 0, over = 0;
    for (int base = blockIdx.x * blockDim.x; base < ncell; base += gridDim.x * blockDim.x) {
        const int c = base + threadIdx.x;
        const int s0 = c < ncell ? start[c] : 0;
        const int n = c < ncell ? start[c + 1] - s0 : -1;
        // the cell's candidate pair count, one thread per cell
        int np = 0;
        double consCrm = 0.0, crm0 = 0.0;
        if (n > 1) {
            np = pair_count(a, c, n, consCrm, crm0);
            a.cellPairs[c] = np;
            a.cellCons[c] = consCrm;
            pairs += (uint32_t)np;
        }
        if (n > 512) ++over;
        // nothing collides in a cell without pairs: it goes on no list
        int cls = -1;
        if (n > 1 && np > 0 && consCrm > 0.0) {
            // a round runs about 13 pairs of a cell, n / 4 of one with few particles
            const int rounds = np / min(13, max(1, n >> 2));
            if (n <= CellShape<Real>::small && np <= kSmallPairs) cls = 3;
            else if (np > kGiantPairs && n > kBigLeast) cls = 5;
            else if (n > CellShape<Real>::arena || (np > kBigPairs && n > kBigLeast)) cls = 4;
            else if (np > kMiddlePairs && n > kBigLeast) cls = 6;
            else cls = rounds > kManyRounds ? 0 : rounds > kSomeRounds ? 1 : 2;
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const unsigned m = __ballot_sync(kFull, cls == k);
            if (!m) continue;
            const int leader = __ffs(m) - 1;
            int b = 0;
            if (lane == leader) b = atomicAdd(work + (k < 6 ? k : 9), __popc(m));
            b = __shfl_sync(kFull, b, leader);
            if (cls == k) {
                const int pos = b + __popc(m & ((1u << lane) - 1u));
                if (k < 3 || k == 6) {
                    const int slot = k == 0 ? pos : k == 1 ? ncell - 1 - pos : k == 2 ? ncell + pos : 2 * ncell - 1 - pos;
                    a.cellItem[slot] = make_int4(c, s0, n, np);
                    a.cellItemC[slot] = make_double2(consCrm, crm0);
                } else {
                    a.cellList[k == 3 ? pos : k == 4 ? ncell - 1 - pos : ncell + pos] = c;
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pairs += __shfl_xor_sync(kFull, pairs, o);
        over += __shfl_xor_sync(kFull, over, o);
    }
    if (lane == 0) {
        if (pairs) atomicAdd(a.counters + C_PAIRS, (unsigned long long)pairs);
        if (over) atomicAdd(a.counters + C_BIG_CELLS, (unsigned long long)over);
    }
}

// copy a small cell's velocities and internal energies between the buffer
// (at s0) and v[comp][k * 32], whole warp
template <typename Real, bool kToBuffer>
__device__ __forceinline__ void copy_cell(const PBuf<Real>& buf, int s0, int n, Real* const (&v)[4])
{
    Real* const b[4] = {buf.v[0] + s0, buf.v[1] + s0, buf.v[2] + s0, buf.ir + s0};
    const int k = threadIdx.x & 31;
    if (k < n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if constexpr (kToBuffer) b[q][k] = v[q][k * 32];
            else v[q][k * 32] = b[q][k];
        }
}

// Collisions of staged large cells, two cells per warp at a time, both in
// the warp's arena: channel 0's cell at its front, channel 1's at its
// back; a cell that does not fit beside the other channel's
// waits until that one is done. The pairs run as a sliding window: every
// lane holds one pending pair of either cell and claims its two particles
// with the pair index (atomicMin); a pair whose index is the lowest claim on
// both goes, tested and carried out by its lane, which then takes the next
// pair not yet handed out: of channel 0 in the lower half of the warp, of
// channel 1 in the upper, or of the other channel when its own has none
// left. A cell's pairs are handed out in increasing order, so a pair goes
// only after every lower pair that shares a particle with it, and the result
// equals running the pairs one after another. The lowest pending pair of a
// cell always goes, so the loop ends after at most the pairs' number of
// rounds. A channel whose pairs are done writes its cell back and takes the
// next.
// Half a warp per cell, because of 32 pairs of one cell of 100-300 particles
// some 13 to 20 go a round, and of 16 about 13; each phase then runs once a
// round for both cells.
template <typename Real>
__device__ void collide_two_cells(const StepArgs<Real>& a, const PBuf<Real>& buf, const Arena<Real>& A,
                                  const LargeLists& L, int istep, uint32_t& colls)
{
    constexpr int N = CellShape<Real>::arena;
    const int nItems = L.all + L.small;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    int cc[2] = {-1, -1}, cbase[2] = {0, 0}, cs0[2] = {0, 0}, cn[2] = {0, 0}, cnp[2] = {0, 0}, cnext[2] = {0, 0};
    double ccons[2] = {0.0, 0.0}, ccrm[2] = {0.0, 0.0};
    Real crmL[2] = {(Real)0, (Real)0};
    int j = -1, ch = 0, k1 = 0, k2 = 0;   // this lane's pending pair
    uint32_t w2 = 0u, w3 = 0u;
    int held = -1;        // an item taken but not yet placed
    bool more = true;
    // the next item index, taken one item ahead (lane 0): the atomic's
    // round trip overlaps the rounds of the cells in work. Indices are
    // handed out in increasing order and the loop runs until it sees one
    // past the end, so an index taken ahead is always used.
    int ahead = 0;
    if (lane == 0) ahead = atomicAdd(a.cellWork + 6, 1);
    // the next pairs, in increasing order, to the lanes that ask for one (all
    // lanes call it): of the half's own channel, or of the other when that
    // has none left; j = -1 for a lane that gets none
    auto hand_out = [&](bool ask) {
        const bool left0 = cc[0] >= 0 && cnext[0] < cnp[0], left1 = cc[1] >= 0 && cnext[1] < cnp[1];
        const int want = !ask ? -1 : lane < 16 ? (left0 ? 0 : left1 ? 1 : -1) : (left1 ? 1 : left0 ? 0 : -1);
        const unsigned m0 = __ballot_sync(kFull, want == 0), m1 = __ballot_sync(kFull, want == 1);
        if (ask) {
            j = -1;
            const int jj = (want > 0 ? cnext[1] : cnext[0]) + __popc((want > 0 ? m1 : m0) & below);
            if (want >= 0 && jj < (want ? cnp[1] : cnp[0])) {
                j = jj;
                ch = want;
                const int base = want ? cbase[1] : cbase[0];
                const PairDraw d = pair_draw(want ? cc[1] : cc[0], istep, jj, want ? cn[1] : cn[0], a.C, k1, k2);
                k1 += base;
                k2 += base;
                w2 = d.b0.z;
                w3 = d.b0.w;
            }
        }
        cnext[0] = min(cnp[0], cnext[0] + __popc(m0));
        cnext[1] = min(cnp[1], cnext[1] + __popc(m1));
    };
    for (;;) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            while (cc[h] < 0 && (more || held >= 0)) {
                int it = held;
                if (it < 0) {
                    it = __shfl_sync(kFull, ahead, 0);
                    if (lane == 0 && it < nItems) ahead = atomicAdd(a.cellWork + 6, 1);
                }
                held = -1;
                if (it >= nItems) {
                    more = false;
                    break;
                }
                int4 rec;
                double2 rc;
                if (it < L.all) {
                    const int slot = L.slot(it, a.M.ncell);
                    rec = a.cellItem[slot];
                    rc = a.cellItemC[slot];
                } else {
                    const int c = a.cellList[it - L.all], s0 = a.startA[c];
                    rec = make_int4(c, s0, a.startA[c + 1] - s0, a.cellPairs[c]);
                    rc = make_double2(a.cellCons[c], a.crmax[c]);
                }
                const int n = rec.z;
                if (n > N) {   // never reached (classify lists no such cell): flag rather than overflow the arena
                    if (lane == 0) atomicOr(a.errorWord, kErrStageCell);
                    continue;
                }
                if (n > N - (cc[h ^ 1] >= 0 ? cn[h ^ 1] : 0)) {   // wait for the other channel
                    held = it;
                    break;
                }
                const int base = h == 0 ? 0 : N - n;
                stage_cell(buf, A, rec.y, n, base, lane, 32);
                cc[h] = rec.x; cbase[h] = base; cs0[h] = rec.y; cn[h] = n; cnp[h] = rec.w; cnext[h] = 0;
                ccons[h] = rc.x; ccrm[h] = rc.y; crmL[h] = (Real)0;
                __syncwarp();
            }
        }
        if (cc[0] < 0 && cc[1] < 0) break;
        hand_out(j < 0);
        // claim both particles with the pair index; the lowest claim goes
        if (j >= 0) {
            atomicMin(&A.claim[k1], j);
            atomicMin(&A.claim[k2], j);
        }
        __syncwarp();
        const bool go = j >= 0 && A.claim[k1] == j && A.claim[k2] == j;
        __syncwarp();
        if (go) {
            PState<Real> p = A.get(k1), q = A.get(k2);
            Real& crm = ch ? crmL[1] : crmL[0];
            const int n = ch ? cn[1] : cn[0];
            if (pair_collide<Real>(p, q, ch ? cc[1] : cc[0], istep, j, w2, w3, a.C, ch ? ccons[1] : ccons[0],
                                   (Real)(ch ? ccrm[1] : ccrm[0]), n <= kSmallMax, crm)) {
                A.put(k1, p);
                A.put(k2, q);
                ++colls;
            }
            A.claim[k1] = INT_MAX;
            A.claim[k2] = INT_MAX;
            j = -1;
        }
        __syncwarp();
        // a channel whose pairs are all done finishes its cell
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (cc[h] < 0 || cnext[h] < cnp[h] || __ballot_sync(kFull, j >= 0 && ch == h) != 0u) continue;
            const double m = largest_speed(warp_max(crmL[h]));
            if (lane == 0 && m > ccrm[h]) a.crmax[cc[h]] = m;
            unstage_cell(buf, A, cs0[h], cn[h], cbase[h], lane, 32);
            __syncwarp();
            cc[h] = -1;
        }
    }
}

template <typename Real>
__global__ void __launch_bounds__(kCellWarps * 32, CellShape<Real>::blocks) collide_kernel(StepArgs<Real> a, int bigBlocks)
{
    extern __shared__ __align__(16) unsigned char cellSmem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* const wsm = cellSmem + (size_t)wib * arena_bytes<Real>(CellShape<Real>::arena);
    const int istep = a.ctl->istep;
    const PBuf<Real> buf = a.A;
    uint32_t colls = 0;

    int nSmall = a.cellWork[3];
    LargeLists L;
    L.middle = middle_by_blocks(a.cellWork, bigBlocks) ? 0 : a.cellWork[9];
    L.many = a.cellWork[0];
    L.some = a.cellWork[1];
    L.all = L.middle + L.many + L.some + a.cellWork[2];
    // few enough cells for half a warp each: the small ones too, since one
    // lane's pairs one after another take longer than a warp's rounds
    L.small = L.all + nSmall <= (int)(gridDim.x * kCellWarps) * 2 ? nSmall : 0;
    nSmall -= L.small;
    if (L.all + L.small > 0) collide_two_cells<Real>(a, buf, Arena<Real>(wsm, CellShape<Real>::arena), L, istep, colls);

    // ---- small cells, 32 per warp, one lane each
    constexpr int kSmallSlots = 32 * CellShape<Real>::small;
    Real* const sv = reinterpret_cast<Real*>(wsm);
    Real* const stage[4] = {sv, sv + kSmallSlots, sv + 2 * kSmallSlots, sv + 3 * kSmallSlots};
    const int* start = a.startA;
    while (nSmall > 0) {
        int g = 0;
        if (lane == 0) g = atomicAdd(a.cellWork + 7, 32);
        g = __shfl_sync(kFull, g, 0);
        if (g >= nSmall) break;
        const bool mine = g + lane < nSmall;
        const int myc = mine ? a.cellList[g + lane] : 0;
        const int ms0 = mine ? start[myc] : 0;
        const int mn = mine ? start[myc + 1] - ms0 : 0;
        const int many = min(32, nSmall - g);
        for (int l = 0; l < many; ++l) {
            Real* const to[4] = {stage[0] + l, stage[1] + l, stage[2] + l, stage[3] + l};
            copy_cell<Real, false>(buf, __shfl_sync(kFull, ms0, l), __shfl_sync(kFull, mn, l), to);
        }
        __syncwarp();
        if (mine) {
            Real* const v[4] = {stage[0] + lane, stage[1] + lane, stage[2] + lane, stage[3] + lane};
            collide_cell_serial<Real>(v, 32, mn, myc, a, istep, colls);
        }
        __syncwarp();
        for (int l = 0; l < many; ++l) {
            Real* const from[4] = {stage[0] + l, stage[1] + l, stage[2] + l, stage[3] + l};
            copy_cell<Real, true>(buf, __shfl_sync(kFull, ms0, l), __shfl_sync(kFull, mn, l), from);
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) colls += __shfl_xor_sync(kFull, colls, o);
    if (lane == 0 && colls) atomicAdd(a.counters + C_COLLISIONS, (unsigned long long)colls);
}

// One cell by the whole block: the sliding window of collide_two_cells over
// kBigThreads threads. The idle threads of a warp take their pairs together
// from a counter; which of them gets which pair does not matter, only that
// every pair below a claimed one is claimed or done, and the barrier before
// the claims are read sees to that. A: the cell's states and claims (an
// Arena, or InPlace for a cell beyond it).
template <typename Real, typename States>
__device__ __forceinline__ void collide_by_block(const States& A, int n, int c, int np, double consCrm, double crm0,
                                                 const StepArgs<Real>& a, int istep, int* sNext,
                                                 unsigned long long* sCrm, uint32_t& colls)
{
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    const Real crm0r = (Real)crm0;
    Real crmLocal = (Real)0;
    // threads with pairs: more than n / 2 at once mostly wait for each
    // other and take issue slots from those that go
    const bool works = tid < min(kBigThreads, max(64, (n >> 1) & ~31));
    int j = -1, k1 = 0, k2 = 0;
    uint32_t w2 = 0u, w3 = 0u;
    bool left = works;  // pairs may be left to hand out (the same in every lane of a warp)
    // the next pairs to the lanes of this warp that ask for one
    auto hand_out = [&](bool ask) {
        const unsigned m = __ballot_sync(kFull, ask);
        if (ask) j = -1;
        if (!left || !m) return;
        int first = 0;
        if (lane == 0) first = atomicAdd(sNext, __popc(m));
        first = __shfl_sync(kFull, first, 0);
        const int jj = first + __popc(m & below);
        if (ask && jj < np) {
            j = jj;
            const PairDraw d = pair_draw(c, istep, j, n, a.C, k1, k2);
            w2 = d.b0.z;
            w3 = d.b0.w;
        }
        left = first < np;
    };
    hand_out(works);
    for (;;) {
        if (j >= 0) {
            atomicMin(&A.claim[k1], j);
            atomicMin(&A.claim[k2], j);
        }
        __syncthreads();
        const bool go = j >= 0 && A.claim[k1] == j && A.claim[k2] == j;
        __syncthreads();
        const int jNow = j, k1Now = k1, k2Now = k2;
        const uint32_t w2Now = w2, w3Now = w3;
        hand_out(go);   // drawn beside this round's collisions, claimed in the next
        if (go) {
            PState<Real> p = A.get(k1Now), q = A.get(k2Now);
            if (pair_collide<Real>(p, q, c, istep, jNow, w2Now, w3Now, a.C, consCrm, crm0r, n > kStagedSum, crmLocal)) {
                A.put(k1Now, p);
                A.put(k2Now, q);
                ++colls;
            }
            A.claim[k1Now] = INT_MAX;
            A.claim[k2Now] = INT_MAX;
        }
        if (!__syncthreads_or(j >= 0)) break;
    }
    // the largest relative speed tested (a double's order is that of
    // its bits when positive)
    const double m = largest_speed(warp_max(crmLocal));
    if (lane == 0 && m > crm0) atomicMax(sCrm, (unsigned long long)__double_as_longlong(m));
}

// Big cells, one at a time by a block, giants first, then the middle cells if
// the blocks take them. A cell beyond the block's arena is run in place in
// the particle buffer, with its claims in the arena's memory or, beyond that
// too (20,480 particles in FP32, 27,648 in FP64), in its cell-id slots.
template <typename Real>
__global__ void __launch_bounds__(kBigThreads, kBigPerSm) collide_big_kernel(StepArgs<Real> a)
{
    extern __shared__ __align__(16) unsigned char cellSmem[];
    __shared__ int sItem, sNext;
    __shared__ unsigned long long sCrm;
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int kArena = CellShape<Real>::big;
    constexpr int kClaims = (int)(arena_bytes<Real>(kArena) / sizeof(int));
    const Arena<Real> A(cellSmem, kArena);
    const int istep = a.ctl->istep, ncell = a.M.ncell;
    const int nBig = a.cellWork[4], nGiant = a.cellWork[5];
    const int nAll = nBig + nGiant + (middle_by_blocks(a.cellWork, (int)gridDim.x) ? a.cellWork[9] : 0);
    const PBuf<Real> buf = a.A;
    uint32_t colls = 0;
    if (nAll > 0)
        for (;;) {
            __syncthreads();   // the last cell's values have been read
            if (tid == 0) {
                sItem = atomicAdd(a.cellWork + 8, 1);
                sNext = 0;
                sCrm = 0ull;
            }
            __syncthreads();
            const int it = sItem;
            if (it >= nAll) break;
            const int c = it < nGiant ? a.cellList[ncell + it]
                          : it < nGiant + nBig ? a.cellList[ncell - 1 - (it - nGiant)]
                                               : a.cellItem[2 * ncell - 1 - (it - nGiant - nBig)].x;
            const int s0 = a.startA[c], n = a.startA[c + 1] - s0, np = a.cellPairs[c];
            const double consCrm = a.cellCons[c], crm0 = a.crmax[c];
            if (n <= kArena) {
                stage_cell(buf, A, s0, n, 0, tid, kBigThreads);
                __syncthreads();
                collide_by_block<Real>(A, n, c, np, consCrm, crm0, a, istep, &sNext, &sCrm, colls);
                unstage_cell(buf, A, s0, n, 0, tid, kBigThreads);
            } else {
                const InPlace<Real> I{{buf.v[0] + s0, buf.v[1] + s0, buf.v[2] + s0, buf.ir + s0},
                                      n <= kClaims ? reinterpret_cast<int*>(cellSmem) : buf.cell + s0};
                for (int k = tid; k < n; k += kBigThreads) I.claim[k] = INT_MAX;
                __syncthreads();
                collide_by_block<Real>(I, n, c, np, consCrm, crm0, a, istep, &sNext, &sCrm, colls);
                if (n > kClaims)
                    for (int k = tid; k < n; k += kBigThreads) I.claim[k] = c;
            }
            __syncthreads();
            if (tid == 0 && sCrm) a.crmax[c] = __longlong_as_double((long long)sCrm);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) colls += __shfl_xor_sync(kFull, colls, o);
    if (lane == 0 && colls) atomicAdd(a.counters + C_COLLISIONS, (unsigned long long)colls);
}

// resident blocks per SM of the collision kernel, set by prepare_kernels
template <typename Real>
struct CellOcc {
    static int blocks;
};
template <typename Real>
int CellOcc<Real>::blocks = 1;

template <typename Real>
cudaError_t prepare_kernels()
{
    constexpr size_t cellBytes = kCellWarps * arena_bytes<Real>(CellShape<Real>::arena), bigBytes = arena_bytes<Real>(CellShape<Real>::big);
    cudaError_t e = cudaFuncSetAttribute(collide_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cellBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(collide_big_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bigBytes);
    if (e != cudaSuccess) return e;
    int nb = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, collide_kernel<Real>, kCellWarps * 32, cellBytes);
    if (e != cudaSuccess) return e;
    CellOcc<Real>::blocks = nb > 0 ? nb : 1;
    return prepare_move<Real>();
}

template <typename Real>
void launch_collide(const StepArgs<Real>& a, const LaunchShape& L, cudaStream_t s, const SideStream& side)
{
    const int ncell = a.M.ncell;
    cudaMemsetAsync(a.cellWork, 0, kWorkWords * sizeof(int), s);
    int gc = (ncell + 255) / 256;
    if (gc > L.smCount * 8) gc = L.smCount * 8;
    classify_kernel<Real><<<gc > 0 ? gc : 1, 256, 0, s>>>(a);
    // the big cells' kernel goes first: its blocks need much of an SM's
    // shared memory, and the other cells' blocks fill what they leave
    side.fork(s);
    const int bigBlocks = L.smCount * kBigPerSm;
    collide_big_kernel<Real><<<bigBlocks, kBigThreads, arena_bytes<Real>(CellShape<Real>::big), side.stream>>>(a);
    int g = (ncell + kCellWarps - 1) / kCellWarps;
    const int cap = L.smCount * min(CellOcc<Real>::blocks, max(1, L.collideBlocksPerSm));
    if (g > cap) g = cap;
    collide_kernel<Real><<<g > 0 ? g : 1, kCellWarps * 32, kCellWarps * arena_bytes<Real>(CellShape<Real>::arena), s>>>(a, bigBlocks);
    side.join(s);
}

// ===========================================================================
// sampling
// ===========================================================================

// Raw moments of one cell's particles, summed in particle order with each
// operation rounded on its own (the oracle's order and rounding).
template <typename Real>
__device__ __forceinline__ void cell_moments(const PBuf<Real>& b, int s0, int n, double m[18])
{
#pragma unroll
    for (int k = 0; k < 18; ++k) m[k] = 0.0;
    for (int k = s0; k < s0 + n; ++k) {
        const double x = (double)b.v[0][k], y = (double)b.v[1][k], z = (double)b.v[2][k], I = (double)b.ir[k];
        const double v2 = da(da(dm(x, x), dm(y, y)), dm(z, z));
        m[0] = da(m[0], 1.0); m[1] = da(m[1], x); m[2] = da(m[2], y); m[3] = da(m[3], z); m[4] = da(m[4], v2);
        m[5] = da(m[5], dm(x, x)); m[6] = da(m[6], dm(x, y)); m[7] = da(m[7], dm(y, y));
        m[8] = da(m[8], dm(y, z)); m[9] = da(m[9], dm(z, z)); m[10] = da(m[10], dm(z, x));
        m[11] = da(m[11], dm(x, v2)); m[12] = da(m[12], dm(y, v2)); m[13] = da(m[13], dm(z, v2));
        m[14] = da(m[14], I); m[15] = da(m[15], dm(x, I)); m[16] = da(m[16], dm(y, I)); m[17] = da(m[17], dm(z, I));
    }
}

// What a step's sampling does, the same for every cell.
struct FoldStep {
    double w;        // the exponential window's weight of the sum so far
    bool steady;     // past NSS
    bool every;      // a step of the GSIS window
    bool exchange;   // the window's last
};
template <typename Real>
__device__ __forceinline__ FoldStep fold_step(const StepArgs<Real>& a, int istep)
{
    const double na = (double)a.C.nscheme;
    const int ngsis = a.C.nevery * a.C.nrepeat;
    return {istep <= a.C.nscheme ? 1.0 : dd(ds(na, 1.0), na), istep > a.C.nss, istep % a.C.nevery == 0,
            ngsis > 0 && istep % ngsis == 0};
}

// updateStepWindowMoments, :3106-3113, for moment k of a cell: the
// exponential window (local), the steady sum past NSS (final_record) and the
// GSIS window sum (every NEVERY steps)
// (s, sSteady, sWindow: the three accumulators' values before the step).
__device__ __forceinline__ void fold_moment(const FoldStep& f, double* acc, int k, double v, double s, double sSteady,
                                            double sWindow)
{
    acc[k] = (f.w == 1.0) ? da(s, v) : da(dm(f.w, s), v);
    if (f.steady) acc[18 + k] = da(sSteady, v);
    if (f.every) acc[36 + k] = da(sWindow, v);
}

// The rest of statistic_macro for cell c once its moments are folded in:
// the sparse-cell state machine and, at an exchange step, the record fields
// from the GSIS window.
// st, accum: the cell's sparseState and sparseAccum, read only on a step of
// the window (f.every; every exchange step is one)
template <typename Real>
__device__ __forceinline__ void sample_cell_tail(const StepArgs<Real>& a, int c, double* acc, const FoldStep& f,
                                                 unsigned char st, int accum)
{
    if (!f.every) return;
    if (st == 1 || st == 2) {
        if (accum < 0) accum = 0;
        ++accum;
    }
    if (f.exchange) {
        const double S = a.M.cellVolume[c];
        const double* inter = acc + 36;
        const double ws = inter[0];
        const bool finite = isfinite(ws);
        bool sparse = (st == 1 || st == 2);
        if (!sparse && finite && ws < 3.0) {
            st = 1;
            accum = a.C.nrepeat > 1 ? a.C.nrepeat : 1;
            sparse = true;
        }
        const bool valid = (ws >= 3.0) && finite;
        a.windowSamples[c] = ws;
        a.windowValid[c] = valid ? 1 : 0;
        double out[18];
        if (sparse) {
            averaged_macro(inter, (double)(accum > 1 ? accum : 1), S, a.C.neff, a.C.nref, a.C.dr, out);
            for (int k = 0; k < 18; ++k) a.record[(size_t)c * 18 + k] = out[k];
        } else if (valid) {
            averaged_macro(inter, (double)a.C.nrepeat, S, a.C.neff, a.C.nref, a.C.dr, out);
            for (int k = 0; k < 18; ++k) a.record[(size_t)c * 18 + k] = out[k];
        }
        if (!sparse)
            for (int k = 0; k < 18; ++k) acc[36 + k] = 0.0;
    }
    a.sparseState[c] = st;
    a.sparseAccum[c] = accum;
}

// statistic_macroPre (:3312-3326) over the sorted buffer: one thread per cell.
template <typename Real>
__global__ void __launch_bounds__(128) sample_pre_kernel(StepArgs<Real> a)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.M.ncell; c += gridDim.x * blockDim.x) {
        const int s0 = a.startA[c];
        const double S = a.M.cellVolume[c];
        double mom[18], out[18];
        cell_moments<Real>(a.A, s0, a.startA[c + 1] - s0, mom);
        if (a.stepMom)
            for (int k = 0; k < 18; ++k) a.stepMom[(size_t)c * 18 + k] = mom[k];
        local_macro_pre(mom, S, a.C.neff, a.C.nref, a.C.dr, out);
        for (int k = 0; k < 18; ++k) a.local[(size_t)c * 18 + k] = out[k];
        record_macro_pre(mom, S, a.C.neff, a.C.nref, a.C.dr, out);
        for (int k = 0; k < 18; ++k) a.record[(size_t)c * 18 + k] = out[k];
    }
}

// statistic_macro of the mixed path, one warp per cell: the lanes sum the
// cell's particles 32 apart (coalesced loads), lane q < 18 then adds up
// moment q of the 32 lanes (four groups of eight, through shared memory)
// and folds it into the cell's accumulators, and lane 0 runs the rest. Its
// FP64 sums run in another order than the one-thread sums, which the FP64
// path keeps (they are the reference's order).
// A cell is a chain of latencies (its slots, its particles, the sums, its
// state), with 24 warps an SM to cover them. So one wave of blocks takes the
// cells in turn, each warp reading the next cell's slots ahead and the state
// with the accumulators, and of the accumulators and state only what the step
// uses; the step's weight and flags are computed once. 372,500 cells at 100
// particles: 467 -> 363 us; 20,800 at 55: 29.4 -> 19.8; 48,640 at 50: 27.4 ->
// 21.5. Two resident blocks without a spilled register took 439 us, four 486.
constexpr int kSampleWarps = 8;
constexpr int kSamplePerSm = 3;   // resident blocks per SM

__global__ void __launch_bounds__(kSampleWarps * 32, kSamplePerSm) sample_warp_kernel(StepArgs<float> a)
{
    __shared__ double part[kSampleWarps][18][33];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int istep = a.ctl->istep;
    const FoldStep f = fold_step(a, istep);
    double (*mine)[33] = part[wib];
    const int stride = gridDim.x * kSampleWarps;
    int c = blockIdx.x * kSampleWarps + wib;
    int sNext = c < a.M.ncell ? a.startA[c] : 0, eNext = c < a.M.ncell ? a.startA[c + 1] : 0;
    for (; c < a.M.ncell; c += stride) {
        const int s0 = sNext, e = eNext;
        if (c + stride < a.M.ncell) {
            sNext = a.startA[c + stride];
            eNext = a.startA[c + stride + 1];
        }
        double* acc = a.acc + (size_t)c * 54;
        // the accumulators' old values, loaded while the particles are summed
        double o0 = 0.0, o1 = 0.0, o2 = 0.0;
        if (lane < 18) {
            o0 = acc[lane];
            if (f.steady) o1 = acc[18 + lane];
            if (f.every) o2 = acc[36 + lane];
        }
        unsigned char st = 0;
        int accum = 0;
        if (f.every && lane == 0) {
            st = a.sparseState[c];
            accum = a.sparseAccum[c];
        }
        double m[18];
#pragma unroll
        for (int q = 0; q < 18; ++q) m[q] = 0.0;
        auto add = [&](float fx, float fy, float fz, float fi) {
            const double x = (double)fx, y = (double)fy, z = (double)fz, I = (double)fi;
            const double v2 = da(da(dm(x, x), dm(y, y)), dm(z, z));
            m[0] = da(m[0], 1.0); m[1] = da(m[1], x); m[2] = da(m[2], y); m[3] = da(m[3], z); m[4] = da(m[4], v2);
            m[5] = da(m[5], dm(x, x)); m[6] = da(m[6], dm(x, y)); m[7] = da(m[7], dm(y, y));
            m[8] = da(m[8], dm(y, z)); m[9] = da(m[9], dm(z, z)); m[10] = da(m[10], dm(z, x));
            m[11] = da(m[11], dm(x, v2)); m[12] = da(m[12], dm(y, v2)); m[13] = da(m[13], dm(z, v2));
            m[14] = da(m[14], I); m[15] = da(m[15], dm(x, I)); m[16] = da(m[16], dm(y, I)); m[17] = da(m[17], dm(z, I));
        };
        // two particles per lane and iteration, their loads issued first
        int k = s0 + lane;
        for (; k + 32 < e; k += 64) {
            const float x1 = a.A.v[0][k], y1 = a.A.v[1][k], z1 = a.A.v[2][k], i1 = a.A.ir[k];
            const float x2 = a.A.v[0][k + 32], y2 = a.A.v[1][k + 32], z2 = a.A.v[2][k + 32], i2 = a.A.ir[k + 32];
            add(x1, y1, z1, i1);
            add(x2, y2, z2, i2);
        }
        if (k < e) add(a.A.v[0][k], a.A.v[1][k], a.A.v[2][k], a.A.ir[k]);
#pragma unroll
        for (int q = 0; q < 18; ++q) mine[q][lane] = m[q];
        __syncwarp();
        double mq = 0.0;
        if (lane < 18) {
            // four partial sums of eight lanes each, then their pairs
            double t[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                t[g] = mine[lane][8 * g];
#pragma unroll
                for (int l = 1; l < 8; ++l) t[g] = da(t[g], mine[lane][8 * g + l]);
            }
            mq = da(da(t[0], t[1]), da(t[2], t[3]));
        }
        __syncwarp();   // the rows are reused for the next cell
        if (lane < 18) {
            if (a.stepMom) a.stepMom[(size_t)c * 18 + lane] = mq;
            fold_moment(f, acc, lane, mq, o0, o1, o2);
        }
        __syncwarp();   // lane 0 reads the folded window sums
        if (lane == 0) sample_cell_tail(a, c, acc, f, st, accum);
    }
}

// A particle's terms of moments 1..17 handed to f(q, term), each rounded on
// its own as the oracle rounds it (moment 0 counts the particles).
template <typename F>
__device__ __forceinline__ void moment_terms(double x, double y, double z, double I, F&& f)
{
    const double v2 = da(da(dm(x, x), dm(y, y)), dm(z, z));
    f(1, x); f(2, y); f(3, z); f(4, v2);
    f(5, dm(x, x)); f(6, dm(x, y)); f(7, dm(y, y)); f(8, dm(y, z)); f(9, dm(z, z)); f(10, dm(z, x));
    f(11, dm(x, v2)); f(12, dm(y, v2)); f(13, dm(z, v2));
    f(14, I); f(15, dm(x, I)); f(16, dm(y, I)); f(17, dm(z, I));
}

// statistic_macro of the FP64 path: the moments in particle order, each
// operation rounded on its own (the oracle's order and rounding). A warp takes
// a run of `group` consecutive cells: for each, the lanes write the terms of
// 32 particles to shared memory, lane q adds up moment q's, a chain of one
// FP64 addition per particle, and folds it into the cell's accumulators; then
// lane g finishes cell g, so that the states of all cells of the run are read
// together. The next particles are loaded while a chain runs. One thread per
// cell, the same sums took twice as long (uncoalesced loads, cells of unlike
// size in a warp: 63,517 tetrahedra at 100 a cell 341 -> 168 us, 48,640 hexahedra
// at 50 116 -> 55 us, steps 11-20 from the freestream).
constexpr int kOrderedWarps = 4;
constexpr int kOrderedGroup = 32;

__global__ void __launch_bounds__(kOrderedWarps * 32, 6) sample_ordered_kernel(StepArgs<double> a, int group)
{
    __shared__ double part[kOrderedWarps][17][33];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int istep = a.ctl->istep;
    const FoldStep f = fold_step(a, istep);
    const int ncell = a.M.ncell;
    double (*mine)[33] = part[wib];
    const int warps = gridDim.x * kOrderedWarps;
    const int groups = (ncell + group - 1) / group;
    for (int gi = blockIdx.x * kOrderedWarps + wib; gi < groups; gi += warps) {
        const int c0 = gi * group;
        const int cells = min(group, ncell - c0);
        // the run's first slots (group <= 32), and the slot past it
        const int sL = a.startA[min(c0 + lane, ncell)];
        const int sEnd = a.startA[c0 + cells];
        // this lane's particle of the 32 about to be summed
        double px, py, pz, pi;
        auto fetch = [&](int k, int e) {
            if (k < e) { px = a.A.v[0][k]; py = a.A.v[1][k]; pz = a.A.v[2][k]; pi = a.A.ir[k]; }
        };
        int s0 = __shfl_sync(kFull, sL, 0);
        int e = cells > 1 ? __shfl_sync(kFull, sL, 1) : sEnd;
        fetch(s0 + lane, e);
        for (int g = 0; g < cells; ++g) {
            const int c = c0 + g;
            const int n = e - s0;
            const int eNext = g + 2 < cells ? __shfl_sync(kFull, sL, (g + 2) & 31) : sEnd;
            double* acc = a.acc + (size_t)c * 54;
            // the accumulators' old values, loaded while the particles are summed
            double o0 = 0.0, o1 = 0.0, o2 = 0.0;
            if (lane < 18) {
                o0 = acc[lane];
                if (f.steady) o1 = acc[18 + lane];
                if (f.every) o2 = acc[36 + lane];
            }
            double mq = lane == 0 ? (double)n : 0.0;
            for (int base = s0; base < e; base += 32) {
                if (base + lane < e)
                    moment_terms(px, py, pz, pi,
                                 [&](int q, double t) { mine[q - 1][lane] = t; });
                // the following 32 particles, of this cell or the next
                if (base + 32 < e) fetch(base + 32 + lane, e);
                else if (g + 1 < cells) fetch(e + lane, eNext);
                __syncwarp();
                if (lane >= 1 && lane < 18) {
                    const int m = min(32, e - base);
                    const double* row = mine[lane - 1];
                    if (m == 32) {
#pragma unroll
                        for (int l = 0; l < 32; ++l) mq = da(mq, row[l]);
                    } else {
                        for (int l = 0; l < m; ++l) mq = da(mq, row[l]);
                    }
                }
                __syncwarp();   // the rows are reused
            }
            if (n == 0 && g + 1 < cells) fetch(e + lane, eNext);
            if (lane < 18) {
                if (a.stepMom) a.stepMom[(size_t)c * 18 + lane] = mq;
                fold_moment(f, acc, lane, mq, o0, o1, o2);
            }
            s0 = e;
            e = eNext;
        }
        __syncwarp();   // the folded sums are read below
        if (f.every && lane < cells)
            sample_cell_tail(a, c0 + lane, a.acc + (size_t)(c0 + lane) * 54, f, a.sparseState[c0 + lane],
                             a.sparseAccum[c0 + lane]);
        __syncwarp();
    }
}

template <typename Real>
void launch_sample(const StepArgs<Real>& a, bool pre, const LaunchShape& L, cudaStream_t s)
{
    const int ncell = a.M.ncell;
    if (pre) {
        sample_pre_kernel<Real><<<max(1, min((ncell + 127) / 128, L.smCount * 16)), 128, 0, s>>>(a);
    } else if constexpr (sizeof(Real) == 4) {
        const int g = (ncell + kSampleWarps - 1) / kSampleWarps;
        sample_warp_kernel<<<max(1, min(g, L.smCount * kSamplePerSm)), kSampleWarps * 32, 0, s>>>(a);
    } else {
        // runs as long as leave every resident warp (24 an SM) two of them
        const int group = max(1, min(kOrderedGroup, ncell / (L.smCount * 48)));
        const int groups = (ncell + group - 1) / group;
        const int g = (groups + kOrderedWarps - 1) / kOrderedWarps;
        sample_ordered_kernel<<<max(1, min(g, L.smCount * 32)), kOrderedWarps * 32, 0, s>>>(a, group);
    }
}

// ===========================================================================
// initial fill (Np_tri_inititial / meshfillpar / velocityLocationGenerate,
// src/MeshparticalInitial.cpp:481-721): particles already counted per cell
// (startA) and per placement tetrahedron (tetFirst: the cell-local index of
// each tetrahedron's first particle, counted on the host) take, in
// tetrahedron order, a point of their tetrahedron from the reference's
// normalised-uniform weights and a velocity u + sig * (unit Box-Muller
// triple: sqrt(-2 ln r) sin th, sqrt(-2 ln r) cos th, sqrt(-2 ln r2) sin th2)
// with Ir = -ln(r3) tN / 2; u = 0, sig = 1, tN = 1 is the reference's own
// unit Maxwellian at rest. Particle k of cell c draws from the Philox
// counters (c, k, kPurposeFill, 0..4): (r, th), (r2, th2), (r3, w0),
// (w1, w2), (w3, -).
// ===========================================================================
template <typename Real>
__global__ void __launch_bounds__(256) fill_kernel(StepArgs<Real> a, FillParams f, const int* __restrict__ tetFirst)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    constexpr bool mixed = sizeof(Real) == 4;
    constexpr double kTwoPi = 6.283185307179586;   // 2 * M_PI
    for (int c = warp; c < a.M.ncell; c += nwarps) {
        const int s0 = a.startA[c];
        const int n = a.startA[c + 1] - s0;
        const int t0 = a.M.placeOff[c], t1 = a.M.placeOff[c + 1];
        if (n == 0 || t1 <= t0) continue;
        const double cx = a.M.cellCenter[(size_t)c * 3 + 0], cy = a.M.cellCenter[(size_t)c * 3 + 1],
                     cz = a.M.cellCenter[(size_t)c * 3 + 2];
        for (int k = lane; k < n; k += 32) {
            int t = t0;
            for (int q = t0 + 1; q < t1; ++q)
                if (tetFirst[q] <= k) t = q;
            const uint32_t cc = (uint32_t)c, kk = (uint32_t)k;
            const U4 b0 = philox4x32_10(U4{cc, kk, kPurposeFill, 0u}, f.keyLo, f.keyHi);
            const U4 b1 = philox4x32_10(U4{cc, kk, kPurposeFill, 1u}, f.keyLo, f.keyHi);
            const U4 b2 = philox4x32_10(U4{cc, kk, kPurposeFill, 2u}, f.keyLo, f.keyHi);
            const U4 b3 = philox4x32_10(U4{cc, kk, kPurposeFill, 3u}, f.keyLo, f.keyHi);
            const U4 b4 = philox4x32_10(U4{cc, kk, kPurposeFill, 4u}, f.keyLo, f.keyHi);
            const double rad1 = sqrt(dm(-2.0, log(unit64(b0.x, b0.y))));
            const double th1 = dm(kTwoPi, unit64(b0.z, b0.w));
            const double rad2 = sqrt(dm(-2.0, log(unit64(b1.x, b1.y))));
            const double th2 = dm(kTwoPi, unit64(b1.z, b1.w));
            const double ir = dm(dm(-log(unit64(b2.x, b2.y)), f.tN), 0.5);
            double x[3];
            place_point(a.M.placeV + (size_t)t * 12, unit64(b2.z, b2.w), unit64(b3.x, b3.y), unit64(b3.z, b3.w),
                        unit64(b4.x, b4.y), x);
            const int o = s0 + k;
            if constexpr (mixed) {
                a.A.x[0][o] = (Real)(x[0] - cx); a.A.x[1][o] = (Real)(x[1] - cy); a.A.x[2][o] = (Real)(x[2] - cz);
            } else {
                a.A.x[0][o] = x[0]; a.A.x[1][o] = x[1]; a.A.x[2][o] = x[2];
            }
            a.A.v[0][o] = (Real)da(f.u[0], dm(f.sig, dm(rad1, sin(th1))));
            a.A.v[1][o] = (Real)da(f.u[1], dm(f.sig, dm(rad1, cos(th1))));
            a.A.v[2][o] = (Real)da(f.u[2], dm(f.sig, dm(rad2, sin(th2))));
            a.A.ir[o] = (Real)ir;
            a.A.cell[o] = c;
        }
    }
}

template <typename Real>
void launch_fill(const StepArgs<Real>& a, const FillParams& f, const int* tetFirst, const LaunchShape& L,
                 cudaStream_t s)
{
    fill_kernel<Real><<<L.smCount * 8, 256, 0, s>>>(a, f, tetFirst);
}

void launch_scan_counts(const int* countSlot, int ncell, int* partial, int* start, StepCtl* ctl, cudaStream_t s)
{
    scan_partial_kernel<<<kScanBlocks, 256, 0, s>>>(countSlot, ncell, partial);
    scan_final_kernel<<<kScanBlocks, 256, 0, s>>>(countSlot, ncell, partial, start, ctl);
}

// ===========================================================================
// macro fields on demand (local from the exponential window, final_record
// from the steady sum): writeAveragedMacro, src/ProcessDSMC.cpp:2790-2820
// ===========================================================================
__global__ void macro_kernel(DevMesh M, DevConsts C, const double* acc, int set, double count, double* out)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < M.ncell; c += gridDim.x * blockDim.x) {
        double m[18];
        for (int k = 0; k < 18; ++k) m[k] = acc[(size_t)c * 54 + set * 18 + k];
        double o[18];
        averaged_macro(m, count, M.cellVolume[c], C.neff, C.nref, C.dr, o);
        for (int k = 0; k < 18; ++k) out[(size_t)c * 18 + k] = o[k];
    }
}

void launch_macro(const DevMesh& M, const DevConsts& C, const double* acc, int set, double count, double* out,
                  int ncell, cudaStream_t s)
{
    int g = (ncell + 255) / 256;
    if (g > 2048) g = 2048;
    macro_kernel<<<g > 0 ? g : 1, 256, 0, s>>>(M, C, acc, set, count, out);
}

// ===========================================================================
// particle upload from cell-major host arrays
// ===========================================================================
__global__ void upload_check_kernel(const int* __restrict__ cell, int n, int ncell, int* flags)
{
    int bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = cell[i];
        if (c < 0 || c >= ncell) bad |= 1;
        else if (i > 0 && cell[i - 1] > c) bad |= 2;
    }
    if (bad) atomicOr(flags, bad);
}

// start[] of ordered cell ids. Only of those: over unordered ids each rise
// from one particle to the next would write its whole range of cells (516,800
// shuffled particles in 6,080 cells: the upload took 28.5 ms when this ran with
// the check, 12.8 now).
__global__ void upload_layout_kernel(const int* __restrict__ cell, int n, int ncell, const int* flags, int* start)
{
    if (*flags) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = cell[i];
        // cells after the previous particle's, up to c, begin at slot i
        for (int q = i > 0 ? cell[i - 1] + 1 : 0; q <= c; ++q) start[q] = i;
        if (i == n - 1)
            for (int q = c + 1; q <= ncell; ++q) start[q] = n;
    }
}

void launch_upload_check(const int* cell, int n, int ncell, int* flags, int* start, cudaStream_t s)
{
    int g = (n + 255) / 256;
    g = g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g);
    upload_check_kernel<<<g, 256, 0, s>>>(cell, n, ncell, flags);
    upload_layout_kernel<<<g, 256, 0, s>>>(cell, n, ncell, flags, start);
}

__global__ void upload_convert_kernel(const double* __restrict__ in, const int* __restrict__ cell,
                                      const double* __restrict__ center, int comp, float* __restrict__ out, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v = in[i];
        if (comp < 3) v = v - center[(size_t)cell[i] * 3 + comp];
        out[i] = (float)v;
    }
}

void launch_upload_convert(const double* in, const int* cell, const double* center, int comp, float* out, int n,
                           cudaStream_t s)
{
    int g = (n + 255) / 256;
    g = g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g);
    upload_convert_kernel<<<g, 256, 0, s>>>(in, cell, center, comp, out, n);
}

__global__ void download_widen_kernel(const float* __restrict__ in, const int* __restrict__ cell,
                                      const double* __restrict__ center, int comp, double* __restrict__ out, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v = (double)in[i];
        // a slot whose particle the move removed (cell -1, before the sort)
        // has no centre
        if (comp < 3 && cell[i] >= 0) v = da(center[(size_t)cell[i] * 3 + comp], v);
        out[i] = v;
    }
}

void launch_download_widen(const float* in, const int* cell, const double* center, int comp, double* out, int n,
                           cudaStream_t s)
{
    const int g = max(1, min((n + 255) / 256, 148 * 16));
    download_widen_kernel<<<g, 256, 0, s>>>(in, cell, center, comp, out, n);
}

// ===========================================================================
// tracing check (dsmc_trace)
// ===========================================================================
template <typename Real>
__global__ void trace_check_kernel(DevMesh M, DevConsts C, int first, int n, const Real* px, const Real* py, const Real* pz,
                                   const Real* vx, const Real* vy, const Real* vz, const double* dt,
                                   const int* cell, int stopAtWall, int* oCell, int* oIfout, int* oFace,
                                   int* oTri, int* oNcross, int* oLast, Real* ox, Real* oy, Real* oz, Real* ovx,
                                   Real* ovy, Real* ovz, double* odt, unsigned long long* counters)
{
    TraceCounts cnt{};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        PRegs<Real> p;
        int c = cell[i];
        if constexpr (sizeof(Real) == 8) {
            p.x[0] = px[i]; p.x[1] = py[i]; p.x[2] = pz[i];
        } else {
            const double* cc = M.cellCenter + (size_t)c * 3;
            p.x[0] = da(cc[0], (double)px[i]); p.x[1] = da(cc[1], (double)py[i]); p.x[2] = da(cc[2], (double)pz[i]);
        }
        p.v[0] = vx[i]; p.v[1] = vy[i]; p.v[2] = vz[i];
        p.ir = (Real)0;
        Stream rs;
        rs.init((uint32_t)(first + i), 0u, kPurposeWall, C.seedLo, C.seedHi);
        double dtleft = dt[i];
        TraceLog log{-1, 0, 0};
        const int out = trace_particle<Real>(M, C, p, c, -1, -1, dtleft, rs, 0, nullptr, cnt, stopAtWall != 0, &log);
        oCell[i] = (out == kTraceRemoved) ? -1 : c;
        oIfout[i] = (out >= 0) ? out : -1;
        oFace[i] = log.hitFace;
        oTri[i] = log.hitTri;
        oNcross[i] = log.ncross;
        if constexpr (sizeof(Real) == 8) {
            ox[i] = p.x[0]; oy[i] = p.x[1]; oz[i] = p.x[2];
        } else {
            // relative to the centre of the last cell the particle was in
            const double* cc = M.cellCenter + (size_t)c * 3;
            ox[i] = (float)ds(p.x[0], cc[0]); oy[i] = (float)ds(p.x[1], cc[1]); oz[i] = (float)ds(p.x[2], cc[2]);
        }
        ovx[i] = p.v[0]; ovy[i] = p.v[1]; ovz[i] = p.v[2];
        odt[i] = dtleft;
        oLast[i] = c;   // cell the position is relative to (mixed precision)
    }
    flush_counts(counters, cnt);
}

template <typename Real>
void launch_trace_check(const DevMesh& M, const DevConsts& C, int first, int n, const Real* px, const Real* py, const Real* pz,
                        const Real* vx, const Real* vy, const Real* vz, const double* dt, const int* cell,
                        int stopAtWall, int* oCell, int* oIfout, int* oFace, int* oTri, int* oNcross, int* oLast,
                        Real* ox, Real* oy, Real* oz, Real* ovx, Real* ovy, Real* ovz, double* odt,
                        unsigned long long* counters, cudaStream_t s)
{
    int g = (n + 255) / 256;
    if (g > 4096) g = 4096;
    trace_check_kernel<Real><<<g > 0 ? g : 1, 256, 0, s>>>(M, C, first, n, px, py, pz, vx, vy, vz, dt, cell, stopAtWall,
                                                           oCell, oIfout, oFace, oTri, oNcross, oLast, ox, oy, oz,
                                                           ovx, ovy, ovz, odt, counters);
}

#define DSMC_INSTANTIATE(Real)                                                                                   \
    template void launch_inject<Real>(const StepArgs<Real>&, const LaunchShape&, cudaStream_t);                  \
    template void launch_move<Real>(const StepArgs<Real>&, const LaunchShape&, cudaStream_t);                    \
    template void launch_sort<Real>(const StepArgs<Real>&, const LaunchShape&, cudaStream_t);                    \
    template void launch_collide<Real>(const StepArgs<Real>&, const LaunchShape&, cudaStream_t, const SideStream&); \
    template void launch_sample<Real>(const StepArgs<Real>&, bool, const LaunchShape&, cudaStream_t);            \
    template void launch_fill<Real>(const StepArgs<Real>&, const FillParams&, const int*, const LaunchShape&,    \
                                    cudaStream_t);                                                               \
    template cudaError_t prepare_kernels<Real>();                                                                \
    template void launch_trace_check<Real>(const DevMesh&, const DevConsts&, int, int, const Real*, const Real*,  \
                                           const Real*, const Real*, const Real*, const Real*, const double*,    \
                                           const int*, int, int*, int*, int*, int*, int*, int*, Real*, Real*,    \
                                           Real*, Real*, Real*, Real*, double*, unsigned long long*, cudaStream_t);
DSMC_INSTANTIATE(float)
DSMC_INSTANTIATE(double)

}  // namespace dsmc
