// neighbor.cu -- cell binning, cell-ordered permutation and the Verlet list.
//
// Semantics follow the reference CPU cell list
// (src/cpu/neighbor/cell_list.cpp:83-314 grid/stencil/binning and :743-895
// list): a pair {i, j} is listed iff its minimum-image separation, computed
// in FP64 on the rebuild-time coordinates, satisfies r^2 < (cutoff+skin)^2.
// Every product and sum of that test is rounded separately (__dmul_rn /
// __dadd_rn), which is exactly the arithmetic of the FP64 oracle, so the
// pair set equals the oracle's bit for bit.  The list itself is a FULL list
// (each pair stored in both rows) in row-major ELL form with a fixed row
// capacity, so the force kernel needs no atomics and sums every row in a
// fixed order.
#include "atvb_common.cuh"
#include "atvb_kernels.cuh"

namespace atvb {

// Sorted place s of atom i: the permutation, the sorted records and the
// reference positions of the build.
ATVB_DEV void sorted_record(const SysParams& P, int i, int s) {
    const double x = P.x[i], y = P.y[i], z = P.z[i], q = P.q[i];
    P.perm[s] = i;
    P.rank[i] = s;
    P.posd4[s] = make_double4(x, y, z, q);
    int4 v;
    v.x = (int)pos_fix(x, P.fix_scale[0]);
    v.y = (int)pos_fix(y, P.fix_scale[1]);
    v.z = (int)pos_fix(z, P.fix_scale[2]);
    v.w = 0;
    P.lpos[s] = v;
    if (P.prec == kMixed) {
        v.w = __float_as_int((float)q);
        reinterpret_cast<int4*>(P.pos4)[s] = v;
    } else {
        const double xx[3] = {x, y, z};
        reinterpret_cast<double4*>(P.pos4)[s] = pack_pos64(xx, P.fix64_scale, q);
    }
    if (P.ntypes)
        P.stype[s] = (unsigned char)P.type[i];
    P.xr[i] = x;
    P.yr[i] = y;
    P.zr[i] = z;
}

// Cell of atom i.
ATVB_DEV int cell_index(const SysParams& P, int i) {
    const double p[3] = {P.x[i], P.y[i], P.z[i]};
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int cd = (int)floor(p[d] * P.cs_inv[d]);
        cd = cd < 0 ? 0 : (cd > P.nc[d] - 1 ? P.nc[d] - 1 : cd);
        c[d] = cd;
    }
    return (c[0] * P.nc[1] + c[1]) * P.nc[2] + c[2];
}

// Stage 1: cell of every atom (original order) and its arrival slot.
__global__ void k_cell_count(const Item* items, int nitems,
                             const SysParams* sp) {
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        const int i = item.begin + threadIdx.x;
        if (i >= P.n)
            continue;
        const int cell = cell_index(P, i);
        P.cell_of[i] = cell;
        P.slot[i] = atomicAdd(&P.cell_count[cell], 1);
    }
}

// Stages 2 and 3: exclusive scan of the cell counts over chunks of kScanChunk
// cells: the chunk sums, then every chunk's block adds up the sums before its
// own and scans its cells.  One block per system took 440 us at 1,000,188 LJ
// atoms (430k cells walked by 1,024 threads); the two launches take 15 us.
__global__ void __launch_bounds__(kChunk)
    k_cell_sums(const Item* items, int nitems, const SysParams* sp) {
    __shared__ int tot[kChunk / 32];
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        const int* __restrict__ count = P.cell_count;
        int v = 0;
#pragma unroll
        for (int k = 0; k < kScanChunk / kChunk; ++k) {
            const int c = item.begin + k * kChunk + threadIdx.x;
            v += c < P.ncell ? count[c] : 0;
        }
        v = __reduce_add_sync(0xffffffffu, v);
        if ((threadIdx.x & 31) == 0)
            tot[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < kChunk / 32; ++w)
                t += tot[w];
            P.cell_sums[item.begin / kScanChunk] = t;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kChunk)
    k_cell_scan(const Item* items, int nitems, const SysParams* sp) {
    constexpr int kPer = kScanChunk / kChunk;
    __shared__ int tot[kChunk / 32], pre[kChunk / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        const int ncell = P.ncell, chunk = item.begin / kScanChunk;
        int before = 0;
        for (int k = threadIdx.x; k < chunk; k += kChunk)
            before += P.cell_sums[k];
        before = __reduce_add_sync(0xffffffffu, before);
        const int c0 = item.begin + threadIdx.x * kPer;
        int v[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            v[k] = c0 + k < ncell ? P.cell_count[c0 + k] : 0;
            sum += v[k];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += t;
        }
        if (lane == 31)
            tot[w] = incl;
        if (lane == 0)
            pre[w] = before;
        __syncthreads();
        int base = incl - sum;
#pragma unroll
        for (int k = 0; k < kChunk / 32; ++k)
            base += pre[k] + (k < w ? tot[k] : 0);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (c0 + k < ncell) {
                P.cell_start[c0 + k] = base;
                P.cell_count[c0 + k] = 0; // ready for the next rebuild
            }
            base += v[k];
        }
        if (item.begin == 0 && threadIdx.x == 0)
            P.cell_start[ncell] = P.n;
        __syncthreads();
    }
}

// Stage 4: scatter atom ids and the fixed-point z that orders them into
// their cells, in arrival order.
__global__ void k_cell_scatter(const Item* items, int nitems,
                               const SysParams* sp) {
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        const int i = item.begin + threadIdx.x;
        if (i >= P.n)
            continue;
        P.perm0[P.cell_start[P.cell_of[i]] + P.slot[i]] =
            make_int2(i, (int)pos_fix(P.z[i], P.fix_scale[2]));
    }
}

// Stage 5: order each cell by z, ties by original index, so the permutation
// (and with it every later summation order) is independent of atomic arrival
// order.  An atom's place in its cell is the number of the cell's atoms
// before it (independent loads; an insertion sort per cell, a serial chain
// through memory, took 39 us for the 13 atoms per cell of a 1,728-ion melt).
// Cells of a column are consecutive, so a column is one run of atoms in z
// order, and the atoms of it that a sphere cuts out lie close together: the
// pair kernel's gathers then touch fewer lines.  The sorted records, the
// permutation and the reference positions are written here too.
ATVB_DEV int sorted_place(const int2* perm0, int a, int b, int2 me) {
    int s = a;
    for (int k = a; k < b; ++k) {
        const int2 o = __ldcg(perm0 + k);
        s += (unsigned)o.y < (unsigned)me.y || (o.y == me.y && o.x < me.x) ? 1 : 0;
    }
    return s;
}

__global__ void k_permute(const Item* items, int nitems, const SysParams* sp) {
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        const int t = item.begin + threadIdx.x;
        if (t >= P.n)
            continue;
        const int2* __restrict__ perm0 = P.perm0;
        const int2 me = perm0[t];
        const int i = me.x;
        const int c = P.cell_of[i];
        const int a = P.cell_start[c], b = P.cell_start[c + 1];
        const int s = sorted_place(perm0, a, b, me);
        sorted_record(P, i, s);
    }
}

// The whole cell sort of a system of at most kSortSmallAtoms atoms in one
// cluster of eight blocks, with cluster barriers between the stages: one
// launch instead of five on every step of an engine too small for the
// conditional build nodes (about 1 us each on the steps without a build).
// Step of an LJ system with one build in seven, five kernels / one cluster:
// 256 atoms 23.7 / 19.6 us, 4,000 28.1 / 23.6, 8,192 31.2 / 26.0, 16,384 35.8
// / 32.3, 32,768 48.8 / 47.3, 49,152 56.4 / 56.6, 65,536 67.2 / 68.2, 98,000
// 87.1 / 93.0: the line is where they meet (eight SMs build for the rest).
// Data of other blocks of the cluster is read past L1 (__ldcg).
constexpr int kSortThreads = 1024, kSortCtas = 8;

ATVB_DEV void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The int at `p` of this block's shared memory, in block `rank` of the cluster.
ATVB_DEV int cluster_peek(const int* p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(r) : "memory");
    return v;
}

__global__ void __cluster_dims__(kSortCtas, 1, 1) __launch_bounds__(kSortThreads)
    k_sort_small(const int* sys_list, const SysParams* sp) {
    __shared__ int tot[kSortThreads / 32];
    __shared__ int cta_total;
    pdl_sync();
    const SysParams& P = sp[sys_list[blockIdx.x / kSortCtas]];
    if (!P.st->rebuild)
        return; // the whole cluster
    constexpr int T = kSortCtas * kSortThreads;
    const int n = P.n, ncell = P.ncell, tid = threadIdx.x;
    const int rank = blockIdx.x % kSortCtas, gtid = rank * kSortThreads + tid;
    const int lane = tid & 31, w = tid >> 5;
    for (int i = gtid; i < n; i += T) {
        const int c = cell_index(P, i);
        P.cell_of[i] = c;
        P.slot[i] = atomicAdd(&P.cell_count[c], 1);
    }
    cluster_barrier();
    // exclusive scan: each thread a run of cells, the runs' totals within the
    // block, the blocks' totals within the cluster
    const int per = (ncell + T - 1) / T;
    const int c0 = min(gtid * per, ncell), c1 = min(c0 + per, ncell);
    int sum = 0;
    for (int c = c0; c < c1; ++c)
        sum += __ldcg(P.cell_count + c);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += t;
    }
    if (lane == 31)
        tot[w] = incl;
    __syncthreads();
    if (w == 0) {
        int t = tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o)
                t += u;
        }
        tot[lane] = t;
        if (lane == 31)
            cta_total = t;
    }
    cluster_barrier();
    int base = incl - sum + (w > 0 ? tot[w - 1] : 0);
    for (int r = 0; r < rank; ++r)
        base += cluster_peek(&cta_total, r);
    for (int c = c0; c < c1; ++c) {
        const int v = __ldcg(P.cell_count + c);
        P.cell_start[c] = base;
        P.cell_count[c] = 0; // ready for the next rebuild
        base += v;
    }
    if (gtid == 0)
        P.cell_start[ncell] = n;
    cluster_barrier();
    for (int i = gtid; i < n; i += T) // cell and slot of this thread's own atoms
        P.perm0[__ldcg(P.cell_start + P.cell_of[i]) + P.slot[i]] =
            make_int2(i, (int)pos_fix(P.z[i], P.fix_scale[2]));
    cluster_barrier();
    for (int t = gtid; t < n; t += T) {
        const int2 me = __ldcg(P.perm0 + t);
        const int c = __ldcg(P.cell_of + me.x);
        sorted_record(P, me.x,
                      sorted_place(P.perm0, __ldcg(P.cell_start + c), __ldcg(P.cell_start + c + 1),
                                   me));
    }
}

// Exact FP64 pair-set test (same rounding as the oracle built with
// -ffp-contract=off): branchy single-wrap minimum image
// (cell_list.h:214-227), then ((dx*dx + dy*dy) + dz*dz).
ATVB_DEV double exact_r2(const double4& a, const double4& b, const double* L,
                         const double* halfL) {
    double d[3] = {__dadd_rn(a.x, -b.x), __dadd_rn(a.y, -b.y),
                   __dadd_rn(a.z, -b.z)};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (d[k] > halfL[k])
            d[k] = __dadd_rn(d[k], -L[k]);
        else if (d[k] < -halfL[k])
            d[k] = __dadd_rn(d[k], L[k]);
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])),
                     __dmul_rn(d[2], d[2]));
}

// The sorted atoms of stencil column `col` around cell (cx, cy, cz): at most
// two contiguous runs [a0, a0 + l0) and [a1, a1 + l1) (two when the z range
// wraps).  Offsets along an axis stay within one period of the cell index,
// so one conditional add or subtract wraps them (also on an aliased axis,
// whose offsets are absolute cell indices).
ATVB_DEV void column_runs(int nc0, int nc1, int nc2, const int* __restrict__ cstart, int4 col,
                          int cx, int cy, int cz, int& a0, int& l0, int& a1, int& l1) {
    int xx = cx + col.x;
    xx += xx < 0 ? nc0 : (xx >= nc0 ? -nc0 : 0);
    int yy = cy + col.y;
    yy += yy < 0 ? nc1 : (yy >= nc1 ? -nc1 : 0);
    const int base = (xx * nc1 + yy) * nc2;
    int lo0, hi0, lo1 = 0, hi1 = -1;
    if (col.z < 0) {
        lo0 = base;
        hi0 = base + nc2 - 1;
    } else {
        const int z0 = cz - col.z, z1 = cz + col.z;
        if (z0 < 0) {
            lo0 = base + z0 + nc2;
            hi0 = base + nc2 - 1;
            lo1 = base;
            hi1 = base + z1;
        } else if (z1 >= nc2) {
            lo0 = base + z0;
            hi0 = base + nc2 - 1;
            lo1 = base;
            hi1 = base + z1 - nc2;
        } else {
            lo0 = base + z0;
            hi0 = base + z1;
        }
    }
    a0 = cstart[lo0];
    l0 = cstart[hi0 + 1] - a0;
    if (hi1 >= lo1) {
        a1 = cstart[lo1];
        l1 = cstart[hi1 + 1] - a1;
    } else {
        a1 = 0;
        l1 = 0;
    }
}

// Special class (1: 1-2, 2: 1-3, 3: 1-4, 0: none) of sorted pair (i, j):
// a scan of i's few special partners, by original index.
ATVB_DEV unsigned special_class(const SysParams& P, int i, int j) {
    const int io = P.perm[i], jo = P.perm[j];
    for (int q = P.sp_first[io]; q < P.sp_first[io + 1]; ++q)
        if (P.sp_j[q] == jo)
            return P.sp_cls[q];
    return 0u;
}

// Stage 6 (items of kListChunk warp tasks): 2^split_log2 warps per cell, each
// for its share of the cell's atoms (one warp per cell once the cells alone
// fill the GPU; the rows do not depend on the split).  Every atom of a cell
// has the same stencil, so the warp resolves the stencil columns once (up to
// 32 at a time, one per lane, into runs of sorted atoms laid end to end by a
// warp prefix sum), loads each window of 32 consecutive candidates once, and
// tests it against kListAtoms atoms of the cell, appending hits to each
// atom's row with a ballot.  Rows list candidates in column order.
//
// The test is FP32, in the frame of the cell's first atom (exact 32-bit
// fixed-point differences, rounded to FP32 once); FOLD adds the minimum
// image of the difference, for boxes where two such coordinates can lie
// further apart than half an edge.  Its error is bounded (apply_box): below
// fband_lo a candidate is certainly listed, at or above fband_hi certainly
// not.  A candidate in between is appended, and a row that got one is
// settled once it is complete (settle_row; exact_rows if it has outgrown its
// places) by the exact FP64 test, so the listed set and its length are exactly
// the FP64 ones.
//
// Bound by instruction issue (63 % of the issue slots at 24 warps per SM).
// What a window costs before its first atom (finding each lane's column,
// loading and converting the candidate) is shared by the atoms of the cell;
// candidates of the error band are settled per row, not per window, so the
// window loop has no rare path.  At 8 atoms per pass and 24 warps, cell sort
// and build per step with one build in nine: 1,000,188 LJ atoms 332 -> 147
// us, the 262,144-ion melt 184 -> 141 us, 24 LJ replicas of 256 to 32,768
// atoms 90 -> 68 us (16 warps: 175 / 171 / 72; 4 atoms per pass: 162 / 163 / 72).
constexpr int kListAtoms = 8;
constexpr int kListWarps = kListChunk;
constexpr int kListBlocks = 6; // per SM: 24 warps of 80 registers

// FP32 squared distance of two points of the cell's frame.
template <bool FOLD>
ATVB_DEV float frame_r2(float Lx, float Ly, float Lz, float ax, float ay, float az, float rx,
                        float ry, float rz) {
    float dx = ax - rx, dy = ay - ry, dz = az - rz;
    if (FOLD) {
        dx = fminf(fabsf(dx), Lx - fabsf(dx));
        dy = fminf(fabsf(dy), Ly - fabsf(dy));
        dz = fminf(fabsf(dz), Lz - fabsf(dz));
    }
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// A point of the frame whose origin is `org`.
ATVB_DEV float3 frame_pos(const SysParams& P, int4 q, int4 org) {
    return make_float3((float)(int)((unsigned)q.x - (unsigned)org.x) * P.Lf_fix[0],
                       (float)(int)((unsigned)q.y - (unsigned)org.y) * P.Lf_fix[1],
                       (float)(int)((unsigned)q.z - (unsigned)org.z) * P.Lf_fix[2]);
}

// Row i has its final length: more than its places is reported.
ATVB_DEV void row_done(const SysParams& P, int i, int len) {
    P.nnbr[i] = min(len, P.cap);
    if (len > P.cap) {
        // the row is cut: pairs are missing until rows are widened
        atomicOr(&P.st->overflow, 1);
        atomicOr(&P.st->status, kStatusRowOverflow);
    }
}

// The rows of cell c among those of atoms [cs, ce) that build_share left open
// (length -1): they have candidates of the error band and, with them, more
// entries than places, so which of those not stored are pairs could not be
// told afterwards, nor whether the row fits.  Built from the start in the same
// order, every candidate decided by the exact FP64 test before it is counted.
// A call inside build_share costs it registers: cell sort and build of a
// million atoms 146.0 us a step without these rows, 147.5 with them, 148.9
// with the call inside (262,144 ions 131.3, 131.8, 133.1).
__device__ __noinline__ void exact_rows(const SysParams& P, int c, int cs, int ce, int* s_max,
                                        unsigned* s_sum) {
    const int lane = threadIdx.x & 31;
    const double L[3] = {P.L[0], P.L[1], P.L[2]};
    const double hL[3] = {P.halfL[0], P.halfL[1], P.halfL[2]};
    const double rl2 = P.rlist2;
    const int nc0 = P.nc[0], nc1 = P.nc[1], nc2 = P.nc[2];
    const int cz = c % nc2, cy = (c / nc2) % nc1, cx = c / (nc1 * nc2);
    for (int i = cs; i < ce; ++i) {
        if (P.nnbr[i] >= 0)
            continue; // warp-uniform
        int* row = P.nbr + (size_t)i * P.cap;
        const double4 a = P.posd4[i];
        int len = 0;
        __syncwarp();
        for (int col = 0; col < P.ncol; ++col) {
            int a0, l0, a1, l1;
            column_runs(nc0, nc1, nc2, P.cell_start, P.cols[col], cx, cy, cz, a0, l0, a1, l1);
            for (int t0 = 0; t0 < l0 + l1; t0 += 32) {
                const int t = t0 + lane;
                const int j = t < l0 ? a0 + t : a1 + t - l0;
                const bool hit =
                    t < l0 + l1 && j != i && exact_r2(a, P.posd4[j], L, hL) < rl2;
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                const int w = len + __popc(m & ((1u << lane) - 1u));
                if (hit && w < P.cap)
                    row[w] = (int)((unsigned)j |
                                   (P.has_special ? special_class(P, i, j) << 30 : 0u));
                len += __popc(m);
            }
        }
        if (lane == 0) {
            row_done(P, i, len);
            atomicMax(s_max, len);
            atomicAdd(s_sum, (unsigned)len);
        }
    }
}

// The entries of atom i's row (cnt of them, all stored) whose FP32 distance is
// in the error band, decided by the exact FP64 test: the row is compacted in
// place, in order.  About one row in a thousand.  Returns the new length.
__device__ __noinline__ int settle_row(const SysParams& P, int i, int org_i, int cnt) {
    const int lane = threadIdx.x & 31;
    int* row = P.nbr + (size_t)i * P.cap;
    const double L[3] = {P.L[0], P.L[1], P.L[2]};
    const double hL[3] = {P.halfL[0], P.halfL[1], P.halfL[2]};
    const float Lx = (float)L[0], Ly = (float)L[1], Lz = (float)L[2];
    const double rl2 = P.rlist2;
    const bool fold = !P.lframe_ok;
    const int4 org = P.lpos[org_i];
    const float3 a = frame_pos(P, P.lpos[i], org);
    int out = 0;
    __syncwarp();
    for (int k0 = 0; k0 < cnt; k0 += 32) {
        const int k = k0 + lane;
        int e = 0;
        bool keep = k < cnt;
        if (keep) {
            e = row[k];
            const int j = e & (int)kRowIdxMask;
            const float3 r = frame_pos(P, P.lpos[j], org);
            const float r2 = fold ? frame_r2<true>(Lx, Ly, Lz, a.x, a.y, a.z, r.x, r.y, r.z)
                                  : frame_r2<false>(Lx, Ly, Lz, a.x, a.y, a.z, r.x, r.y, r.z);
            if (!(r2 < P.fband_lo))
                keep = exact_r2(P.posd4[i], P.posd4[j], L, hL) < rl2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep)
            row[out + __popc(m & ((1u << lane) - 1u))] = e;
        out += __popc(m);
        __syncwarp();
    }
    return out;
}

template <bool FOLD, bool SP>
ATVB_DEV void build_share(const SysParams& P, int c, int cs, int ce, int lane,
                          float4* __restrict__ sr, int4* __restrict__ sc, int* s_max,
                          unsigned* s_sum, int* s_open) {
    const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
    // every field the loops use, read once: the row stores below could alias
    // SysParams as far as the compiler knows
    const int4* __restrict__ lp = P.lpos;
    const int* __restrict__ cstart = P.cell_start;
    const float sx = P.Lf_fix[0], sy = P.Lf_fix[1], sz = P.Lf_fix[2];
    const float flo = P.fband_lo, fhi = P.fband_hi;
    const float Lx = (float)P.L[0], Ly = (float)P.L[1], Lz = (float)P.L[2];
    const int nc0 = P.nc[0], nc1 = P.nc[1], nc2 = P.nc[2], ncol = P.ncol;
    const unsigned cap = (unsigned)P.cap;
    const int4* __restrict__ cols = P.cols;
    const int cz = c % nc2, cy = (c / nc2) % nc1, cx = c / (nc1 * nc2);
    const int4 org = lp[cs];
    int incl = 0, total = 0;
    for (int i0 = cs; i0 < ce; i0 += kListAtoms) {
        const int ni = min(kListAtoms, ce - i0);
        __syncwarp();
        if (lane < ni) {
            const int4 q = lp[i0 + lane];
            sr[lane] = make_float4((float)(int)((unsigned)q.x - (unsigned)org.x) * sx,
                                   (float)(int)((unsigned)q.y - (unsigned)org.y) * sy,
                                   (float)(int)((unsigned)q.z - (unsigned)org.z) * sz, 0.0f);
        }
        unsigned* const rows = reinterpret_cast<unsigned*>(P.nbr) + (size_t)i0 * cap;
        unsigned off[kListAtoms]; // a * cap + the length of atom i0 + a's row so far
#pragma unroll
        for (int a = 0; a < kListAtoms; ++a)
            off[a] = a * cap;
        unsigned amb = 0; // bit a: this lane appended a candidate of the band
        for (int c0 = 0; c0 < ncol; c0 += 32) {
            if (ncol > 32 || i0 == cs) {
                int a0 = 0, l0 = 0, a1 = 0, l1 = 0;
                if (c0 + lane < ncol)
                    column_runs(nc0, nc1, nc2, cstart, cols[c0 + lane], cx, cy, cz, a0, l0,
                                a1, l1);
                const int tot = l0 + l1;
                incl = tot;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(full, incl, o);
                    if (lane >= o)
                        incl += t;
                }
                // candidate t of this column: t + x up to place y, then t + z
                const int excl = incl - tot;
                __syncwarp();
                sc[lane] = make_int4(a0 - excl, excl + l0, a1 - l0 - excl, 0);
                total = __shfl_sync(full, incl, 31);
            }
            __syncwarp();
            // candidate t = b + lane of the window, and its position
            auto fetch = [&](int b, int4& q) {
                const int t = b + lane;
                // owner column: the first lane whose inclusive sum exceeds t
                int own = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int probe = __shfl_sync(full, incl, own + step - 1);
                    if (probe <= t)
                        own += step;
                }
                const int4 k = sc[own & 31];
                const int j = t < total ? (t < k.y ? t + k.x : t + k.z) : -1;
                if (j >= 0)
                    q = lp[j];
                return j;
            };
            int4 qn = make_int4(0, 0, 0, 0);
            int jn = total > 0 ? fetch(0, qn) : -1;
            for (int b = 0; b < total; b += 32) {
                const int j = jn;
                const int4 q = qn;
                if (b + 32 < total)
                    jn = fetch(b + 32, qn);
                float rx = (float)(int)((unsigned)q.x - (unsigned)org.x) * sx;
                const float ry = (float)(int)((unsigned)q.y - (unsigned)org.y) * sy;
                const float rz = (float)(int)((unsigned)q.z - (unsigned)org.z) * sz;
                if (j < 0)
                    rx = __int_as_float(0x7fc00000); // NaN: never a hit
                const int jrel = j - i0; // == a: the atom itself
#pragma unroll
                for (int a = 0; a < kListAtoms; ++a) {
                    if (a >= ni)
                        break; // warp-uniform
                    const float4 r = sr[a];
                    const float r2 = frame_r2<FOLD>(Lx, Ly, Lz, r.x, r.y, r.z, rx, ry, rz);
                    // no branches but the one on a: a divergent region costs
                    // more than the few instructions it would skip
                    const bool hit = r2 < fhi && jrel != a;
                    const unsigned m = __ballot_sync(full, hit);
                    const unsigned w = off[a] + (unsigned)__popc(m & lt);
                    amb = hit && !(r2 < flo) ? amb | (1u << a) : amb;
                    unsigned e = (unsigned)j;
                    if (SP && hit)
                        e |= special_class(P, i0 + a, j) << 30;
                    if (hit && w < (a + 1u) * cap)
                        rows[w] = e;
                    off[a] += (unsigned)__popc(m);
                }
            }
        }
        amb = __reduce_or_sync(full, amb);
        int cnt = 0; // row length of atom i0 + lane
#pragma unroll
        for (int a = 0; a < kListAtoms; ++a) {
            if (a >= ni)
                break;
            int len = (int)(off[a] - a * cap);
            if (amb & (1u << a)) {
                if (len <= (int)cap) {
                    len = settle_row(P, i0 + a, cs, len);
                } else { // left to exact_rows
                    len = -1;
                    *s_open = 1;
                }
            }
            if (lane == a)
                cnt = len;
        }
        const int wmax = __reduce_max_sync(full, cnt);
        const int wsum = __reduce_add_sync(full, max(cnt, 0));
        if (lane == 0) {
            atomicMax(s_max, wmax);
            atomicAdd(s_sum, (unsigned)wsum);
        }
        if (lane < ni)
            row_done(P, i0 + lane, cnt);
    }
}

__global__ void __launch_bounds__(32 * kListWarps, kListBlocks)
    k_build_list(const Item* items, int nitems, const SysParams* sp, int split_log2) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float4 sr[kListWarps][kListAtoms];
    __shared__ int4 sc[kListWarps][32];
    // the longest row and the number of entries of the rows built so far by
    // this block, added to the system once per block and system (one atomic
    // of each per atom serialises on one address: 2,000,376 of them took
    // 0.5 ms of the build of 1,000,188 LJ atoms)
    __shared__ int s_max;
    __shared__ unsigned s_sum;
    __shared__ int s_open[kListWarps]; // the warp's share has rows for exact_rows
    int cur = -1;
    auto flush = [&] { // block-uniform
        __syncthreads();
        if (threadIdx.x == 0 && cur >= 0) {
            SysState* st = sp[cur].st;
            if (s_max > 0)
                atomicMax(&st->max_nnbr, s_max);
            if (s_sum)
                atomicAdd(&st->list_entries, (unsigned long long)s_sum);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_max = 0;
            s_sum = 0;
        }
        __syncthreads();
    };
    pdl_sync();
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const Item item = items[it];
        const SysParams& P = sp[item.sys];
        if (!P.st->rebuild)
            continue;
        if (item.sys != cur) {
            flush();
            cur = item.sys;
        }
        const int task = item.begin + warp;
        const int c = task >> split_log2;
        if (c >= P.ncell)
            continue; // warp-uniform
        // this warp's share of the cell's atoms
        const int c_lo = P.cell_start[c], c_n = P.cell_start[c + 1] - c_lo;
        const int part = task & ((1 << split_log2) - 1);
        const int cs = c_lo + ((c_n * part) >> split_log2);
        const int ce = c_lo + ((c_n * (part + 1)) >> split_log2);
        if (cs >= ce)
            continue;
        if (lane == 0)
            s_open[warp] = 0;
        __syncwarp();
        if (P.lframe_ok) {
            if (P.has_special)
                build_share<false, true>(P, c, cs, ce, lane, sr[warp], sc[warp], &s_max, &s_sum,
                                         &s_open[warp]);
            else
                build_share<false, false>(P, c, cs, ce, lane, sr[warp], sc[warp], &s_max,
                                          &s_sum, &s_open[warp]);
        } else {
            if (P.has_special)
                build_share<true, true>(P, c, cs, ce, lane, sr[warp], sc[warp], &s_max, &s_sum,
                                        &s_open[warp]);
            else
                build_share<true, false>(P, c, cs, ce, lane, sr[warp], sc[warp], &s_max,
                                         &s_sum, &s_open[warp]);
        }
        __syncwarp();
        const bool open = s_open[warp] != 0;
        __syncwarp();
        if (open)
            exact_rows(P, c, cs, ce, &s_max, &s_sum);
    }
    if (cur >= 0)
        flush();
}

// Binning and the sorted repack: after these the sorted positions (pos4)
// that the PME chain reads are final, so that chain may start beside the
// list build.
void launch_sort_cells(const LaunchCfg& lc, cudaStream_t s, bool pdl) {
    if (lc.nsmall) {
        launch_k(k_sort_small, lc.nsmall * kSortCtas, kSortThreads, 0, s, pdl, lc.small_list,
                 lc.sp);
        pdl = lc.pdl;
    }
    if (lc.sort_atoms.n) {
        const ItemList &A = lc.sort_atoms, &S = lc.scan;
        launch_k(k_cell_count, A.grid, kChunk, 0, s, pdl, A.d, A.n, lc.sp);
        launch_k(k_cell_sums, S.grid, kChunk, 0, s, lc.pdl, S.d, S.n, lc.sp);
        launch_k(k_cell_scan, S.grid, kChunk, 0, s, lc.pdl, S.d, S.n, lc.sp);
        launch_k(k_cell_scatter, A.grid, kChunk, 0, s, lc.pdl, A.d, A.n, lc.sp);
        launch_k(k_permute, A.grid, kChunk, 0, s, lc.pdl, A.d, A.n, lc.sp);
    }
}

void launch_build_list(const LaunchCfg& lc, cudaStream_t s, bool pdl) {
    launch_k(k_build_list, lc.list.grid, 32 * kListChunk, 0, s, pdl, lc.list.d, lc.list.n, lc.sp,
             lc.list_split_log2);
}

void launch_rebuild(const LaunchCfg& lc, cudaStream_t s) {
    launch_sort_cells(lc, s, false);
    launch_build_list(lc, s, false);
}

} // namespace atvb
