// k_nblist.cu -- the optional cutoff mode of the nonbond pass: a Verlet
// neighbour list over per-window cell lists, rebuilt on the device.
//
// The reference's live path has no cutoff: its nonbond kernel evaluates every
// pair (nonbond_force_cuda.cu:31-174; the `rCut2` it is handed is unused), and
// its neighbour-list and cell-list kernels (neighborlist_cuda.cu:11-137,
// cell_list_cuda.cu:13-35) are built but never called.  Here a cutoff rc > 0
// truncates all three nonbond terms (LJ, Coulomb, IS-SPA correction) at rc with
// no shift: a pair counts iff its FP32 squared minimum-image distance is below
// rc^2.  Per step:
//   check    every atom's displacement since the last build; any beyond half
//            the skin (or the first step) flags a rebuild, and then the launch's
//            last block makes the cells: cell of every atom (cells per window
//            edge nc = floor(box / (1.0001 (rc + skin))), or the whole window as
//            one cell when nc < 3), cell starts, atoms into their cells;
//   pairs    per atom, the row's pairs closer than rc; flagged, the row first:
//            every partner within rc + skin from the 27 neighbouring cells (or
//            the whole window), with the exclusion bit from the atom's sorted
//            exclusion list (excluded pairs keep the IS-SPA correction,
//            nonbond_force_cuda.cu:153-162).
// Between the steps of one graph the check is the update's (nbl_leapfrog_kernel),
// so such a step is pairs and update.  As six launches (check, bin, scan, scatter,
// rows, pairs) and the update a step spent most of its time in launches with
// nothing to do.  Us per solvent-free step, rc 12 A, a build in about 25 steps:
// 264 atoms 13.3 -> 10.1, 1100 15.4 -> 10.4, 8800 21.9 -> 17.3, 66 000 68.9 ->
// 67.2, 264 000 272 -> 254.
// A pair within rc now was within rc + skin at the last build, because no atom
// has since moved more than skin / 2, so the pairs evaluated are exactly the
// pairs within rc.  Every pair's force is rounded to the fixed-point grid on
// its own and summed as integers, so the force does not depend on the order of
// a row, on the skin or on when the list was rebuilt.
#include <climits>
#include <cmath>

#include "kernels.h"
#include "md_device.cuh"
#include "philox.h"

namespace isspa {
namespace {

constexpr int kNblThreads = 256;  // 8 warps: one atom per warp
constexpr unsigned kFull = 0xffffffffu;

// Cell coordinate in [0, nc) of a coordinate wrapped into the box (any finite
// or non-finite x maps into range; non-finite positions are reported by the
// force checks).
__device__ __forceinline__ int cell_coord(float x, float scale, int nc) {
    int c = (int)floorf(x * scale) % nc;
    return c < 0 ? c + nc : c;
}

// j in the sorted exclusion list ex[lo, end)?
__device__ __forceinline__ bool excluded(const int *ex, int lo, int end, int j) {
    int hi = end;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ex[mid] < j) lo = mid + 1;
        else hi = mid;
    }
    return lo < end && ex[lo] == j;
}

__device__ __forceinline__ bool nbl_moved(const NbListArgs &a, int i, float4 p) {
    const WinDev &W = a.win[a.atom_win[i]];
    const float L = W.box, h = W.hbox;
    const float4 r = a.ref[i];
    const float d2 = dist2f(mimg(p.x - r.x, L, h), mimg(p.y - r.y, L, h), mimg(p.z - r.z, L, h));
    return !(d2 <= a.half_skin2);  // NaN (before the first build) rebuilds
}

__device__ __forceinline__ int cell_index(int4 wc, float4 p) {  // wc: first cell, cells per edge, scale bits, -
    const int nc = wc.y;
    const float sc = __int_as_float(wc.z);
    if (nc <= 1) return wc.x;
    return wc.x + (cell_coord(p.x, sc, nc) * nc + cell_coord(p.y, sc, nc)) * nc + cell_coord(p.z, sc, nc);
}

// Exclusive scan over the block of one value per thread; `carry` runs on from
// call to call.
template <int T>
__device__ __forceinline__ int scan_block(int v, int *s_warp, int &carry) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // s_warp has been read
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    int before = carry + x - v;
#pragma unroll
    for (int q = 0; q < T / 32; ++q) {
        const int y = s_warp[q];
        if (q < wid) before += y;
        carry += y;
    }
    return before;
}

// The cells of the current positions by one block, about once in thirty steps:
// atoms counted per cell and given their places by shared-memory atomics (8800
// atoms: a check with the build takes 21 us, 28 with global ones).  Positions are
// read through L2 (they may be this launch's), indices clamped instead of
// predicated, so that the loads of one kind go out together.  Up to kNblBlockCells
// cells (32 KB); beyond, nbl_bin_kernel, nbl_scan_kernel and nbl_scatter_kernel do
// it on the whole chip, a check in every step: us per step that way / this way,
// 1100 atoms 14.3 / 10.4, 8800 22.8 / 17.3, 22 000 33.2 / 29.4, 66 000 68.6 / 67.2,
// so the limit lies near where one block's share would cost what they do.
constexpr int kNblCheckThreads = 256;
constexpr int kNblBlockCells = 8192;
constexpr int kNblPerThread = 4;  // a row's candidates in flight per lane
__device__ __noinline__ void nbl_cells_block(const NbListArgs &a, int *s_cell /* [n_cells] */) {
    constexpr int kT = kNblCheckThreads, kU = 8;
    __shared__ int s_warp[kT / 32];
    const int t = threadIdx.x;
    if (t == 0) {
        a.stats[0] += 1;  // builds so far
        a.stats[1] = 0;   // fullest row of this build
    }
    for (int c = t; c < a.n_cells; c += kT) s_cell[c] = 0;
    __syncthreads();
    for (int base = t; base < a.n_atoms; base += kU * kT) {
        int4 wc[kU];
        float4 p[kU];
        int w[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = min(base + u * kT, a.n_atoms - 1);
            w[u] = a.atom_win[i];
            p[u] = __ldcg(a.pos + i);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) wc[u] = a.wcell[w[u]];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = base + u * kT;
            if (i >= a.n_atoms) break;
            const int c = cell_index(wc[u], p[u]);
            a.cell_of[i] = c;
            atomicAdd(s_cell + c, 1);
        }
    }
    int carry = 0;
    for (int base = 0; base < a.n_cells; base += kT) {
        const int c = base + t;
        if (base == 0) __syncthreads();  // counts complete
        const int v = c < a.n_cells ? s_cell[c] : 0;
        const int before = scan_block<kT>(v, s_warp, carry);
        if (c < a.n_cells) {
            a.cell_start[c] = before;
            s_cell[c] = before;
        }
    }
    if (t == 0) a.cell_start[a.n_cells] = carry;
    __syncthreads();
    for (int base = t; base < a.n_atoms; base += kU * kT) {
        int c[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) c[u] = a.cell_of[min(base + u * kT, a.n_atoms - 1)];
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (base + u * kT < a.n_atoms) a.cell_atoms[atomicAdd(s_cell + c[u], 1)] = base + u * kT;
    }
}

__global__ void nbl_bin_kernel(NbListArgs a) {
    if (!*a.flag) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_atoms) return;
    const int c = cell_index(a.wcell[a.atom_win[i]], a.pos[i]);
    a.cell_of[i] = c;
    atomicAdd(a.cell_count + c, 1);
}

// Starts and scatter cursors from the counts, which are cleared for the next
// build; one block.
__global__ void __launch_bounds__(1024) nbl_scan_kernel(NbListArgs a) {
    if (!*a.flag) return;
    __shared__ int s_warp[32];
    const int t = threadIdx.x;
    if (t == 0) {
        a.stats[0] += 1;
        a.stats[1] = 0;
    }
    int carry = 0;
    for (int base = 0; base < a.n_cells; base += 1024) {
        const int c = base + t;
        const int before = scan_block<1024>(c < a.n_cells ? a.cell_count[c] : 0, s_warp, carry);
        if (c < a.n_cells) {
            a.cell_start[c] = before;
            a.cell_cursor[c] = before;
            a.cell_count[c] = 0;
        }
    }
    if (t == 0) a.cell_start[a.n_cells] = carry;
}

__global__ void nbl_scatter_kernel(NbListArgs a) {
    if (!*a.flag) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.n_atoms) a.cell_atoms[atomicAdd(a.cell_cursor + a.cell_of[i], 1)] = i;
}

// True in the last block of the launch to come here (in all its threads, with the
// other blocks' writes visible); every thread calls it, and `count` is zero at rest.
__device__ __forceinline__ bool last_block(unsigned int *count) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(count, 1u) == gridDim.x - 1;
    __syncthreads();
    if (s_last && threadIdx.x == 0) *count = 0u;
    if (s_last) __threadfence();
    return s_last != 0;
}

__global__ void __launch_bounds__(kNblCheckThreads) nbl_check_kernel(NbListArgs a) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool move = i < a.n_atoms && nbl_moved(a, i, a.pos[i]);
    if (__any_sync(kFull, move) && (threadIdx.x & 31) == 0) atomicOr(a.flag, 1);
    extern __shared__ int s_cell[];
    if (last_block(a.count) && a.block_cells && __ldcg(a.flag)) nbl_cells_block(a, s_cell);
}

// The update followed by the check of the next step (same arithmetic as
// leapfrog_kernel and nbl_check_kernel, whose completion count it shares).
__global__ void __launch_bounds__(kNblCheckThreads) nbl_leapfrog_kernel(LeapfrogArgs f, NbListArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const uint32_t step = *f.step_ptr;
    bool move = false;
    if (i < f.n_atoms) {
        leapfrog_atom(f, i, step, nullptr);
        move = nbl_moved(a, i, f.pos[i]);
    }
    if (__any_sync(kFull, move) && (threadIdx.x & 31) == 0) atomicOr(a.flag, 1);
    if (!last_block(a.count)) return;
    if (threadIdx.x == 0) {
        *f.step_ptr = step + 1u;
        if (f.ov_epoch) ++*f.ov_epoch;
    }
    extern __shared__ int s_cell[];
    if (__ldcg(a.flag)) nbl_cells_block(a, s_cell);
}

// One warp: atom i's partners within rc + skin, compacted by ballot; returns
// their number.  Entries are j | (excluded << 31); a row holds at most row_cap of
// them (the count beyond that is kept and reported).  With rows == nullptr only
// the counts are taken (sizing the rows at engine creation).
// The 27 cells (the lanes hold their starts) are walked as one list of
// candidates, kNblPerThread to a lane at a time: cell by cell the walk is a chain
// of 27 x 3 dependent loads (8800 atoms: a pairs launch with the build 61 us, as
// one list 42).
// (A call of its own: inlined, its registers cost the pairs pass a third of its
// warps.)
__device__ __noinline__ int nbl_build_row(const NbListArgs &a, int i, int lane, float4 xi) {
    constexpr int kU = kNblPerThread;
    const WinDev &W = a.win[a.atom_win[i]];
    const int4 wc = a.wcell[a.atom_win[i]];
    const float L = W.box, h = W.hbox;
    const int e0 = a.excl_start[i], e1 = a.excl_start[i + 1];
    const int ex0 = e0 < e1 ? a.excl[e0] : INT_MAX, ex1 = e0 < e1 ? a.excl[e1 - 1] : -1;
    int *row = a.rows ? a.rows + (long long)i * a.row_cap : nullptr;
    const bool cells = wc.y > 1;
    // lane's cell: its atoms are candidates [upto - its number, upto), at
    // cell_atoms[candidate + shift]
    int upto = 0, shift = 0, total = W.n_atoms;
    if (cells) {
        const int nc = wc.y;
        const int r = a.cell_of[i] - wc.x;
        const int cz = r % nc, cy = (r / nc) % nc, cx = r / (nc * nc);
        int k0 = 0, n = 0;
        if (lane < 27) {
            const int c = wc.x + (((cx + lane / 9 + nc - 1) % nc) * nc + (cy + lane / 3 % 3 + nc - 1) % nc) * nc +
                          (cz + lane % 3 + nc - 1) % nc;
            k0 = a.cell_start[c];
            n = a.cell_start[c + 1] - k0;
        }
        upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, upto, o);
            if (lane >= o) upto += y;
        }
        shift = k0 - (upto - n);
        total = __shfl_sync(kFull, upto, 31);
    }
    int count = 0;
    for (int base = 0; base < total; base += 32 * kU) {
        int j[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = base + 32 * u + lane;
            j[u] = W.atom_off + q;
            if (cells) {  // the first cell with upto > q
                int c = 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    if (__shfl_sync(kFull, upto, c + o - 1) <= q) c += o;
                const int at = q + __shfl_sync(kFull, shift, c);
                j[u] = q < total ? a.cell_atoms[at] : -1;
            }
            if (q >= total || j[u] == i) j[u] = -1;
        }
        float4 xj[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) xj[u] = a.pos[max(j[u], 0)];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const float d2 = dist2f(mimg(xi.x - xj[u].x, L, h), mimg(xi.y - xj[u].y, L, h), mimg(xi.z - xj[u].z, L, h));
            const bool hit = j[u] >= 0 && d2 < a.list2;
            const unsigned m = __ballot_sync(kFull, hit);
            if (hit && row) {
                const bool ex = j[u] >= ex0 && j[u] <= ex1 && excluded(a.excl, e0, e1, j[u]);
                const int slot = count + __popc(m & ((1u << lane) - 1u));
                if (slot < a.row_cap) row[slot] = j[u] | (ex ? INT_MIN : 0);
            }
            __syncwarp();
            count += __popc(m);
        }
    }
    if (lane == 0) {
        a.row_n[i] = count;
        a.ref[i] = xi;
        atomicMax(a.stats + 1, count);
        if (row && count > a.row_cap) atomicOr(a.status, kStatusListFull);
    }
    return count;
}

__global__ void nbl_count_kernel(NbListArgs a) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i < a.n_atoms) nbl_build_row(a, i, threadIdx.x & 31, a.pos[i]);
}

// One warp per atom over its row: the pairs closer than rc, each force rounded
// to the fixed-point grid on its own (order-free integer sums).  Pair forces
// as the all-pairs kernel: LJ r^-6 (12A r^-6 - 6B) / r^2 (nonbond_force_cuda.cu:
// 131-132), Coulomb q q / r^3 (:136), IS-SPA correction with the partner's
// rmax (:141-147), excluded pairs the correction only (:153-162).
//
// A step of a few thousand atoms is one wave of warps that each wait for a chain
// of loads (row, partner, its type, its parameters, its position).  All but the
// positions outlive a step, so a programmatic launch fetches them while the
// kernel before it ends, for the row's first 32 kNblAhead entries: that kernel
// (the update or the check) triggers after its own wait, when the last launch of
// this one is complete.  (Rows are zeroed at the start: any entry names an atom.)
constexpr int kNblAhead = 2;
// A pairs launch that has found the rebuild flag: its last block clears it.
__device__ __forceinline__ void done_reading_flag(const NbListArgs &a) {
    if (last_block(a.count + 1) && threadIdx.x == 0) *a.flag = 0;
}

template <bool ALL, int BLOCKS>
__global__ void __launch_bounds__(kNblThreads, BLOCKS) nbl_pairs_kernel(NbListArgs a, BondedArgs b, int n_bonded) {
    if ((int)blockIdx.x < n_bonded) {  // bonded terms of the same step, a thread each
        pdl_wait();
        pdl_trigger();
        bonded_term(b, (long long)blockIdx.x * kNblThreads + threadIdx.x, FixAdd{b.facc, b.status});
        if (__ldcg(a.flag) != 0) done_reading_flag(a);
        return;
    }
    const int i = (int)(((blockIdx.x - n_bonded) * blockDim.x + threadIdx.x) / 32);
    const int lane = threadIdx.x & 31;
    const bool mine = i < a.n_atoms;  // warp-uniform
    const int terms = ALL ? 7 : a.terms;
    const float epf = 1.0f - 1.0f / kEp;
    const float kfar = -2.0f * epf / 3.0f;
    const int *row = a.rows + (long long)i * a.row_cap;
    const float2 *ljab = nullptr;
    float L = 0.f, h = 0.f;
    int n = 0;
    struct Entry {
        int e;
        float rm;
        float2 ab;
    };
    auto entry = [&](int k) {  // the row's entry k and its partner's parameters
        Entry q;
        q.e = __ldcg(row + k);  // through L2: another SM may have rebuilt the row
        const int2 ty = a.atype[q.e & INT_MAX];
        q.rm = __ldg(a.rmax + ty.y);
        q.ab = __ldg(ljab + ty.x);
        return q;
    };
    Entry ahead[kNblAhead] = {};
    if (mine) {
        const WinDev &W = a.win[a.atom_win[i]];
        L = W.box;
        h = W.hbox;
        ljab = a.ljab + a.atype[i].x * a.n_lj_types;
        n = min(__ldcg(a.row_n + i), a.row_cap);
#pragma unroll
        for (int u = 0; u < kNblAhead; ++u) ahead[u] = entry(min(lane + 32 * u, a.row_cap - 1));
    }
    pdl_wait();
    pdl_trigger();
    const bool rebuild = __ldcg(a.flag) != 0;  // the same for the whole launch
    long long fx = 0, fy = 0, fz = 0;
    if (mine) {
        const float4 xi = a.pos[i];
        auto pair = [&](const Entry &q, float4 xj) {
            const float rx = mimg(xi.x - xj.x, L, h);
            const float ry = mimg(xi.y - xj.y, L, h);
            const float rz = mimg(xi.z - xj.z, L, h);
            const float d2 = dist2f(rx, ry, rz);
            if (!(d2 < a.cut2)) return;
            const float ri = rsqrtf(d2);
            const float ri2 = ri * ri;
            const float qq = xi.w * xj.w;
            float fs = 0.0f;
            if (terms & 4) {
                const float two = 2.0f * q.rm;
                const float r2 = q.rm * q.rm;
                fs = d2 > __fmul_rn(two, two) ? kfar * qq * ri2 * ri
                                              : -qq * (epf / (24.0f * r2 * r2)) * (8.0f * q.rm - 3.0f * d2 * ri);
            }
            if (q.e >= 0) {
                if (terms & 1) {
                    const float r6 = ri2 * ri2 * ri2;
                    fs += r6 * fmaf(12.0f * q.ab.x, r6, -6.0f * q.ab.y) * ri2;
                }
                if (terms & 2) fs += qq * ri2 * ri;
            }
            const float px = fs * rx, py = fs * ry, pz = fs * rz;
            check_force(a.status, px, py, pz);
            fx += to_fix(px);
            fy += to_fix(py);
            fz += to_fix(pz);
        };
        int k = lane;
        if (rebuild) {
            n = min(nbl_build_row(a, i, lane, xi), a.row_cap);
            __syncwarp();
        } else {
            float4 xj[kNblAhead];
#pragma unroll
            for (int u = 0; u < kNblAhead; ++u) xj[u] = a.pos[ahead[u].e & INT_MAX];
#pragma unroll
            for (int u = 0; u < kNblAhead; ++u, k += 32)
                if (k < n) pair(ahead[u], xj[u]);
        }
        for (; k < n; k += 32) {
            const Entry q = entry(k);
            pair(q, a.pos[q.e & INT_MAX]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(kFull, fx, o);
        fy += __shfl_xor_sync(kFull, fy, o);
        fz += __shfl_xor_sync(kFull, fz, o);
    }
    if (lane < 3 && mine) {
        const long long v = lane == 0 ? fx : (lane == 1 ? fy : fz);
        if (v) atomicAdd(a.facc + 3 * (long long)i + lane, (unsigned long long)v);
    }
    if (rebuild) done_reading_flag(a);
}

unsigned check_blocks(int n) { return (unsigned)((n + kNblCheckThreads - 1) / kNblCheckThreads); }
unsigned warp_blocks(int n) { return (unsigned)(((long long)n * 32 + kNblThreads - 1) / kNblThreads); }

}  // namespace

// Above this the pairs pass is bound by its gathers in flight and takes 40
// registers (six blocks an SM); below, by the length of a warp's chain, with 64
// (us per solvent-free step, 40 / 64 registers: 8800 atoms 19.6 / 18.1, 22 000
// 29.6 / 29.9, 66 000 67.5 / 71.6, 264 000 255 / 293).
constexpr int kNblDenseAtoms = 16000;

bool nblist_block_cells(int n_cells) { return n_cells <= kNblBlockCells; }

void launch_nblist_check(const NbListArgs &a, cudaStream_t s) {
    if (a.n_atoms <= 0) return;
    const unsigned blocks = check_blocks(a.n_atoms);
    launch_chain_smem(nbl_check_kernel, blocks, kNblCheckThreads, a.block_cells ? sizeof(int) * a.n_cells : 0, s, a);
    if (a.block_cells) return;
    nbl_bin_kernel<<<blocks, kNblCheckThreads, 0, s>>>(a);
    nbl_scan_kernel<<<1, 1024, 0, s>>>(a);
    nbl_scatter_kernel<<<blocks, kNblCheckThreads, 0, s>>>(a);
}

void launch_nblist_count(const NbListArgs &a, cudaStream_t s) {
    if (a.n_atoms <= 0) return;
    launch_nblist_check(a, s);
    nbl_count_kernel<<<warp_blocks(a.n_atoms), kNblThreads, 0, s>>>(a);
}

void launch_nblist_pairs(const NbListArgs &a, cudaStream_t s, const BondedArgs &b) {
    if (a.n_atoms <= 0) return;
    const int nb = bonded_blocks(b, kNblThreads);
    const unsigned blocks = nb + warp_blocks(a.n_atoms);
    if (a.n_atoms > kNblDenseAtoms) {
        if (a.terms == 7) launch_chain(nbl_pairs_kernel<true, 6>, blocks, kNblThreads, s, a, b, nb);
        else launch_chain(nbl_pairs_kernel<false, 6>, blocks, kNblThreads, s, a, b, nb);
    } else {
        if (a.terms == 7) launch_chain(nbl_pairs_kernel<true, 4>, blocks, kNblThreads, s, a, b, nb);
        else launch_chain(nbl_pairs_kernel<false, 4>, blocks, kNblThreads, s, a, b, nb);
    }
}

void launch_nblist_leapfrog(const LeapfrogArgs &f, const NbListArgs &a, cudaStream_t s) {
    if (f.n_atoms > 0)
        launch_chain_smem(nbl_leapfrog_kernel, check_blocks(f.n_atoms), kNblCheckThreads, sizeof(int) * a.n_cells, s, f, a);
}

}  // namespace isspa
