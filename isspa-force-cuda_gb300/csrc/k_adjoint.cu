// k_adjoint.cu -- reverse-mode gradient of the mean COM-axis force.
//
// For one frame, J = sum_i c_i . F_i with c_i = +n/2 on restraint group 0 and
// -n/2 on group 1 (n: unit COM separation).  Writing the IS-SPA force of point
// p on atom i as F_ip = s_p G_ip + H_ip (s_p = w_p/n_p; G the multipole and
// tabulated-LJ parts per unit density, H the constant-density dielectric part,
// reference src/isspa_force_cuda.cu:274-312):
//   lambda_p   = dJ/ds_p = sum_i c_i . G_ip                       (points kernel)
//   dJ/dT_f[k] = sum c_i . (-vtot_i s_p r/d) x lerp weight of entry k (points kernel)
//   dJ/dT_g[k] = sum_p lambda_p/n_p dw_p/dT_g[k], w_p = prod_j g_j  (density kernel)
//   dJ/dA, dJ/dB of the nonbond LJ (nonbond_force_cuda.cu:131-132) and of the
//   scaled 1-4 LJ (dih_force_cuda.cu:70-74), which are linear in A and B.
// MC points are the field pass's (regenerated from the Philox counters of the
// frame's step); gradients accumulate in FP64 per window.
//
// GB300's FP64 pipe takes a warp instruction every 16 cycles per SM (an FP32
// one: a quarter of a cycle), whether one lane or 32 are active, so the points
// and density kernels work in double-float on the FP32 pipe and leave FP64 to
// the sums.  16 windows x 550 atoms, nMC 50, per launch: points 6.76 ms in FP64,
// 0.30 in double-float; density 12.0 ms, 2.4 with the double-float body, 0.91
// once the warp reconverges after each lane's own atoms, 0.81 with one FP32 test
// per atom and point, 0.82 with the product's exponent; pairs 0.88 ms with a thread
// per atom, 0.07 with a warp.
// The error against 64-bit references is the FP32 fields' and coordinates'
// either way (6e-6 of dJ/dT_g at those sizes, before and after).
#include <algorithm>
#include <cuda_runtime.h>

#include "dfloat.cuh"
#include "kernels.h"

namespace isspa {
namespace {

constexpr int kAdjThreads = 128;
constexpr int kAdjStage = 1024;  // most atoms staged at a time (32 groups of 32)

__device__ __forceinline__ DF df_const(double c) { return DF{(float)c, (float)(c - (double)(float)c)}; }  // folded

// <P1>, <P2>, <P3> of a Langevin dipole in a field x.  Below 5 the backward
// continued fraction r_l = x / (2l+1 + x r_(l+1)) is carried as numerators and
// denominators, A_l = x B_(l+1), B_l = (2l+1) B_(l+1) + x A_(l+1) (all terms
// positive), so that <P_m> = r_1 ... r_m = x^m B_(m+1) / B_1 takes one division
// instead of one per level; 18 levels leave 1e-19 at x = 5.  Above, the closed
// forms with coth x = (1 + q) / (1 - q), q = exp(-2x).
__device__ __forceinline__ void langevin_df(DF x, DF &p1, DF &p2, DF &p3) {
    if (x.hi < 5.0f) {
        DF A{0.f, 0.f}, B{1.f, 0.f}, b2 = B, b3 = B, b4 = B;
#pragma unroll 3
        for (int l = 18; l >= 1; --l) {
            const DF nb = df_add(df_mulf(B, (float)(2 * l + 1)), df_mul(x, A));
            A = df_mul(x, B);
            B = nb;
            if (l == 4) b4 = B;
            if (l == 3) b3 = B;
            if (l == 2) b2 = B;
        }
        p1 = df_div(A, B);  // A_1 = x B_2
        const DF x2 = df_mul(x, x);
        p2 = df_div(df_mul(x2, b3), B);
        p3 = df_div(df_mul(df_mul(x2, x), b4), B);
    } else {
        const DF q = df_from(exp(-2.0 * df_double(x)));
        const DF c = df_div(df_addf(q, 1.0f), df_addf(df_neg(q), 1.0f));
        const DF ix = df_div(DF{1.f, 0.f}, x), ix2 = df_mul(ix, ix), cx = df_mul(c, ix);
        p1 = df_add(c, df_neg(ix));
        p2 = df_addf(df_mulf(df_add(ix2, df_neg(cx)), 3.0f), 1.0f);
        p3 = df_add(df_add(c, df_mulf(df_mul(ix2, df_add(c, df_neg(ix))), 15.0f)), df_mulf(ix, -6.0f));
    }
}

// hi + lo in FP64 with one FP64 instruction: a float widens to a double with
// integer operations (exponent rebiased by 896, mantissa moved up by 29 bits;
// zeros and infinities / NaN keep their exponents).
__device__ __forceinline__ double widen(float v) {
    const unsigned u = __float_as_uint(v), m = u & 0x7fffffffu;
    unsigned e = (m >> 3) + 0x38000000u;
    e = m >= 0x7f800000u ? (m >> 3) | 0x7ff00000u : e;
    e = m < 0x00800000u ? 0u : e;
    return __hiloint2double((int)((u & 0x80000000u) | e), (int)(m < 0x00800000u ? 0u : u << 29));
}
__device__ __forceinline__ double df_sum(DF a) { return widen(a.hi) + widen(a.lo); }

// A block's window and point; a lane past the window's points repeats the tile's
// first (valid false).
__device__ __forceinline__ void adj_tile(const AdjointArgs &a, int &w, long long &p, bool &valid) {
    const int2 tile = a.tiles[blockIdx.x];
    w = tile.x;
    const WinDev W = a.win[w];
    valid = (long long)tile.y + threadIdx.x < (long long)W.n_atoms * a.n_mc;
    p = W.point_off + tile.y + (valid ? threadIdx.x : 0);
}

// One weighted atom, staged for a block of points: weights c_i = s_i n with n
// the window's COM axis.
struct AdjAtom {
    float4 x;
    float cs_hi, cs_lo;  // -vtot s_i
    float rm2;
    int frow;
};

// lambda_p and dJ/dT_f of one point per thread.  Per pair, with e the unit
// field, w = e.r, g = w / r^2 and the per-unit-density amplitudes a_l:
//   n . G = -q_i vtot r^-3 [ (n.r) 3 X / r^2 - (n.e) (Y + a1) ] - vtot (n.r) T_f / r,
//   X = g (w (2.5 a2 + 35/6 a3 g) - 2.5 a3) + a1 w - a2/2,
//   Y = (7.5 a3 g + 3 a2) g - 1.5 a3 / r^2
// (the multipole terms of src/isspa_force_cuda.cu:274-289 projected on n).
__global__ void __launch_bounds__(kAdjThreads) adjoint_points_kernel(AdjointArgs a) {
    __shared__ AdjAtom s_at[kAdjThreads];
    int w;
    long long p;
    bool valid;
    adj_tile(a, w, p, valid);
    const WinDev W = a.win[w];
    const float4 raw = a.raw_e[p], raw0 = a.raw_e0[p];
    const float4 P = a.q0[p];
    const DF sp = df_div(DF{raw.w, 0.f}, DF{(float)(int)raw0.w, 0.f});
    const DF e2 = df_norm2(raw.x, raw.y, raw.z);
    const DF im = e2.hi > 0.0f ? df_rsqrt(e2) : DF{0.f, 0.f};
    DF A1, a2, a3;
    langevin_df(df_mul(e2, im), A1, a2, a3);
    A1 = df_mulf(A1, kP0);
    a2 = df_mulf(a2, kQ0);
    a3 = df_mulf(a3, kO0);
    const DF ex = df_mulf(im, raw.x), ey = df_mulf(im, raw.y), ez = df_mulf(im, raw.z);
    const double *n3 = a.axis + 3 * w;
    const DF nx = df_from(n3[0]), ny = df_from(n3[1]), nz = df_from(n3[2]);
    const DF en = df_add(df_add(df_mul(ex, nx), df_mul(ey, ny)), df_mul(ez, nz));
    const DF c0 = df_mulf(a2, -0.5f), kx = df_mulf(a2, 2.5f), ky = df_mul(a3, df_const(35.0 / 6.0)),
             k25 = df_mulf(a3, -2.5f), y1 = df_mulf(a3, 7.5f), y0 = df_mulf(a2, 3.0f), u15 = df_mulf(a3, -1.5f);
    const DF f_inv = df_div(DF{1.f, 0.f}, DF{a.f_dr, 0.f});
    const float L = W.box, h = W.hbox;
    DF lam{0.f, 0.f};
    const int k1 = a.adj_off[w + 1];
    for (int k0 = a.adj_off[w]; k0 < k1; k0 += kAdjThreads) {
        const int kn = min(kAdjThreads, k1 - k0);
        __syncthreads();
        if (threadIdx.x < kn) {
            const int i = a.adj_atoms[k0 + threadIdx.x];
            const int it = a.atype[i].y;
            const float rm = __ldg(a.rmax + it);
            const DF cs = df_from(-(double)__ldg(a.vtot + it) * a.adj_s[k0 + threadIdx.x]);
            s_at[threadIdx.x] = AdjAtom{a.pos[i], cs.hi, cs.lo, __fmul_rn(rm, rm), it * a.n_f};
        }
        __syncthreads();
        for (int k = 0; k < kn; ++k) {
            const AdjAtom at = s_at[k];
            const float rx = mimg(P.x - at.x.x, L, h), ry = mimg(P.y - at.x.y, L, h), rz = mimg(P.z - at.x.z, L, h);
            const DF d2 = df_norm2(rx, ry, rz);
            const DF ri = df_rsqrt(d2), ri2 = df_mul(ri, ri), ri3 = df_mul(ri2, ri);
            const DF er = df_add(df_add(df_mulf(ex, rx), df_mulf(ey, ry)), df_mulf(ez, rz));
            const DF nr = df_add(df_add(df_mulf(nx, rx), df_mulf(ny, ry)), df_mulf(nz, rz));
            const DF g = df_mul(er, ri2);
            const DF X = df_add(df_fma(g, df_fma(er, df_fma(ky, g, kx), k25), c0), df_mul(A1, er));
            const DF Z = df_mulf(df_mul(ri2, X), 3.0f);
            const DF Y = df_add(df_add(df_mul(df_fma(y1, g, y0), g), df_mul(u15, ri2)), A1);
            DF G = df_mulf(df_mul(ri3, df_add(df_mul(nr, Z), df_neg(df_mul(en, Y)))), at.x.w);
            const DF cs{at.cs_hi, at.cs_lo};
            const float d2f = dist2f(rx, ry, rz);
            if (valid && d2f <= at.rm2) {
                const int bin = (int)__fmaf_rn(__fsub_rn(__fsqrt_rn(d2f), a.f_r0), a.f_inv, 0.5f);
                if (bin >= 0 && bin < a.n_f) {
                    const DF fr = df_table_frac(df_mul(d2, ri), a.f_r0, f_inv, bin);
                    const long long fi = at.frow + bin;
                    const float2 tv = __ldg(a.ftab + fi);
                    const DF tab = df_lerp(tv.x, tv.y, fr);
                    const DF cr = df_mul(nr, ri);
                    G = df_fma(cr, tab, G);
                    const DF c = df_mul(df_mul(cr, cs), sp), cf = df_mul(c, fr);
                    double *df = a.dJ_df + (long long)w * a.n_ftab;
                    atomicAdd(df + fi, df_sum(df_add(c, df_neg(cf))));
                    if (fi + 1 < a.n_ftab) atomicAdd(df + fi + 1, df_sum(cf));
                }
            }
            lam = df_fma(G, cs, lam);
        }
    }
    if (valid) a.lam[p] = df_double(lam);
}

// The density product is held as prod 2^prod_e with prod within 2^+-32, so that
// neither it nor its low word is lost where FP64 would hold them; a factor v0 + f (v1
// - v0) that leads out of that range is taken from FP64 as m 2^e (tables have zeros in
// the core, seldom values that small: a factor 0 is the common case here).
constexpr float kRange = 4294967296.0f;  // 2^32
__device__ __forceinline__ bool in_range(float v) { return fabsf(v) >= 1.0f / kRange && fabsf(v) <= kRange; }
__device__ __forceinline__ DF density_factor(float v0, float v1, DF f, int &e) {
    if (v0 == 0.0f && v1 == 0.0f) return DF{0.0f, 0.0f};
    const double fd = df_double(f);
    return df_from(frexp((double)v0 * (1.0 - fd) + (double)v1 * fd, &e));
}

// dJ/dT_g of one point per thread, in two sweeps over the point's in-range
// atoms: the density product, then every factor's share lambda/n * prod / g.
// The window's atoms are tested once in FP32 (once per sweep for windows beyond
// one stage), 32 to a mask in shared memory, and each lane then walks its own
// masks: the lanes' in-range atoms differ (a quarter of the atoms are inside
// rmax of some lane of the warp at 550 atoms, 6 % of one lane's), so the
// double-float work runs as often as the busiest lane has atoms instead of once
// per atom that any lane has.  Strided groups spread a chain's atoms over masks.
__global__ void __launch_bounds__(kAdjThreads, 10) adjoint_density_kernel(AdjointArgs a) {
    extern __shared__ float4 s_x[];  // [stage] atoms, then [stage / 32][kAdjThreads] masks
    const int stage = a.stage;
    auto s_mask = reinterpret_cast<unsigned(*)[kAdjThreads]>(s_x + stage);
    int w;
    long long p;
    bool valid;
    adj_tile(a, w, p, valid);
    const WinDev W = a.win[w];
    const double lam = a.lam[p];
    const float4 P = a.q0[p];
    const int n = (int)a.raw_e0[p].w;
    const DF dJdw = df_div(df_from(lam), DF{(float)n, 0.f});
    const int owner = W.atom_off + (int)((p - W.point_off) / a.n_mc);
    const float rm = __ldg(a.rmax + a.atype[owner].y);
    // a lane with nothing to add takes no atom as in range
    const float rm2 = valid && lam != 0.0 ? __fmul_rn(rm, rm) : -1.0f;
    const float L = W.box, h = W.hbox;
    const DF g_inv = df_div(DF{1.f, 0.f}, DF{a.g_dr, 0.f});
    int zeros = 0;
    bool forced = false;
    DF prod{1.0f, 0.0f};  // of the nonzero factors, times 2^prod_e
    int prod_e = 0;
    double *dg = a.dJ_dg + (long long)w * a.n_gtab;
    const int N = W.n_atoms, t = threadIdx.x;
    for (int pass = 0; pass < 2; ++pass) {
        for (int j0 = 0; j0 < N; j0 += stage) {
            const int jn = min(stage, N - j0);
            const int nq = (jn + 31) >> 5;  // groups: atoms q, q + nq, q + 2 nq, ...
            if (pass == 0 || N > stage) {
                __syncthreads();
                for (int i = t; i < jn; i += kAdjThreads) {
                    float4 x = a.pos[W.atom_off + j0 + i];
                    x.w = __int_as_float(a.atype[W.atom_off + j0 + i].y * a.n_g);
                    s_x[i] = x;
                }
                __syncthreads();
                for (int q = 0; q < nq; ++q) {
                    unsigned mask = 0u, bit = 1u;
#pragma unroll 4
                    for (int k = q; k < jn; k += nq, bit <<= 1) {
                        const float4 xj = s_x[k];
                        const float d2 = dist2f(mimg(P.x - xj.x, L, h), mimg(P.y - xj.y, L, h), mimg(P.z - xj.z, L, h));
                        if (d2 <= rm2) mask |= bit;
                    }
                    s_mask[q][t] = mask;  // read back by this thread only
                }
            }
            int q = 0;
            unsigned mask = s_mask[0][t];
            for (;;) {
                while (mask == 0u && ++q < nq) mask = s_mask[q][t];
                if (mask == 0u) break;
                const int k = q + (__ffs(mask) - 1) * nq;
                mask &= mask - 1;
                const float4 xj = s_x[k];
                const float rx = mimg(P.x - xj.x, L, h), ry = mimg(P.y - xj.y, L, h), rz = mimg(P.z - xj.z, L, h);
                const int bin = (int)__fmul_rn(__fsub_rn(__fsqrt_rn(dist2f(rx, ry, rz)), a.g_r0), a.g_inv);
                forced |= bin < 0;
                if (bin >= 0 && bin < a.n_g - 1) {
                    const DF fr = df_table_frac(df_root(df_norm2(rx, ry, rz)), a.g_r0, g_inv, bin);
                    const int gi = __float_as_int(xj.w) + bin;
                    const bool next = gi + 1 < a.n_gtab;
                    const float g0 = __ldg(a.g_table + gi), g1 = next ? __ldg(a.g_table + gi + 1) : 0.0f;
                    DF g = df_lerp(g0, g1, fr);
                    int ge = 0;
                    if (pass == 0) {
                        const DF p = df_mul(prod, g);
                        if (in_range(p.hi)) {
                            prod = p;
                        } else if ((g = density_factor(g0, g1, fr, ge)).hi == 0.0f) {
                            ++zeros;
                        } else {
                            prod = df_mul(prod, g);
                            const int up = fabsf(prod.hi) < 1.0f / kRange ? 32 : 0;
                            prod = df_scale(prod, up ? kRange : 1.0f);
                            prod_e += ge - up;
                        }
                    } else if (!forced) {
                        // of zero factors only a single one's own share survives
                        if (!in_range(g.hi)) g = density_factor(g0, g1, fr, ge);
                        if (zeros > 1 || (zeros == 1 && g.hi != 0.0f)) continue;
                        const DF d = df_mul(dJdw, zeros ? prod : df_div(prod, g));
                        const int de = zeros ? prod_e : prod_e - ge;
                        if (de != 0) {
                            const double v = scalbn(df_double(d), de), vf = v * df_double(fr);
                            atomicAdd(dg + gi, v - vf);
                            if (next) atomicAdd(dg + gi + 1, vf);
                        } else if (d.hi != 0.0f) {
                            const DF df = df_mul(d, fr);
                            atomicAdd(dg + gi, df_sum(df_add(d, df_neg(df))));
                            if (next) atomicAdd(dg + gi + 1, df_sum(df));
                        }
                    }
                }
            }
            __syncwarp();  // the lanes leave the loop above at different times
        }
        // the second sweep has nothing to do for a lane whose every share is zero
        if (forced || zeros >= 2)
            for (int q = 0; N <= stage && q < (N + 31) >> 5; ++q) s_mask[q][t] = 0u;
        __syncwarp();
    }
}

// Nonbond LJ coefficient adjoint of every weighted atom (one warp each) against
// all atoms of its window; exclusions as the nonbond kernel.
__global__ void __launch_bounds__(kAdjThreads) adjoint_pairs_kernel(AdjointArgs a) {
    const int k = (blockIdx.x * kAdjThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= a.n_adj) return;  // warp-uniform
    const int i = a.adj_atoms[k];
    const int w = a.atom_win[i];
    const WinDev W = a.win[w];
    const double c0 = a.cvec[3 * i], c1 = a.cvec[3 * i + 1], c2 = a.cvec[3 * i + 2];
    const float4 xi = a.pos[i];
    const int ti = a.atype[i].x;
    const float L = W.box, h = W.hbox;
    const int e0 = a.excl_start[i], e1 = a.excl_start[i + 1];
    double *dA = a.dJ_dA + (long long)w * a.n_ljtab, *dB = a.dJ_dB + (long long)w * a.n_ljtab;
    for (int j = W.atom_off + lane; j < W.atom_off + W.n_atoms; j += 32) {
        if (j == i) continue;
        int lo = e0, hi = e1;  // j in the sorted exclusion list?
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (a.excl[mid] < j) lo = mid + 1;
            else hi = mid;
        }
        if (lo < e1 && a.excl[lo] == j) continue;
        const float4 xj = a.pos[j];
        const double rx = mimg(xi.x - xj.x, L, h), ry = mimg(xi.y - xj.y, L, h), rz = mimg(xi.z - xj.z, L, h);
        const double r2 = 1.0 / (rx * rx + ry * ry + rz * rz);
        const double r8 = (r2 * r2) * (r2 * r2);
        const double cr = (c0 * rx + c1 * ry + c2 * rz) * r8;
        const int kk = a.nbp[ti * a.n_lj_types + a.atype[j].x];
        atomicAdd(dA + kk, 12.0 * cr * (r2 * r2 * r2));
        atomicAdd(dB + kk, -6.0 * cr);
    }
}

// Scaled 1-4 LJ coefficient adjoint (force +f r14 on atom x, -f r14 on atom w).
__global__ void adjoint_14_kernel(AdjointArgs a) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= a.n_dihs) return;
    const int raw = a.dih_type[d];
    if (!(raw & 0x40000000)) return;
    const int4 at = a.dihs[d];
    const double dc0 = a.cvec[3 * at.x] - a.cvec[3 * at.w], dc1 = a.cvec[3 * at.x + 1] - a.cvec[3 * at.w + 1],
                 dc2 = a.cvec[3 * at.x + 2] - a.cvec[3 * at.w + 2];
    if (dc0 == 0.0 && dc1 == 0.0 && dc2 == 0.0) return;
    const int w = a.atom_win[at.x];
    const WinDev W = a.win[w];
    const float4 px = a.pos[at.x], pw = a.pos[at.w];
    const double rx = mimg(px.x - pw.x, W.box, W.hbox), ry = mimg(px.y - pw.y, W.box, W.hbox),
                 rz = mimg(px.z - pw.z, W.box, W.hbox);
    const double rm = rx * rx + ry * ry + rz * rz;
    const double r6 = 1.0 / (rm * rm * rm);
    const double scnb = a.sc14[raw & 0x3FFFFFFF].y;
    const double cr = dc0 * rx + dc1 * ry + dc2 * rz;
    const int kk = a.nbp[a.atype[at.x].x * a.n_lj_types + a.atype[at.w].x];
    atomicAdd(a.dJ_dA + (long long)w * a.n_ljtab + kk, cr * 12.0 * r6 * r6 / (scnb * rm));
    atomicAdd(a.dJ_dB + (long long)w * a.n_ljtab + kk, cr * -6.0 * r6 / (scnb * rm));
}

}  // namespace

void launch_adjoint(const AdjointArgs &a, cudaStream_t s) {
    if (a.n_tiles > 0) {
        const unsigned blocks = (unsigned)a.n_tiles;
        adjoint_points_kernel<<<blocks, kAdjThreads, 0, s>>>(a);
        const size_t smem = (size_t)a.stage * sizeof(float4) + (size_t)(a.stage / 32) * kAdjThreads * sizeof(unsigned);
        adjoint_density_kernel<<<blocks, kAdjThreads, smem, s>>>(a);
    }
    if (a.n_adj > 0) adjoint_pairs_kernel<<<(a.n_adj + 3) / 4, kAdjThreads, 0, s>>>(a);
    if (a.n_dihs > 0) adjoint_14_kernel<<<(a.n_dihs + 127) / 128, 128, 0, s>>>(a);
}

int adjoint_point_tile() { return kAdjThreads; }
int adjoint_stage(int max_atoms) { return std::min(kAdjStage, (max_atoms + 31) / 32 * 32); }

}  // namespace isspa
