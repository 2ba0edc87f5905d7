// kernels.cu -- hand-written sm_103a kernels of the KoMD hot path.
//
// Per step (komd_gpu_step): integrate0 -> com/wrap/bin -> scan -> scatter ->
// cell sort+gather -> pair (LJ, FENE, ATM neighbour list) -> [bonded] ->
// [limit] -> [ATM triplets] -> integrate1.  On the Verlet path with FP32
// forces the drift is one kernel (k_step0_fused), the container kernels run
// only on a rebuild, the LJ pass sweeps the triplets itself (k_lj_atm,
// pair_tile.cu) and integrate1 rides on the ATM flush.
//
// Citations are to Snapex2409/KoMD, src/.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "engine.cuh"
#include "kernels.cuh"
#include "atm_device.cuh"

namespace komd {

// double -> float rounded to nearest (ties to even) from the bits, in integer
// instructions (GB300 converts FP64 -> FP32 on its narrow FP64 pipe): the 29
// dropped mantissa bits decide the rounding, and a carry out of the mantissa
// moves into the exponent as IEEE rounding does.  Results outside the FP32
// normal range (zero, subnormal, overflow, NaN) take the conversion
// instruction.  Bitwise equal to __double2float_rn.
__device__ __forceinline__ float d2f_rn(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ffu) - 1023 + 127;   // the FP32 biased exponent
    if (e < 1 || e > 254) return __double2float_rn(x);
    const unsigned long long mant = b & 0xfffffffffffffULL;
    unsigned f = ((unsigned)e << 23) | (unsigned)(mant >> 29);
    const unsigned rest = (unsigned)(mant & 0x1fffffffULL);
    f += (rest > 0x10000000u || (rest == 0x10000000u && (f & 1u))) ? 1u : 0u;
    return __uint_as_float(f | ((unsigned)(b >> 32) & 0x80000000u));
}

// float -> double (exact) from the bits, likewise
__device__ __forceinline__ double f2d(float x) {
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    if (m - 0x00800000u >= 0x7f000000u) return (double)x;   // zero, subnormal, infinity, NaN
    return __longlong_as_double((long long)(((unsigned long long)(b & 0x80000000u) << 32) +
                                            ((unsigned long long)m << 29) + (896ULL << 52)));
}

// an infinity or a NaN, from the exponent bits (a comparison would run on the FP64 pipe)
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

// ===========================================================================
// container: COM, periodic wrap, binning (LinkedCells.cpp:65-121,390-400;
// MoleculeContainer.cpp:55-75).  One thread per molecule.
// ===========================================================================
// (int64)(x / cs) clamped to [0, nd - 1] (writeIndices).  The truncated quotient
// is read off x * (1 / cs) where that is not within 1e-9 of an integer (its
// error is below 4e-10 for quotients up to 1e6); the IEEE division, which costs the
// narrow FP64 pipe several times as much, runs for the rest.
__device__ __forceinline__ int cell_index(double x, double cs, double ics, int nd) {
    const double t = dmul(x, ics);
    const int q0 = __double2int_rz(t);
    const long long fr = __double_as_longlong(dsub(t, (double)q0));   // ordered as the value where positive
    long long q;
    if (q0 >= 0 && q0 < 1000000 && fr > __double_as_longlong(1e-9) && fr < __double_as_longlong(1.0 - 1e-9)) q = q0;
    else q = __double2ll_rz(ddiv(x, cs));
    if (q < 0) q = 0;
    if (q > nd - 1) q = nd - 1;
    return (int)q;
}

// On a step without a rebuild a molecule matters only if it wraps.  True when its
// centre of mass is inside the domain by more than the error of this FP32 estimate:
// with k sites of positive mass the rounded inputs, the products, the k - 1 additions
// and those of the total mass are each within 2^-24 (the division 2^-22) of
// sum |m r| / sum m.  The range of tm keeps underflow of the products far below that.
// 18 FP64 operations and three divisions of a three-site molecule need not run:
// 300,000 sites, 17.0 -> 7.0 us a step.
__device__ __forceinline__ bool com_inside(const BinArgs &a, int s0, int s1) {
    float c[3] = {0.f, 0.f, 0.f}, ca[3] = {0.f, 0.f, 0.f}, tm = 0.f;
    bool in = true;
    for (int s = s0; s < s1; s++) {
        const float ms = d2f_rn(a.m[s]);
        in = in && ms > 0.f;
        for (int d = 0; d < 3; d++) {
            const float x = d2f_rn(a.r[3 * s + d]) * ms;
            c[d] += x;
            ca[d] += fabsf(x);
        }
        tm += ms;
    }
    in = in && tm > 1e-20f && tm < 1e20f;
    const float im = __fdividef(1.0f, tm), k = 6.0e-8f * (float)(2 * (s1 - s0) + 16);
    for (int d = 0; d < 3; d++) {
        const float x = c[d] * im, tol = fmaf(ca[d] * im, k, 1e-20f);
        in = in && x - tol > a.in_lo[d] && x + tol < a.in_hi[d];
    }
    return in;   // false for NaN
}

__device__ __forceinline__ void com_wrap_bin_body(const BinArgs &a, int bid, int nblk) {
    const Grid &g = a.g;
    const int n_mol = a.n_mol;
    const int *__restrict__ mol_off = a.mol_off;
    double *__restrict__ r = a.r;
    const double *__restrict__ m = a.m;
    double *__restrict__ com = a.com;
    int *__restrict__ mol_cell = a.mol_cell, *__restrict__ mol_rank = a.mol_rank;
    int *__restrict__ cell_count = a.cell_count, *__restrict__ cell_mcount = a.cell_mcount;
    double *__restrict__ bias = a.bias;
    const int *__restrict__ rebuild = a.rebuild;
    const unsigned char *__restrict__ exact_com = a.exact_com;
    if (a.wrapped && rebuild && !*rebuild) return;   // k_step0_fused wrapped this step; no rebuild
    const bool bin = !(rebuild && !*rebuild);        // no rebuild in this step: cells stay as built
    for (int k = bid * blockDim.x + threadIdx.x; k < n_mol; k += nblk * blockDim.x) {
    const int s0 = a.single ? k : mol_off[k], s1 = a.single ? k + 1 : mol_off[k + 1];
    if (!bin && com_inside(a, s0, s1)) continue;   // no wrap; the centre is formed again before anything reads it
    // com += r * m ; M += m ; com /= M   (updateCOM, no FMA).  For a single
    // site of power-of-two mass the scaling is exact and the result is r
    // itself (up to the sign of a zero), so the FP64 division is skipped.
    double c[3] = {0.0, 0.0, 0.0}, tm = 0.0;
    if (s1 - s0 == 1 && exact_com && exact_com[k]) {
        tm = m[s0];
        for (int d = 0; d < 3; d++) c[d] = r[3 * s0 + d];
    } else {
        for (int s = s0; s < s1; s++) {
            const double ms = m[s];
            for (int d = 0; d < 3; d++) c[d] = dadd(c[d], dmul(r[3 * s + d], ms));
            tm = dadd(tm, ms);
        }
        for (int d = 0; d < 3; d++) c[d] = ddiv(c[d], tm);
    }
    // Periodic_Kernel: strict comparisons against the domain bounds
    double off[3];
    bool moved = false;
    for (int d = 0; d < 3; d++) {
        off[d] = 0.0;
        if (c[d] < g.low[d]) off[d] = g.L[d];
        if (c[d] > g.high[d]) off[d] = -g.L[d];
        moved |= (off[d] != 0.0);
    }
    if (moved) {
        double c2[3] = {0.0, 0.0, 0.0};
        for (int s = s0; s < s1; s++) {
            const double ms = m[s];
            for (int d = 0; d < 3; d++) {
                const double x = dadd(r[3 * s + d], off[d]);
                r[3 * s + d] = x;
                c2[d] = dadd(c2[d], dmul(x, ms));
            }
            if (bias)   // the cell-local position r - bias is unchanged by the wrap
                for (int d = 0; d < 3; d++)
                    if (off[d] != 0.0) bias[3 * s + d] = dadd(bias[3 * s + d], off[d]);
        }
        if (s1 - s0 == 1 && exact_com && exact_com[k]) {
            for (int d = 0; d < 3; d++) c[d] = r[3 * s0 + d];
        } else {
            for (int d = 0; d < 3; d++) c[d] = ddiv(c2[d], tm);
        }
    }
    for (int d = 0; d < 3; d++) com[3 * k + d] = c[d];
    if (!bin) continue;
    // writeIndices: (int64)((com - low) / cs) clamped to [0, nd-1]
    int b[3];
    for (int d = 0; d < 3; d++) b[d] = cell_index(dsub(c[d], g.low[d]), g.cs, g.ics, g.nd[d]);
    const int cell = b[0] + g.nd[0] * (b[1] + g.nd[1] * b[2]);
    mol_cell[k] = cell;
    mol_rank[k] = atomicAdd(&cell_mcount[cell], 1);
    if (!a.single) atomicAdd(&cell_count[cell], s1 - s0);   // else the scan takes the molecules' counts
    }
}
__global__ void k_com_wrap_bin(BinArgs a) {
    pdl_trigger();
    pdl_wait();
    com_wrap_bin_body(a, blockIdx.x, gridDim.x);
}

// exclusive scans of the cells' site and molecule counts (length nc; one block
// of 1024 threads over tiles of 4096 cells, four consecutive cells a thread);
// the counts are zeroed once read, ready for the next binning.  Without site
// counts (q.a null: one site per molecule) both scans are the molecules'.
// work: the Verlet list build's unit counter, reset here for this rebuild.
__device__ __forceinline__ void scan2_body(const ScanArgs &q) {
    __shared__ int2 s_w[2][32];
    const int nc = q.nc;
    int *__restrict__ a = q.a, *__restrict__ sa = q.sa, *__restrict__ b = q.b, *__restrict__ sb = q.sb;
    if (q.rebuild && !*q.rebuild) return;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (q.work && t == 0) *q.work = 0;
    int ca = 0, cb = 0;   // sums of the tiles before
    for (int base = 0, turn = 0; base < nc; base += 4096, turn ^= 1) {
        const int i = base + 4 * t;
        int va[4] = {0, 0, 0, 0}, vb[4] = {0, 0, 0, 0};
        const bool whole = i + 4 <= nc;
        if (whole) {
            const int4 y = *reinterpret_cast<const int4 *>(b + i);
            vb[0] = y.x; vb[1] = y.y; vb[2] = y.z; vb[3] = y.w;
            *reinterpret_cast<int4 *>(b + i) = make_int4(0, 0, 0, 0);
            if (a) {
                const int4 x = *reinterpret_cast<const int4 *>(a + i);
                va[0] = x.x; va[1] = x.y; va[2] = x.z; va[3] = x.w;
                *reinterpret_cast<int4 *>(a + i) = make_int4(0, 0, 0, 0);
            }
        } else {
            for (int k = 0; k < 4 && i + k < nc; k++) {
                vb[k] = b[i + k];
                b[i + k] = 0;
                if (a) {
                    va[k] = a[i + k];
                    a[i + k] = 0;
                }
            }
        }
        const int ta = va[0] + va[1] + va[2] + va[3], tb = vb[0] + vb[1] + vb[2] + vb[3];
        int xa = ta, xb = tb;   // inclusive warp scan
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(0xffffffffu, xa, o), yb = __shfl_up_sync(0xffffffffu, xb, o);
            if (lane >= o) { xa += ya; xb += yb; }
        }
        if (lane == 31) s_w[turn][w] = make_int2(xa, xb);
        __syncthreads();
        const int2 mine = s_w[turn][lane];   // every warp scans the 32 warp sums itself
        int wa = mine.x, wb = mine.y;
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(0xffffffffu, wa, o), yb = __shfl_up_sync(0xffffffffu, wb, o);
            if (lane >= o) { wa += ya; wb += yb; }
        }
        const int suma = __shfl_sync(0xffffffffu, wa, 31), sumb = __shfl_sync(0xffffffffu, wb, 31);
        int pa = ca + __shfl_sync(0xffffffffu, wa - mine.x, w) + xa - ta;
        int pb = cb + __shfl_sync(0xffffffffu, wb - mine.y, w) + xb - tb;
        int ea[4], eb[4];
        for (int k = 0; k < 4; k++) {
            ea[k] = pa; pa += va[k];
            eb[k] = pb; pb += vb[k];
        }
        if (whole) {
            const int4 y = make_int4(eb[0], eb[1], eb[2], eb[3]);
            *reinterpret_cast<int4 *>(sb + i) = y;
            *reinterpret_cast<int4 *>(sa + i) = a ? make_int4(ea[0], ea[1], ea[2], ea[3]) : y;
        } else {
            for (int k = 0; k < 4 && i + k < nc; k++) {
                sb[i + k] = eb[k];
                sa[i + k] = a ? ea[k] : eb[k];
            }
        }
        ca += suma;
        cb += sumb;
    }
    if (t == 0) { sa[nc] = a ? ca : cb; sb[nc] = cb; }
}
__global__ void __launch_bounds__(1024) k_scan2(ScanArgs q) {
    pdl_trigger();
    pdl_wait();
    scan2_body(q);
}

__device__ __forceinline__ void scatter_mol_body(const ScatterArgs &a, int bid, int nblk) {
    if (a.rebuild && !*a.rebuild) return;
    for (int k = bid * blockDim.x + threadIdx.x; k < a.n_mol; k += nblk * blockDim.x)
        a.cell_mols[a.cell_mstart[a.mol_cell[k]] + a.mol_rank[k]] = k;
}
__global__ void k_scatter_mol(ScatterArgs a) {
    pdl_trigger();
    pdl_wait();
    scatter_mol_body(a, blockIdx.x, gridDim.x);
}

// One warp per domain cell: order the cell's molecules by index (ascending
// site index, the reference's cell-list order), assign slots and gather the
// cell-ordered arrays.  A lane holds a molecule, and its place is the summed
// size of the cell's molecules with a lower index, counted over warp shuffles.
__device__ __forceinline__ void cell_sort_body(const SortArgs &a, int bid, int nblk) {
    const Grid &g = a.g;
    const int *__restrict__ mol_off = a.mol_off, *__restrict__ cell_mstart = a.cell_mstart;
    const int *__restrict__ cell_start = a.cell_start, *__restrict__ cell_mols = a.cell_mols;
    const double *__restrict__ r = a.r;
    const float2 *__restrict__ site_lj = a.site_lj;
    const int *__restrict__ key = a.key;
    int *__restrict__ slot_site = a.slot_site, *__restrict__ site_slot = a.site_slot;
    float4 *__restrict__ pos4 = a.pos4;
    int *__restrict__ skey = a.skey;
    float *__restrict__ seps = a.seps;
    double *__restrict__ posd = a.posd, *__restrict__ seps_d = a.seps_d, *__restrict__ sig_d = a.sig_d;
    double *__restrict__ bias = a.bias;
    float4 *__restrict__ ref4 = a.ref4;
    int *__restrict__ slot_cell = a.slot_cell, *__restrict__ zkey = a.zkey;
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    if (a.rebuild && !*a.rebuild) return;
    for (int cell = bid * warps + (threadIdx.x >> 5); cell < g.ncell; cell += nblk * warps) {
        const int ms = cell_mstart[cell], mc = cell_mstart[cell + 1] - ms;
        const int ss = cell_start[cell];
        int cx, cy, cz;
        cell_coords(g, cell, cx, cy, cz);
        const double cen[3] = {cell_centre(g, 0, cx), cell_centre(g, 1, cy), cell_centre(g, 2, cz)};
        for (int base = 0; base < mc; base += 32) {
            const int t = base + lane;
            const int mine = (t < mc) ? cell_mols[ms + t] : INT_MAX;
            int s0 = mine, size = 1;
            if (!a.single && t < mc) {
                s0 = mol_off[mine];
                size = mol_off[mine + 1] - s0;
            }
            int off = 0;
            for (int cb = 0; cb < mc; cb += 32) {
                int other = mine, osize = size;
                if (cb != base) {
                    const int u = cb + lane;
                    other = u < mc ? cell_mols[ms + u] : INT_MAX;
                    osize = !a.single && u < mc ? mol_off[other + 1] - mol_off[other] : 1;
                }
                const int nu = min(32, mc - cb);
                if (a.single) {
                    for (int u = 0; u < nu; u++) off += __shfl_sync(0xffffffffu, other, u) < mine ? 1 : 0;
                } else {
                    for (int u = 0; u < nu; u++) {
                        const int o = __shfl_sync(0xffffffffu, other, u), z = __shfl_sync(0xffffffffu, osize, u);
                        off += o < mine ? z : 0;
                    }
                }
            }
            if (t < mc) {
                for (int s = s0; s < s0 + size; s++) {
                    const int slot = ss + off + (s - s0);
                    slot_site[slot] = s;
                    site_slot[s] = slot;
                    const double x = r[3 * s], y = r[3 * s + 1], z = r[3 * s + 2];
                    const float2 lj = site_lj[s];   // sqrt(eps), sigma/2
                    const float4 p4 = make_float4(__double2float_rn(x - cen[0]), __double2float_rn(y - cen[1]),
                                                  __double2float_rn(z - cen[2]), lj.y);
                    pos4[slot] = p4;
                    skey[slot] = key[s];
                    seps[slot] = lj.x;
                    if (bias) {
                        bias[3 * s] = cen[0]; bias[3 * s + 1] = cen[1]; bias[3 * s + 2] = cen[2];
                        ref4[s] = p4;
                        slot_cell[slot] = cell;
                        // the half-list order key: z quantized over the box (see vl_above)
                        long long q = (long long)floor((z - g.low[2]) / g.L[2] * (double)kZq);
                        zkey[slot] = (int)(q < 0 ? 0 : (q >= kZq ? kZq - 1 : q));
                    }
                    if (posd) {
                        posd[3 * slot] = x; posd[3 * slot + 1] = y; posd[3 * slot + 2] = z;
                        seps_d[slot] = a.eps[s];
                        sig_d[slot] = a.sig[s];
                    }
                }
            }
        }
    }
}
__global__ void __launch_bounds__(kBlock) k_cell_sort(SortArgs a) {
    pdl_trigger();
    pdl_wait();
    cell_sort_body(a, blockIdx.x, gridDim.x);
}

// ===========================================================================
// ATM triplets in FP64 (ATM.cpp:22-62 / ATM_NOLIST.cpp:124-159): one warp per
// site i, every pair (a, b) of i's neighbours inside cutoff_3b with
// |r_a - r_b| inside too.  Force on i only (each triplet is visited from all
// three vertices, no atomics: the sums are reproducible).  With A=|r_ia|^2,
// B=|r_ib|^2, C=|r_ab|^2:
//   V = nu [ (ABC)^-3/2 + 3/8 P (ABC)^-5/2 ],  P = (A+B-C)(A-B+C)(-A+B+C)
//   dV/dA = nu (ABC)^-5/2 [ -3/2 BC + 3/8 dP/dA - 15/16 P/A ]
//   F_i(physical) = -2 (dV/dA e_a + dV/dB e_b),  e_a = r_i - r_a
// which equals the reference's comp_force terms (comp_force = 2 dV/dA).
//
// GB300's FP64 pipe (about 1/64 of the FP32 rate) bounds this kernel, so only
// the triplets reach it: the lanes test the candidate pairs in FP32 with a
// 1e-4 margin over the cutoff (the vectors' rounding is below 1e-6 of it),
// queue the hits by ballot and evaluate 32 queued pairs at a time, with the
// exact FP64 test of C.  A, 1/A and 1/sqrt(A) are staged once per neighbour.
// 32,000 sites of liquid argon: 1688 -> 418 us a launch (every candidate tested
// and both roots taken in FP64 before), sensors' form 3051 -> 928 us.
// ===========================================================================
struct AtmStageD { double x, y, z, A, iA, wA; };   // r_i - r_a, |.|^2, its reciprocal and reciprocal root

template <bool MEASURE, bool COMPAT>
__global__ void __launch_bounds__(kBlock) k_atm_d(AtmParams p) {
    extern __shared__ float4 s_dyn[];
    __shared__ int s_q[kWarpsPerBlock][64];
    __shared__ double s_part[kWarpsPerBlock][8];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int cap = p.nl_cap;
    float4 *sf = s_dyn + wib * cap;   // FP32 vector and code (the candidate test)
    AtmStageD *sd = reinterpret_cast<AtmStageD *>(s_dyn + warps * cap) + wib * cap;
    const AtmEntryD *nl = reinterpret_cast<const AtmEntryD *>(p.nl);
    const double rc2 = p.rc2;
    const float pre2 = (float)(p.rc2 * (1.0 + 1e-4));
    double a_e = 0.0, a_w[6] = {0, 0, 0, 0, 0, 0};
    int a_t = 0;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    for (int i = blockIdx.x * warps + wib; i < p.n; i += gridDim.x * warps) {
        const int ni = p.nl_count[i];
        for (int k = lane; k < ni; k += 32) {
            const AtmEntryD e = nl[(size_t)i * cap + k];
            const double A = e.x * e.x + e.y * e.y + e.z * e.z;
            sf[k] = make_float4((float)e.x, (float)e.y, (float)e.z, __int_as_float((int)e.code));
            sd[k] = AtmStageD{e.x, e.y, e.z, A, __drcp_rn(A), rsqrt(A)};
        }
        __syncwarp();
        double gx = 0.0, gy = 0.0, gz = 0.0;
        auto triplet = [&](int q, bool valid) {
            if (!valid) return;
            const AtmStageD ea = sd[q & 0xffff], eb = sd[q >> 16];
            const double cx = eb.x - ea.x, cy = eb.y - ea.y, cz = eb.z - ea.z;
            const double C = cx * cx + cy * cy + cz * cz;
            if (dabove(C, rc2)) return;
            const double A = ea.A, B = eb.A;
            const double wc = rsqrt(C);
            const double sv = ea.wA * eb.wA * wc;       // 1/(abc)
            const double s2 = sv * sv;
            const double s5 = s2 * s2 * sv;
            const double S = A + B + C;
            const double t1 = fma(-2.0, C, S), t2 = fma(-2.0, B, S), t3 = fma(-2.0, A, S);
            const double u = t2 * t3, v = t1 * t3, w = t1 * t2;
            const double P = t1 * u;
            const double K = u + v + w, nP = -2.5 * P;
            // 8/3 dV/dA: u + v - w - 4 B C - 5/2 P / A  (B: v and A C; C: u and A B)
            const double vA = s5 * fma(nP, ea.iA, fma(-2.0, w, fma(-4.0 * B, C, K)));
            const double vB = s5 * fma(nP, eb.iA, fma(-2.0, v, fma(-4.0 * A, C, K)));
            gx = fma(vA, ea.x, fma(vB, eb.x, gx));
            gy = fma(vA, ea.y, fma(vB, eb.y, gy));
            gz = fma(vA, ea.z, fma(vB, eb.z, gz));
            if (MEASURE) {
                const double vC = s5 * fma(nP, wc * wc, fma(-2.0, u, fma(-4.0 * A, B, K)));
                a_e += s2 * sv * fma(0.375 * P, s2, 1.0);   // a third of it per visit, applied at the end
                a_t++;
                double wt = 1.0 / 3.0;
                if (p.virial_compat) {
                    const int ca = __float_as_int(sf[q & 0xffff].w), cb = __float_as_int(sf[q >> 16].w);
                    const int k = 1 + ((ca & 32) ? 0 : 1) + ((cb & 32) ? 0 : 1);
                    wt = p.atm_direct ? 0.0 : 1.0 / (double)k;
                }
                // pair-decomposed virial sum_pairs P_ab d (x) d with P_ab = -2 dV/d(r_ab^2)
                const double sc = -0.75 * wt;
                const double pa = sc * vA, pb = sc * vB, pc = sc * vC;
                a_w[0] += pa * ea.x * ea.x + pb * eb.x * eb.x + pc * cx * cx;
                a_w[1] += pa * ea.x * ea.y + pb * eb.x * eb.y + pc * cx * cy;
                a_w[2] += pa * ea.y * ea.y + pb * eb.y * eb.y + pc * cy * cy;
                a_w[3] += pa * ea.x * ea.z + pb * eb.x * eb.z + pc * cx * cz;
                a_w[4] += pa * ea.y * ea.z + pb * eb.y * eb.z + pc * cy * cz;
                if (!p.virial_compat) a_w[5] += pa * ea.z * ea.z + pb * eb.z * eb.z + pc * cz * cz;
            }
        };
        int qn = 0;
        const int half = ni / 2;
        for (int a0 = 0; a0 < ni; a0 += 32) {   // round robin (a, a + d mod n): every pair once
            const int a = a0 + lane;
            const bool av = a < ni;
            float4 ea = make_float4(0.f, 0.f, 0.f, 0.f);
            if (av) ea = sf[a];
            for (int d = 1; d <= half; d++) {
                bool hit = false;
                int b = 0;
                if (av && !(2 * d == ni && a >= d)) {
                    b = a + d;
                    if (b >= ni) b -= ni;
                    const float4 eb = sf[b];
                    const float cx = eb.x - ea.x, cy = eb.y - ea.y, cz = eb.z - ea.z;
                    hit = !(cx * cx + cy * cy + cz * cz > pre2);
                    if (COMPAT) {
                        const int nba = __float_as_int(ea.w) & 31, nbb = __float_as_int(eb.w) & 31;
                        hit = hit && ((nba == 13 && nbb == 13) || (nba != 13 && nbb != 13 && nba != nbb));
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) s_q[wib][qn + __popc(m & lt)] = a | (b << 16);
                qn += __popc(m);
                if (qn >= 32) {
                    __syncwarp();
                    const int q = s_q[wib][lane], tail = s_q[wib][32 + lane];
                    __syncwarp();
                    qn -= 32;
                    if (lane < qn) s_q[wib][lane] = tail;
                    __syncwarp();
                    triplet(q, true);
                }
            }
        }
        __syncwarp();
        if (qn > 0) triplet(lane < qn ? s_q[wib][lane] : 0, lane < qn);
        const double gs = warp_sum3(gx, gy, gz, lane);
        if ((lane & 7) == 0 && lane < 24) {
            // reference sign: +2 nu (vA e_a + vB e_b); physical: the negative
            const double sc = 0.75 * p.sign * p.nu;
            p.f[3 * (size_t)p.slot_site[i] + (lane >> 3)] += sc * gs;
        }
        __syncwarp();   // the staging is refilled by the next vertex
    }
    if (MEASURE) {
        double vals[8] = {a_e * (1.0 / 3.0), 0.0, a_w[0], a_w[1], a_w[2], a_w[3], a_w[4], a_w[5]};
        for (int k = 0; k < 8; k++) {
            double x = vals[k];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            vals[k] = x;
        }
        const int visits = __reduce_add_sync(0xffffffffu, a_t);
        if (lane == 0) {
            for (int k = 0; k < 8; k++) s_part[wib][k] = vals[k];
            s_part[wib][1] = (double)visits / 3.0;
        }
        __syncthreads();
        if (threadIdx.x < R_NSLOTS) {
            const int t = threadIdx.x;
            double sum = 0.0;
            int src = -1;
            if (t == R_UATM) src = 0;
            else if (t == R_TRIPS) src = 1;
            else if (t >= R_W0 && t <= R_W5) src = 2 + (t - R_W0);
            if (src >= 0)
                for (int w = 0; w < warps; w++) sum += s_part[w][src];
            // nu scaling of energy and virial
            if (t == R_UATM || (t >= R_W0 && t <= R_W5)) sum *= p.nu;
            p.partials[(size_t)blockIdx.x * R_NSLOTS + t] = sum;
        }
    }
}

// the warp sums of K values (2 or 8), the lanes splitting the values on the way:
// lane l ends with value l / (32 / K); 9 additions a lane for eight values
// instead of 40 (GB300's FP64 pipe bounds these reductions)
template <typename T, int K>
__device__ __forceinline__ T warp_sum_split(T (&v)[K], int lane) {
    int o = 16;
#pragma unroll
    for (int k = K; k > 1; k >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < k / 2; q++) {
            const T send = up ? v[q] : v[q + k / 2], keep = up ? v[q + k / 2] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// FP32 ATM kernel with ballot compaction: lanes test candidate pairs (a, b)
// of the vertex's neighbour list (round-robin pairing a, a+d mod n, so each
// unordered pair is tested once) and queue the ones inside the cutoff; the
// triplet arithmetic then always runs on 32 queued pairs at a time.  All
// queued pairs share vertex i, so each lane keeps a private force sum.
// Bound by instruction issue, half of it the tests: they run without branches,
// the partner stepped by one, the neighbour cells that COMPAT admits in a bit mask
// (32,000 sites of liquid argon 40 -> 33 us).
//
// MEASURE runs a resident grid whose warps stride over the vertices: a vertex's
// energy and virial leave the lanes' FP32 partials through a tree that leaves
// value k in lane 4 k, so that one conversion and one FP64 addition per vertex
// carry all seven into the warp's sums (a tree, conversions and a division per
// vertex kept the FP64 pipe 76 % busy: 525 -> 380 us at 256,000 sites).
template <bool MEASURE, bool COMPAT>
__global__ void __launch_bounds__(kBlock) k_atm_q(AtmParams p) {
    pdl_wait();
    extern __shared__ float4 s_dyn[];
    __shared__ unsigned s_q[kWarpsPerBlock][64];
    __shared__ float s_qc[kWarpsPerBlock][64];
    __shared__ double s_part[kWarpsPerBlock][8];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cap = p.nl_cap;
    float4 *se = s_dyn + wib * cap;
    float4 *sq = s_dyn + kWarpsPerBlock * cap + wib * cap;   // (A, 1/A, 1/sqrt(A), -) per entry
    const float rc2 = p.rc2f;
    double m_sum = 0.0;   // lane 4 k (k < 8): the warp's sum of value k
    int m_t = 0;          // triplet visits (each triplet is visited from its three vertices)
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));

    for (int i = blockIdx.x * kWarpsPerBlock + wib; i < p.n; i += gridDim.x * kWarpsPerBlock) {
    float gx = 0.f, gy = 0.f, gz = 0.f;
    float m_e = 0.f, m_w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto triplet = [&](unsigned e, float C, bool valid) {
        if (!valid) return;
        const int a = (int)(e & 0xffffu), b = (int)(e >> 16);
        const float4 ea = se[a], eb = se[b];
        const float4 qa = sq[a], qb = sq[b];
        const float A = qa.x, B = qb.x;
        const float wc = rsqrt_ftz(C);
        const float sv = qa.z * qb.z * wc;                  // 1/(abc)
        const float s2 = sv * sv;
        const float s5 = s2 * s2 * sv;
        const float t1 = A + B - C, t2 = A - B + C, t3 = B + C - A;
        const float u = t2 * t3, v = t1 * t3, w = t1 * t2;
        const float P = t1 * u;
        float vA = s5 * (-1.5f * B * C + 0.375f * (u + v - w) - 0.9375f * P * qa.y);
        float vB = s5 * (-1.5f * A * C + 0.375f * (u - v + w) - 0.9375f * P * qb.y);
        float vC = s5 * (-1.5f * A * B + 0.375f * (-u + v + w) - 0.9375f * P * (wc * wc));
        float Vn = s2 * sv * (1.0f + 0.375f * P * s2);   // V / nu
        if (p.sw) {   // switched cutoff: V Sa Sb Sc and its derivatives in A, B, C
            float Sa, dSa, Sb, dSb, Sc, dSc;
            sw_eval(A, p.sw_rc2, p.sw_iw, Sa, dSa);
            sw_eval(B, p.sw_rc2, p.sw_iw, Sb, dSb);
            sw_eval(C, p.sw_rc2, p.sw_iw, Sc, dSc);
            const float sbc = Sb * Sc, sac = Sa * Sc, sab = Sa * Sb;
            vA = sbc * (vA * Sa + Vn * dSa);
            vB = sac * (vB * Sb + Vn * dSb);
            vC = sab * (vC * Sc + Vn * dSc);
            Vn = Vn * Sa * sbc;
        }
        gx += vA * ea.x + vB * eb.x;
        gy += vA * ea.y + vB * eb.y;
        gz += vA * ea.z + vB * eb.z;
        if (MEASURE) {
            m_e += Vn * (1.0f / 3.0f);
            m_t++;
            float wt;
            if (p.virial_compat) {
                const int ca = __float_as_int(ea.w), cb = __float_as_int(eb.w);
                const int k = 1 + ((ca & 32) ? 0 : 1) + ((cb & 32) ? 0 : 1);
                wt = p.atm_direct ? 0.0f : 1.0f / (float)k;
            } else {
                wt = 1.0f / 3.0f;
            }
            const float pa = -2.0f * vA * wt, pb = -2.0f * vB * wt, pc = -2.0f * vC * wt;
            const float cx = eb.x - ea.x, cy = eb.y - ea.y, cz = eb.z - ea.z;
            m_w[0] += pa * ea.x * ea.x + pb * eb.x * eb.x + pc * cx * cx;
            m_w[1] += pa * ea.x * ea.y + pb * eb.x * eb.y + pc * cx * cy;
            m_w[2] += pa * ea.y * ea.y + pb * eb.y * eb.y + pc * cy * cy;
            m_w[3] += pa * ea.x * ea.z + pb * eb.x * eb.z + pc * cx * cz;
            m_w[4] += pa * ea.y * ea.z + pb * eb.y * eb.z + pc * cy * cz;
            if (!p.virial_compat) m_w[5] += pa * ea.z * ea.z + pb * eb.z * eb.z + pc * cz * cz;
        }
    };

    {
        const int ni = p.nl_count[i];
        for (int k = lane; k < ni; k += 32) {
            const float4 e = p.nl[(size_t)i * cap + k];
            const float A = e.x * e.x + e.y * e.y + e.z * e.z;
            se[k] = e;
            sq[k] = make_float4(A, 1.0f / A, rsqrt_ftz(A), 0.f);
        }
        __syncwarp();
        int qn = 0;
        const int half = ni / 2;
        for (int a0 = 0; a0 < ni; a0 += 32) {
            const int a = a0 + lane;
            const bool av = a < ni;
            const float4 ea = se[av ? a : 0];
            // COMPAT: the neighbour cells (13: the home cell) that may pair with a's
            const int nba = __float_as_int(ea.w) & 31;
            const unsigned may = !COMPAT ? 0xffffffffu : nba == 13 ? 1u << 13 : ~(1u << 13 | 1u << nba);
            const int rounds = !av ? 0 : (2 * half == ni && a >= half) ? half - 1 : half;   // that pair is a - d's
            int b = av ? a : 0;
            for (int d = 1; d <= half; d++) {
                b = b + 1 == ni ? 0 : b + 1;
                const float4 eb = se[b];
                const float cx = eb.x - ea.x, cy = eb.y - ea.y, cz = eb.z - ea.z;
                const float C = cx * cx + cy * cy + cz * cz;
                const bool hit = d <= rounds && C <= rc2 && (!COMPAT || (may >> (__float_as_int(eb.w) & 31)) & 1u);
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int pos = qn + __popc(m & lt);
                    s_q[wib][pos] = (unsigned)a | ((unsigned)b << 16);
                    s_qc[wib][pos] = C;
                }
                qn += __popc(m);
                if (qn >= 32) {
                    __syncwarp();
                    const unsigned e = s_q[wib][lane];
                    const float ce = s_qc[wib][lane];
                    const bool mv = lane < qn - 32;
                    const unsigned te = mv ? s_q[wib][lane + 32] : 0u;
                    const float tc = mv ? s_qc[wib][lane + 32] : 0.f;
                    __syncwarp();
                    if (mv) { s_q[wib][lane] = te; s_qc[wib][lane] = tc; }
                    __syncwarp();
                    qn -= 32;
                    triplet(e, ce, true);
                }
            }
        }
        __syncwarp();
        if (qn > 0) {
            const bool v = lane < qn;
            const unsigned e = v ? s_q[wib][lane] : 0u;
            const float ce = v ? s_qc[wib][lane] : 1.f;
            triplet(e, ce, v);
        }
        // lanes 0, 8 and 16 take a component each: one conversion and one fused
        // operation on the FP64 pipe for the three
        const float gs = warp_sum3(gx, gy, gz, lane);
        const int site = p.slot_site[i];
        if ((lane & 7) == 0 && lane < 24)   // reference: +2 nu (...); physical: -2 nu (...)
            p.f[3 * (size_t)site + (lane >> 3)] += p.share * (double)gs;
        if (MEASURE) {
            float vals[8] = {m_e, 0.f, m_w[0], m_w[1], m_w[2], m_w[3], m_w[4], m_w[5]};
            const double v = (double)warp_sum_split<float, 8>(vals, lane);
            m_sum += v;
            if (p.e_site && lane == 0) p.e_site[site] = p.nu * v;
        }
        __syncwarp();   // the staging is refilled by the next vertex
    }
    }
    if (MEASURE) {
        const int visits = __reduce_add_sync(0xffffffffu, m_t);   // a third of a triplet per visit
        if ((lane & 3) == 0) s_part[wib][lane >> 2] = lane == 4 ? (double)visits / 3.0 : m_sum;
        __syncthreads();
        if (threadIdx.x < R_NSLOTS) {
            const int t = threadIdx.x;
            double sum = 0.0;
            int src = -1;
            if (t == R_UATM) src = 0;
            else if (t == R_TRIPS) src = 1;
            else if (t >= R_W0 && t <= R_W5) src = 2 + (t - R_W0);
            if (src >= 0)
                for (int w = 0; w < kWarpsPerBlock; w++) sum += s_part[w][src];
            if (t == R_UATM || (t >= R_W0 && t <= R_W5)) sum *= p.nu;
            p.partials[(size_t)blockIdx.x * R_NSLOTS + t] = sum;
        }
    }
}

// ===========================================================================
// bonded terms (no reference counterpart): harmonic bond and angle, FP32
// arithmetic on FP64 differences, FP64 atomic accumulation into f.
// ===========================================================================
__global__ void k_bonds(int nb, const int *__restrict__ bonds, const double *__restrict__ r, double *f, float kb,
                        float r0, double *partials, int measure) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0, w[6] = {0, 0, 0, 0, 0, 0};
    if (t < nb) {
        const int i = bonds[2 * t], j = bonds[2 * t + 1];
        const float dx = (float)(r[3 * i] - r[3 * j]), dy = (float)(r[3 * i + 1] - r[3 * j + 1]),
                    dz = (float)(r[3 * i + 2] - r[3 * j + 2]);
        const float rr = sqrtf(dx * dx + dy * dy + dz * dz);
        const float dl = rr - r0;
        const float fs = -kb * dl / rr;
        atomicAdd(&f[3 * i], (double)(fs * dx)); atomicAdd(&f[3 * i + 1], (double)(fs * dy));
        atomicAdd(&f[3 * i + 2], (double)(fs * dz));
        atomicAdd(&f[3 * j], (double)(-fs * dx)); atomicAdd(&f[3 * j + 1], (double)(-fs * dy));
        atomicAdd(&f[3 * j + 2], (double)(-fs * dz));
        if (measure) {
            e = 0.5 * (double)kb * (double)dl * (double)dl;
            w[0] = fs * dx * dx; w[1] = fs * dx * dy; w[2] = fs * dy * dy;
            w[3] = fs * dx * dz; w[4] = fs * dy * dz; w[5] = fs * dz * dz;
        }
    }
    if (measure) {
        const int lane = threadIdx.x & 31;
        double vals[8] = {e, w[0], w[1], w[2], w[3], w[4], w[5], 0.0};
        const double x = warp_sum_split<double, 8>(vals, lane);   // value k in lane 4 k
        const int k = lane >> 2;
        if ((lane & 3) == 0 && k < 7) atomicAdd(&partials[k == 0 ? R_UBOND : R_W0 + k - 1], x);
    }
}

__global__ void k_angles(int na, const int *__restrict__ angles, const double *__restrict__ r, double *f, float ka,
                         float th0, double *partials, int measure) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0, w[6] = {0, 0, 0, 0, 0, 0};
    if (t < na) {
        const int i = angles[3 * t], j = angles[3 * t + 1], k = angles[3 * t + 2];
        float u[3], v[3];
        for (int d = 0; d < 3; d++) {
            u[d] = (float)(r[3 * i + d] - r[3 * j + d]);
            v[d] = (float)(r[3 * k + d] - r[3 * j + d]);
        }
        const float uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        const float vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        const float uv = u[0] * v[0] + u[1] * v[1] + u[2] * v[2];
        const float inu = rsqrtf(uu), inv_ = rsqrtf(vv);
        float cs = uv * inu * inv_;
        cs = fminf(1.0f, fmaxf(-1.0f, cs));
        const float th = acosf(cs);
        const float dth = th - th0;
        const float sn = fmaxf(sqrtf(1.0f - cs * cs), 1e-6f);
        const float pre = ka * dth / sn;
        float fi[3], fk[3];
        for (int d = 0; d < 3; d++) {
            fi[d] = pre * (v[d] * inu * inv_ - cs * u[d] * inu * inu);
            fk[d] = pre * (u[d] * inu * inv_ - cs * v[d] * inv_ * inv_);
            atomicAdd(&f[3 * i + d], (double)fi[d]);
            atomicAdd(&f[3 * k + d], (double)fk[d]);
            atomicAdd(&f[3 * j + d], -(double)(fi[d] + fk[d]));
        }
        if (measure) {
            e = 0.5 * (double)ka * (double)dth * (double)dth;
            w[0] = u[0] * fi[0] + v[0] * fk[0]; w[1] = u[0] * fi[1] + v[0] * fk[1];
            w[2] = u[1] * fi[1] + v[1] * fk[1]; w[3] = u[0] * fi[2] + v[0] * fk[2];
            w[4] = u[1] * fi[2] + v[1] * fk[2]; w[5] = u[2] * fi[2] + v[2] * fk[2];
        }
    }
    if (measure) {
        const int lane = threadIdx.x & 31;
        double vals[8] = {e, w[0], w[1], w[2], w[3], w[4], w[5], 0.0};
        const double x = warp_sum_split<double, 8>(vals, lane);   // value k in lane 4 k
        const int k = lane >> 2;
        if ((lane & 3) == 0 && k < 7) atomicAdd(&partials[k == 0 ? R_UBOND : R_W0 + k - 1], x);
    }
}

// The same forces without the sensors for small molecules: a thread evaluates every
// term of a connected component (BondBlock: up to kBondComps components whose sites
// lie in one range of kBondSites), so nothing is summed by atomics.  Positions and
// forces pass through shared memory: coalesced, and the terms' reads and sums stay on
// chip.  Bound by its FP64 instructions (33 for a three-site molecule; conversions are
// in integers).  300,000 sites of three-site molecules: k_bonds + k_angles 20.1 ->
// 16.8 us; a thread per site, which evaluates a term once from each of its sites,
// took 25.7.
__global__ void __launch_bounds__(kBondComps) k_bonded_mol(const int4 *__restrict__ blocks,
                                                           const int *__restrict__ comp_off,
                                                           const int4 *__restrict__ terms,
                                                           const double *__restrict__ r, double *__restrict__ f,
                                                           float kb, float r0, float ka, float th0) {
    pdl_wait();
    __shared__ double s_r[3 * kBondSites], s_f[3 * kBondSites];
    const int4 b = blocks[blockIdx.x];   // components [x, y), sites [z, w)
    const int n3 = 3 * (b.w - b.z), c = b.x + (int)threadIdx.x;
    const size_t base = 3 * (size_t)b.z;
    constexpr int kRows = 3 * kBondSites / kBondComps;
    double x[kRows], y[kRows];   // all loads in flight at once
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int t = threadIdx.x + k * kBondComps;
        x[k] = t < n3 ? r[base + t] : 0.0;
        y[k] = t < n3 ? f[base + t] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        s_r[threadIdx.x + k * kBondComps] = x[k];
        s_f[threadIdx.x + k * kBondComps] = y[k];
    }
    const int t0 = c < b.y ? comp_off[c] : 0, t1 = c < b.y ? comp_off[c + 1] : 0;
    __syncthreads();
    for (int t = t0; t < t1; t++) {
        const int4 q = terms[t];   // sites; z < 0: a bond
        const int i = 3 * (q.x - b.z), j = 3 * (q.y - b.z);
        float u[3];
        for (int d = 0; d < 3; d++) u[d] = d2f_rn(dsub(s_r[i + d], s_r[j + d]));
        const float uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        if (q.z < 0) {
            const float rr = sqrtf(uu);
            const float fs = -kb * (rr - r0) / rr;
            for (int d = 0; d < 3; d++) {
                const double g = f2d(fs * u[d]);
                s_f[i + d] = dadd(s_f[i + d], g);
                s_f[j + d] = dsub(s_f[j + d], g);
            }
            continue;
        }
        const int k = 3 * (q.z - b.z);
        float v[3];
        for (int d = 0; d < 3; d++) v[d] = d2f_rn(dsub(s_r[k + d], s_r[j + d]));
        const float vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        const float uv = u[0] * v[0] + u[1] * v[1] + u[2] * v[2];
        const float inu = rsqrtf(uu), inv_ = rsqrtf(vv);
        float cs = uv * inu * inv_;
        cs = fminf(1.0f, fmaxf(-1.0f, cs));
        const float dth = acosf(cs) - th0;
        const float sn = fmaxf(sqrtf(1.0f - cs * cs), 1e-6f);
        const float pre = ka * dth / sn;
        for (int d = 0; d < 3; d++) {
            const float fi = pre * (v[d] * inu * inv_ - cs * u[d] * inu * inu);
            const float fk = pre * (u[d] * inu * inv_ - cs * v[d] * inv_ * inv_);
            s_f[i + d] = dadd(s_f[i + d], f2d(fi));
            s_f[k + d] = dadd(s_f[k + d], f2d(fk));
            s_f[j + d] = dsub(s_f[j + d], f2d(fi + fk));
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n3; t += kBondComps) f[base + t] = s_f[t];
}

// Limit_Force (Limit.cpp:19-25): clamp with Kokkos::min / max semantics
__global__ void k_limit(int n, const double *__restrict__ eps, const double *__restrict__ sig, double limit,
                        double *__restrict__ f) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double fmax = limit * eps[s] / sig[s];
    for (int d = 0; d < 3; d++) {
        double x = f[3 * s + d];
        x = (fmax < x) ? fmax : x;
        x = (x < -fmax) ? -fmax : x;
        f[3 * s + d] = x;
    }
}

// ===========================================================================
// velocity Verlet (Integrator.cpp:28-37), FP64 without contraction
// ===========================================================================
// hdtm[s] = (dt * 0.5) / m[s], the reference's dtInv2m (Integrator.cpp:29), computed
// once at upload with the same IEEE division.  With a Verlet list (bias !=
// nullptr) the drift also writes the site's FP32 position in its build cell's
// frame, (float)(r - bias) -- a periodic wrap that follows moves both alike, and a
// rebuild rewrites it -- and flags a rebuild when that has moved more than skin/2
// since the build.
__device__ __forceinline__ void local_position(int s, const double (&x)[3], const double *__restrict__ bias,
                                               const float4 *__restrict__ ref4, const int *__restrict__ site_slot,
                                               float4 *__restrict__ pos4, float half_skin2, int *__restrict__ rebuild) {
    const int slot = site_slot[s];
    const float4 q = ref4[s];
    float4 p = pos4[slot];
    p.x = d2f_rn(dsub(x[0], bias[3 * s]));
    p.y = d2f_rn(dsub(x[1], bias[3 * s + 1]));
    p.z = d2f_rn(dsub(x[2], bias[3 * s + 2]));
    pos4[slot] = p;
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    if (dx * dx + dy * dy + dz * dz > half_skin2) *rebuild = 1;
}
__global__ void k_step0(int n, double *__restrict__ r, double *__restrict__ v, const double *__restrict__ f,
                        const double *__restrict__ hdtm, double dt,
                        const double *__restrict__ bias, const float4 *__restrict__ ref4,
                        const int *__restrict__ site_slot, float4 *__restrict__ pos4, float half_skin2,
                        int *__restrict__ rebuild) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double c = hdtm[s];
    double x[3];
    for (int d = 0; d < 3; d++) {
        const double vv = dadd(v[3 * s + d], dmul(f[3 * s + d], c));
        v[3 * s + d] = vv;
        x[d] = dadd(r[3 * s + d], dmul(vv, dt));
        r[3 * s + d] = x[d];
    }
    if (bias) local_position(s, x, bias, ref4, site_slot, pos4, half_skin2, rebuild);
}

// Verlet path with single-site molecules whose COM is exactly the position
// (power-of-two masses): integrate0, the skin test, the periodic wrap with
// its bias update (k_com_wrap_bin's operations) and the FP32 cell-local
// position in one pass over the sites.  The results are those of the separate
// kernels; on a rebuild step the cell sort rewrites pos4 afterwards.
__device__ __forceinline__ bool dkey_nan(double x) {
    return (__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

// Block-cooperative copies of a block's rows (3 doubles per site) between a
// caller's host buffer and shared memory in 16-byte pieces: over the host link
// whole contiguous lines move instead of 8-byte pieces strided by 24 bytes.
constexpr int kIoBlock = 256;   // sites per block of the kernels that do host I/O

__device__ __forceinline__ void rows_in(const double *src, double *dst_s, int base, int cnt) {
    const double *p = src + 3 * (size_t)base;
    const int m = 3 * cnt;
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        const double2 *p2 = reinterpret_cast<const double2 *>(p);
        for (int k = threadIdx.x; k < m / 2; k += blockDim.x) {
            const double2 q = p2[k];
            dst_s[2 * k] = q.x;
            dst_s[2 * k + 1] = q.y;
        }
        if ((m & 1) && threadIdx.x == 0) dst_s[m - 1] = p[m - 1];
    } else {
        for (int k = threadIdx.x; k < m; k += blockDim.x) dst_s[k] = p[k];
    }
}

__device__ __forceinline__ void rows_out(const double *src_s, double *dst, int base, int cnt) {
    double *p = dst + 3 * (size_t)base;
    const int m = 3 * cnt;
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        double2 *p2 = reinterpret_cast<double2 *>(p);
        for (int k = threadIdx.x; k < m / 2; k += blockDim.x) p2[k] = make_double2(src_s[2 * k], src_s[2 * k + 1]);
        if ((m & 1) && threadIdx.x == 0) p[m - 1] = src_s[m - 1];
    } else {
        for (int k = threadIdx.x; k < m; k += blockDim.x) p[k] = src_s[k];
    }
}

// the drift of site s past its new position x: periodic wrap with its bias
// update (b: the site's bias), the FP32 cell-local position and the skin test.
// The centres of mass are formed by the binning of a rebuild (k_com_wrap_bin),
// before anything reads them.
__device__ __forceinline__ void drift_finish(const Step0Args &a, int s, int slot, double (&x)[3], double (&b)[3]) {
    const Grid &g = a.g;
    // Periodic_Kernel on the COM (= the position): strict comparisons, made on
    // order-preserving integer keys (the FP64 pipe is the bottleneck here);
    // the cell-local position x - bias is unchanged by a wrap
    double off[3];
    bool moved = false;
    for (int d = 0; d < 3; d++) {
        off[d] = 0.0;
        const long long kx = dkey(x[d]);
        if (!dkey_nan(x[d])) {
            if (kx < dkey(g.low[d])) {
                off[d] = g.L[d];
                moved = true;
            }
            if (kx > dkey(g.high[d])) {
                off[d] = -g.L[d];
                moved = true;
            }
        }
    }
    if (moved) {   // r += shift over all three components, as Periodic_Kernel
        for (int d = 0; d < 3; d++) {
            x[d] = dadd(x[d], off[d]);
            b[d] = dadd(b[d], off[d]);
            a.bias[3 * s + d] = b[d];
        }
    }
    float4 p = a.pos4[slot];
    const float4 q = a.ref4[s];
    p.x = d2f_rn(dsub(x[0], b[0]));
    p.y = d2f_rn(dsub(x[1], b[1]));
    p.z = d2f_rn(dsub(x[2], b[2]));
    a.pos4[slot] = p;
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    if (dx * dx + dy * dy + dz * dz > a.half_skin2) *a.rebuild = 1;
    for (int d = 0; d < 3; d++) a.r[3 * s + d] = x[d];
}

// r_in / v_in: where this step's positions and velocities are read (the
// engine's own arrays, or a caller's host buffers reached over the host link);
// r_out: an extra host copy of the new positions (nullptr: none).  Launched
// with kIoBlock threads per block.
__device__ __forceinline__ void step0_fused_body(const Step0Args &a, int bid) {
    __shared__ double s_r[3 * kIoBlock], s_v[3 * kIoBlock];
    const int n = a.n;
    double *r = a.r, *v = a.v;
    const double *__restrict__ f = a.f, *__restrict__ hdtm = a.hdtm;
    const double dt = a.dt;
    const double *__restrict__ bias = a.bias;
    const int *__restrict__ site_slot = a.site_slot;
    const double *r_in = a.r_in, *v_in = a.v_in;
    double *r_out = a.r_out;
    const int t = threadIdx.x;
    const int base = bid * blockDim.x, s = base + t;
    const int cnt = min((int)blockDim.x, n - base);
    const bool host_in = r_in != r;   // uniform: the whole step reads the caller's buffers
    if (host_in) {
        rows_in(r_in, s_r, base, cnt);
        rows_in(v_in, s_v, base, cnt);
        __syncthreads();
    }
    if (s < n) {
        const double c = hdtm[s];
        double x[3], b[3], vi[3], ri[3];
        for (int d = 0; d < 3; d++) {
            vi[d] = host_in ? s_v[3 * t + d] : v[3 * s + d];
            ri[d] = host_in ? s_r[3 * t + d] : r[3 * s + d];
        }
        for (int d = 0; d < 3; d++) {
            const double vv = dadd(vi[d], dmul(f[3 * s + d], c));
            v[3 * s + d] = vv;
            x[d] = dadd(ri[d], dmul(vv, dt));
            b[d] = bias[3 * s + d];
        }
        drift_finish(a, s, site_slot[s], x, b);
        if (r_out)   // each thread overwrites only the entries it read
            for (int d = 0; d < 3; d++) s_r[3 * t + d] = x[d];
    }
    if (r_out) {
        __syncthreads();
        rows_out(s_r, r_out, base, cnt);
    }
}
__global__ void __launch_bounds__(kIoBlock) k_step0_fused(Step0Args a) {
    pdl_trigger();
    pdl_wait();
    step0_fused_body(a, blockIdx.x);
}

__global__ void k_step1(int n, double *__restrict__ v, const double *__restrict__ f, const double *__restrict__ hdtm,
                        int *__restrict__ err, int *__restrict__ rebuild) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (rebuild && s == 0) *rebuild = 0;   // every consumer of this step's flag has run
    if (s >= n) return;
    const double c = hdtm[s];
    bool bad = false;
    for (int d = 0; d < 3; d++) {
        const double vv = dadd(v[3 * s + d], dmul(f[3 * s + d], c));
        v[3 * s + d] = vv;
        bad |= not_finite(vv);
    }
    if (bad) atomicOr(&err[E_NONFINITE], 1);
}

// ===========================================================================
// sensors
// ===========================================================================
// TemperatureSensor::measure (sites inside [low, high]) + kinetic tensor
// (PressureSensor::MomentumKernel) over the first n_terms sites (TERMS).
// Grid-stride over the sites (a resident grid, so each thread sums several
// sites before the fixed-tree warp and block reductions).  The block that
// finishes last sums the blocks' rows in their order into acc and zeroes
// acc's other slots, so a measure needs neither a clearing nor a second
// kernel: the sums are deterministic.  done: a counter, zero between launches.
// STEP1: with integrate1 of the step before (k_step1's operations; a thermostatted step).
template <bool TERMS, bool STEP1>
__global__ void __launch_bounds__(kBlock) k_kinetic(Grid g, int n, int n_terms, const double *__restrict__ r,
                                                    double *__restrict__ v, const double *__restrict__ m,
                                                    double *partials, double *__restrict__ acc, unsigned *done,
                                                    const double *__restrict__ f, const double *__restrict__ hdtm,
                                                    int *__restrict__ err, int *__restrict__ rebuild) {
    pdl_wait();
    if (STEP1 && rebuild && blockIdx.x == 0 && threadIdx.x == 0) *rebuild = 0;   // its consumers have run
    __shared__ double s_part[kWarpsPerBlock][8];
    __shared__ bool s_last;
    constexpr int kVals = TERMS ? 8 : 2;
    double vals[kVals];
    for (int k = 0; k < kVals; k++) vals[k] = 0.0;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const double x = r[3 * s], y = r[3 * s + 1], z = r[3 * s + 2];
        double vx = v[3 * s], vy = v[3 * s + 1], vz = v[3 * s + 2];
        const double ms = m[s];
        if (STEP1) {
            const double c = hdtm[s];
            vx = dadd(vx, dmul(f[3 * s], c));
            vy = dadd(vy, dmul(f[3 * s + 1], c));
            vz = dadd(vz, dmul(f[3 * s + 2], c));
            v[3 * s] = vx;
            v[3 * s + 1] = vy;
            v[3 * s + 2] = vz;
            if (not_finite(vx) || not_finite(vy) || not_finite(vz)) atomicOr(&err[E_NONFINITE], 1);
        }
        if (x >= g.low[0] && y >= g.low[1] && z >= g.low[2] && x <= g.high[0] && y <= g.high[1] && z <= g.high[2]) {
            vals[0] = dadd(vals[0], dmul(ms, dadd(dadd(dmul(vx, vx), dmul(vy, vy)), dmul(vz, vz))));
            vals[1] = dadd(vals[1], 1.0);
        }
        if constexpr (TERMS) {
            if (s < n_terms) {
                vals[2] += vx * vx * ms; vals[3] += vx * vy * ms; vals[4] += vy * vy * ms;
                vals[5] += vx * vz * ms; vals[6] += vy * vz * ms; vals[7] += vz * vz * ms;
            }
        }
    }
    const int t = threadIdx.x, lane = t & 31, wib = t >> 5;
    const double mine = warp_sum_split<double, kVals>(vals, lane);
    if (lane % (32 / kVals) == 0) s_part[wib][lane / (32 / kVals)] = mine;
    __syncthreads();
    if (t < kVals) {   // this block's row: R_NSLOTS doubles apart, the values in front
        double sum = 0.0;
        for (int w = 0; w < kWarpsPerBlock; w++) sum += s_part[w][t];
        partials[(size_t)blockIdx.x * R_NSLOTS + t] = sum;
        __threadfence();
    }
    __syncthreads();
    if (t == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (wib < kVals) {   // a value per warp, the rows over the lanes
        double sum = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) sum += __ldcg(&partials[(size_t)b * R_NSLOTS + wib]);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) s_part[0][wib] = sum;
    }
    __syncthreads();
    if (t < R_NSLOTS) {
        int src = -1;
        if (t == R_MV2) src = 0;
        else if (t == R_NBOX) src = 1;
        else if (TERMS && t >= R_K0 && t <= R_K5) src = 2 + t - R_K0;
        acc[t] = src >= 0 ? s_part[0][src] : 0.0;
    }
    if (t == 0) *done = 0u;
}

// RDF over molecule COMs (RDFSensor::RDF_Kernel, RDFSensor.cpp:61-72):
// minimum image delta - L*round(delta/L), bin (uint64)(r/dr) clamped.
__device__ __forceinline__ void rdf_pair(const double *ca, const double *cb, Grid g, double max_r, double dr,
                                         long long nbins, double *bins) {
    double q[3];
    for (int d = 0; d < 3; d++) {
        const double delta = dsub(ca[d], cb[d]);
        q[d] = dsub(delta, dmul(g.L[d], (double)(long long)round(ddiv(delta, g.L[d]))));
    }
    const double rr = sqrt(dadd(dadd(dmul(q[0], q[0]), dmul(q[1], q[1])), dmul(q[2], q[2])));
    if (rr > max_r) return;
    unsigned long long b = (unsigned long long)ddiv(rr, dr);
    if (b > (unsigned long long)(nbins - 1)) b = nbins - 1;
    atomicAdd(&bins[b], 1.0);
}

// Cell path (max_r <= cell edge).  A block takes part of a home cell's
// molecules: it stages the 27 neighbour cells' COMs in shared memory in FP32
// relative to the home cell's centre (formed in FP64, then rounded); for each
// home molecule a warp's lanes test 32 staged molecules at a time against
// max_r with a margin and queue the hits of higher index -- the reference
// counts ordered pairs, and (k, o) and (o, k) give the same bin exactly (the
// differences are negatives, and rounding is symmetric), so each pair is
// evaluated once and counted twice.  The queued pairs take rdf_pair_bin's FP64
// arithmetic, whose bins are the reference's.  The counts go to a per-block
// shared histogram of integers (hist_smem) or straight to bins, and the block
// adds its integer counts to bins at the end: the sums are exact, whatever the
// order.  The FP64 pipe bounds it: 32,000 molecules, max_r 2.5 and 100 bins,
// 326 -> 135 us a sample (a warp per cell, ordered pairs, two divisions a pair).
constexpr int kRdfWarps = 4;
constexpr int kRdfStage = 640;
constexpr int kRdfSmemBins = 2048;   // with the staging arrays, under the 48 KB default

// what a bin needs of the RDF's parameters; lo, up, top: the high words of
// 0.4 L, 0.6 L and 1.4 L
struct RdfArgs {
    double max_r, dr, idr;
    float pre2;
    long long nbins;
    int lo[3], up[3], top[3];
};

// the bin of a pair, or -1 beyond max_r: RDF_Kernel's arithmetic.  The minimum
// image round(delta / L) is 0 below 0.4 L and +-1 between 0.6 L and 1.4 L,
// whatever the quotient's rounding.  Away from the bin edges and max_r the bin
// is read off sqrt(r2) / dr by a product with 1 / dr (both within 2e-15 of the
// reference's values, the distance to the edges at least 1e-9 of a bin).  The
// divisions and the square root of the reference run for the rest.
__device__ __forceinline__ long long rdf_pair_bin(const double *ca, const double *cb, const Grid &g,
                                                  const RdfArgs &a) {
    double q[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        q[d] = dsub(ca[d], cb[d]);
        const int hi = __double2hiint(q[d]) & 0x7fffffff;
        if (hi >= a.lo[d]) {
            if (hi > a.up[d] && hi < a.top[d]) {
                q[d] = dsub(q[d], copysign(g.L[d], q[d]));
            } else {
                const double img = (double)(long long)round(ddiv(q[d], g.L[d]));
                q[d] = dsub(q[d], dmul(g.L[d], img));
            }
        }
    }
    const double r2 = dadd(dadd(dmul(q[0], q[0]), dmul(q[1], q[1])), dmul(q[2], q[2]));
    const double t = dmul(sqrt_d(r2, rsqrt_d(r2)), a.idr);
    const int q0 = __double2int_rz(t);
    const long long fr = __double_as_longlong(dsub(t, (double)q0));   // ordered as the value where positive
    if (q0 >= 0 && q0 + 2 < a.nbins && q0 < 1000000 && fr > __double_as_longlong(1e-9) &&
        fr < __double_as_longlong(1.0 - 1e-9))
        return q0;   // below the last bin, so below max_r too
    const double rr = sqrt(r2);
    if (rr > a.max_r) return -1;
    unsigned long long b = (unsigned long long)ddiv(rr, a.dr);
    if (b > (unsigned long long)(a.nbins - 1)) b = a.nbins - 1;
    return (long long)b;
}

__global__ void __launch_bounds__(32 * kRdfWarps) k_rdf_cells(Grid g, const double *__restrict__ com,
                                                              const int *__restrict__ cell_mstart,
                                                              const int *__restrict__ cell_mols, RdfArgs a,
                                                              bool hist_smem, int split, double *bins) {
    extern __shared__ unsigned s_hist[];   // nbins counts when hist_smem
    const long long nbins = a.nbins;
    __shared__ float4 s_p[kRdfStage];      // home-cell coordinates, molecule
    __shared__ double s_sh[27][3], s_ctr[3];
    __shared__ int s_st[27], s_pre[28], s_im[27];
    __shared__ int s_q[kRdfWarps][64];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (hist_smem)
        for (int b = threadIdx.x; b < nbins; b += blockDim.x) s_hist[b] = 0u;
    const int cell = blockIdx.x / split, part = blockIdx.x - cell * split;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (w == 0) {
        int cx, cy, cz, cnt = 0;
        cell_coords(g, cell, cx, cy, cz);
        if (lane < 27) {
            const NbCell q = neighbour_cell(g, cx, cy, cz, lane);
            const int s0 = cell_mstart[q.cell];
            cnt = cell_mstart[q.cell + 1] - s0;
            s_st[lane] = s0;
            s_im[lane] = q.crosses;
            for (int d = 0; d < 3; d++) s_sh[lane][d] = q.shift[d];
        }
        int inc = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane < 27) s_pre[lane] = inc - cnt;
        if (lane == 26) s_pre[27] = inc;
        if (lane < 3) s_ctr[lane] = cell_centre(g, lane, lane == 0 ? cx : (lane == 1 ? cy : cz));
    }
    __syncthreads();
    const int hs = s_st[13], hn = s_pre[14] - s_pre[13];
    const int total = part * kRdfWarps < hn ? s_pre[27] : 0;
    const double ctr[3] = {s_ctr[0], s_ctr[1], s_ctr[2]};
    auto rel = [&](int o, int nb) {   // FP32 COM relative to the home centre, through the periodic shift
        const double *c = com + 3 * (size_t)o;
        double x = c[0], y = c[1], z = c[2];
        if (s_im[nb]) {
            x = dadd(x, s_sh[nb][0]);
            y = dadd(y, s_sh[nb][1]);
            z = dadd(z, s_sh[nb][2]);
        }
        return make_float4(d2f_rn(dsub(x, ctr[0])), d2f_rn(dsub(y, ctr[1])), d2f_rn(dsub(z, ctr[2])),
                           __int_as_float(o));
    };
    for (int sb = 0; sb < total; sb += kRdfStage) {
        const int ns = min(kRdfStage, total - sb);
        if (sb > 0) __syncthreads();
        for (int t = threadIdx.x; t < ns; t += blockDim.x) {
            const int gi = sb + t;
            int nb = 0, e = 27;
            while (e - nb > 1) {
                const int mid = (nb + e) >> 1;
                if (s_pre[mid] <= gi) nb = mid;
                else e = mid;
            }
            s_p[t] = rel(cell_mols[s_st[nb] + (gi - s_pre[nb])], nb);
        }
        __syncthreads();
        for (int h = part * kRdfWarps + w; h < hn; h += split * kRdfWarps) {
            const int k = cell_mols[hs + h];
            const float4 hp = rel(k, 13);
            auto count = [&](int c) {
                if (c < 0) return;
                const long long b = rdf_pair_bin(com + 3 * (size_t)k, com + 3 * (size_t)__float_as_int(s_p[c].w), g,
                                                 a);
                if (b < 0) return;
                if (hist_smem) atomicAdd(&s_hist[b], 2u);
                else atomicAdd(&bins[b], 2.0);
            };
            int qn = 0;
            for (int c0 = 0; c0 < ns; c0 += 32) {
                const int c = c0 + lane;
                bool hit = false;
                if (c < ns) {
                    const float4 pj = s_p[c];
                    const float dx = hp.x - pj.x, dy = hp.y - pj.y, dz = hp.z - pj.z;
                    hit = __float_as_int(pj.w) > k && dx * dx + dy * dy + dz * dz <= a.pre2;
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) s_q[w][qn + __popc(m & lt)] = c;
                qn += __popc(m);
                if (qn >= 32) {
                    __syncwarp();
                    const int c1 = s_q[w][lane], c2 = s_q[w][32 + lane];
                    __syncwarp();
                    qn -= 32;
                    if (lane < qn) s_q[w][lane] = c2;
                    __syncwarp();
                    count(c1);
                }
            }
            __syncwarp();
            count(lane < qn ? s_q[w][lane] : -1);
            __syncwarp();
        }
    }
    if (hist_smem) {
        __syncthreads();
        for (int b = threadIdx.x; b < nbins; b += blockDim.x)
            if (s_hist[b]) atomicAdd(&bins[b], (double)s_hist[b]);
    }
}

__global__ void k_rdf_all(Grid g, int n_mol, const double *__restrict__ com, double max_r, double dr,
                          long long nbins, double *bins) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_mol) return;
    for (int o = 0; o < n_mol; o++)
        if (o != k) rdf_pair(com + 3 * k, com + 3 * o, g, max_r, dr, nbins, bins);
}

// Sums the per-block partial rows: one block of 256 threads per slot, a fixed
// thread-to-row mapping, fixed shuffle trees and a fixed order over the
// warps, so the result is deterministic.
constexpr int kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_sum_partials(int nblocks, const double *__restrict__ partials,
                                                              double *__restrict__ out) {
    pdl_wait();
    __shared__ double s_w[kSumThreads / 32];
    const int slot = blockIdx.x, t = threadIdx.x, lane = t & 31;
    double s = 0.0;
    for (int b = t; b < nblocks; b += kSumThreads) s += partials[(size_t)b * R_NSLOTS + slot];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) s_w[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
        double y = 0.0;
        for (int w = 0; w < kSumThreads / 32; w++) y += s_w[w];
        out[slot] += y;
    }
}

// VelocityScaling (VelocityScaling.cpp:12-25): v *= beta; beta from the
// caller, or (acc != nullptr) sqrt(T_target / T) with T from the summed
// kinetic slots as TemperatureSensor computes it.  A non-finite T (an
// overflowed force upstream) leaves v unscaled and raises E_NONFINITE, which
// the host reads after the step.
__global__ void k_velocity_scale(int n, double *__restrict__ v, const double *__restrict__ acc, double t_target,
                                 SciNum factor, double beta_in, int *__restrict__ err) {
    pdl_trigger();
    pdl_wait();
    __shared__ double s_beta;
    if (threadIdx.x == 0) {
        double beta = beta_in;
        if (acc) {
            const double t = sci_temperature(factor, acc[R_MV2], acc[R_NBOX]);
            if (!isfinite(t)) {
                beta = 1.0;
                if (blockIdx.x == 0 && err) atomicOr(&err[E_NONFINITE], 1);
            } else {
                beta = t > 0.0 ? __dsqrt_rn(__ddiv_rn(t_target, t)) : 1.0;
            }
        }
        s_beta = beta;
    }
    __syncthreads();
    const double beta = s_beta;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 3 * n; k += gridDim.x * blockDim.x)
        v[k] = __dmul_rn(v[k], beta);
}

// ===========================================================================
// launchers
// ===========================================================================
static inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// threads per block of the per-site kernels: 256 where that gives two blocks per
// SM, else 64, so that a small system's FP64 work (the narrow pipe: 16 cycles a
// warp instruction on its SM) spreads over more SMs
static inline int site_block(const Engine &e, long long n) { return n >= 512ll * e.num_sms ? 256 : 64; }

BinArgs bin_args(const Engine &e) {
    BinArgs a = BinArgs{e.g, (int)e.n_mol, e.mol_off, e.r, e.m, e.com, e.mol_cell, e.mol_rank, e.cell_count, e.cell_mcount,
                   e.verlet ? e.bias : nullptr, e.verlet ? e.rebuild : nullptr, e.exact_com, e.fused_drift ? 1 : 0,
                   e.n_mol == e.n ? 1 : 0, {}, {}};
    for (int d = 0; d < 3; d++) {
        a.in_lo[d] = nextafterf((float)e.g.low[d], INFINITY);
        a.in_hi[d] = nextafterf((float)e.g.high[d], -INFINITY);
    }
    return a;
}
ScanArgs scan_args(const Engine &e) {
    return ScanArgs{e.g.ncell, e.n_mol == e.n ? nullptr : e.cell_count, e.cell_start, e.cell_mcount, e.cell_mstart,
                    e.verlet ? e.rebuild : nullptr, e.vb_next};
}
ScatterArgs scatter_args(const Engine &e) {
    return ScatterArgs{(int)e.n_mol, e.mol_cell, e.mol_rank, e.cell_mstart, e.cell_mols,
                       e.verlet ? e.rebuild : nullptr};
}
SortArgs sort_args(const Engine &e) {
    return SortArgs{e.g, e.mol_off, e.cell_mstart, e.cell_start, e.cell_mols, e.r, e.eps, e.sig, e.site_lj, e.key,
                    e.slot_site, e.site_slot, e.pos4, e.skey, e.seps, e.posd, e.seps_d, e.sig_d,
                    e.verlet ? e.bias : nullptr, e.verlet ? e.ref4 : nullptr, e.verlet ? e.slot_cell : nullptr,
                    e.verlet ? e.zkey : nullptr, e.verlet ? e.rebuild : nullptr, e.n_mol == e.n ? 1 : 0};
}
Step0Args step0_args(const Engine &e) {
    const float hs = (float)(0.5 * e.cfg.skin);
    return Step0Args{(int)e.n, e.r, e.v, e.f, e.hdtm, e.cfg.delta_t, e.g, e.bias, e.ref4, hs * hs, e.rebuild,
                     e.site_slot, e.pos4, e.hin_r ? e.hin_r : e.r, e.hin_v ? e.hin_v : e.v, e.hout_r};
}
FlushArgs flush_args(const Engine &e, double scale_fix, const float4 *own) {
    return FlushArgs{(int)e.n, e.site_slot, e.atm_acc, e.f, scale_fix, e.v, e.hdtm, e.err,
                     e.verlet ? e.rebuild : nullptr, e.hout_f, e.hout_v, own};
}

void launch_container(Engine &e, cudaStream_t st) {
    const Grid &g = e.g;
    // without a Verlet list the rebuild flag is null: the kernels rebuild unconditionally
    // the per-cell counts are zero here: zeroed at allocation, and by the scan
    // of every binning after reading them
    // grid-stride kernels on a resident grid: steps without a rebuild launch few blocks
    const int res = e.num_sms * 8;
    const int mb = site_block(e, e.n_mol);
    launch_pdl(k_com_wrap_bin, std::min(nblk(e.n_mol, mb), res * (256 / mb)), mb, 0, st, bin_args(e));
    launch_pdl(k_scan2, 1, 1024, 0, st, scan_args(e));
    launch_pdl(k_scatter_mol, std::min(nblk(e.n_mol, 256), res), 256, 0, st, scatter_args(e));
    // four warps a block: with few cells the chain of loads bounds the sort, not its throughput
    launch_pdl(k_cell_sort, std::min(nblk(g.ncell, 4), 2 * res), 128, 0, st, sort_args(e));
    if (e.verlet) {
        launch_vlist_build(e, st);
    }
}

PairParams pair_params(Engine &e) {
    PairParams p;
    p.g = e.g;
    p.cell_start = e.cell_start;
    p.slot_site = e.slot_site;
    p.pos4 = e.pos4;
    p.posd = e.posd;
    p.skey = e.skey;
    p.seps = e.seps;
    p.seps_d = e.seps_d;
    p.sig_d = e.sig_d;
    p.f = e.f;
    p.counts = e.counts;
    p.nl = e.nl;
    p.nl_count = e.nl_count;
    p.nl_cap = e.nl_cap;
    p.err = e.err;
    p.partials = e.partials;
    p.lj_hist = nullptr;
    p.lj_bins = e.cfg.lj_bins;
    p.max_sigma = e.cfg.max_sigma;
    p.rc2 = e.cfg.cutoff * e.cfg.cutoff;
    p.rc3sq = e.cfg.cutoff_3b * e.cfg.cutoff_3b;
    p.rc2f = (float)p.rc2;
    p.rc3sqf = (float)p.rc3sq;
    const bool atm = (e.cfg.terms & KOMD_TERM_ATM) != 0;
    const bool lj = (e.cfg.terms & KOMD_TERM_LJ) != 0;
    p.scan2 = 0.0;
    if (lj) p.scan2 = p.rc2;
    if (atm && p.rc3sq > p.scan2) p.scan2 = p.rc3sq;
    p.pre2 = pair_pre2(e.g, p.scan2);
    p.stiffness = e.cfg.stiffness;
    p.use_lj = lj ? 1 : 0;
    p.lj_fscale = e.lj_fscale;
    p.lj_scaled = e.lj_fscale != 1.0;
    // constants for one species: sqrt(eps eps) is eps while the square stays normal
    p.uniform = e.uniform && e.eps0 > 1e-30f && e.eps0 < 1e30f;
    p.multi_key = e.multi_key;
    p.lj_fscalef = (float)e.lj_fscale;
    p.virial_compat = e.cfg.virial_mode == KOMD_VIRIAL_COMPAT;
    p.offtab = e.offtab;
    p.rebuild = e.rebuild;
    p.rebuild_done = e.verlet ? e.rebuild : nullptr;
    p.vl = e.vl;
    p.vl_count = e.vl_count;
    p.vl_cap = e.vl_cap;
    const double rl = std::max(lj ? e.cfg.cutoff : 0.0, atm ? e.cfg.cutoff_3b : 0.0) + e.cfg.skin;
    p.rl2 = rl * rl;
    p.slot_cell = e.slot_cell;
    p.zkey = e.zkey;
    p.vb_next = e.vb_next;
    p.nboff = e.nboff;
    p.rebuild_count = e.rebuild_count;
    p.eps0 = e.eps0;
    p.sig0 = e.sig0;
    sw_params(e.cfg.cutoff, e.cfg.switch_width, p.sw, p.sw_rc2, p.sw_iw);
    p.fown = nullptr;   // set by the half-list pass's launchers (half_own)
    return p;
}

// measures and FP64: a resident grid whose warps stride over the vertices (one
// row of partial sums per block, whatever the list capacity)
int atm_grid(const Engine &e) { return std::min(nblk(e.n, kWarpsPerBlock), e.num_sms * 16); }
// warps per block of the FP64 kernel: eight, fewer where their staging (64
// bytes a neighbour) would pass 96 KB
static int atm_warps(const Engine &e) {
    int w = kWarpsPerBlock;
    while (w > 1 && (size_t)w * e.nl_cap * (sizeof(AtmStageD) + sizeof(float4)) > 96 * 1024) w >>= 1;
    return w;
}

// The FP32 force path runs the tiled kernel (pair_tile.cu, one CTA per cell);
// FP64 mode, FENE and the LJ sensor histograms use pair_cell.cu.  FENE acts
// between sites of one molecule ID only: without such a pair the term is
// empty.  Returns the number of blocks whose partial sums were written.
int launch_pair(Engine &e, cudaStream_t st, bool measure, double *lj_hist) {
    PairParams p = pair_params(e);
    p.lj_hist = lj_hist;
    const bool emit = (e.cfg.terms & KOMD_TERM_ATM) != 0;
    const bool fene = (e.cfg.terms & KOMD_TERM_FENE) != 0 && e.multi_key;
    if (e.verlet && !lj_hist) return launch_lj_vlist(e, p, measure, emit, st);
    if (e.cfg.precision == KOMD_FP32 && !fene && !lj_hist) {
        launch_pair_tile(p, e.g.ncell, measure, emit, st);
        return e.g.ncell;
    }
    return launch_pair_cell(e, p, measure, emit, fene, st);
}

void launch_bonded(Engine &e, cudaStream_t st, bool measure, double *acc) {
    if (!measure && e.bond_blocks > 0 && e.bond_sites == e.n) {
        launch_pdl(k_bonded_mol, e.bond_blocks, kBondComps, 0, st, e.bond_block, e.comp_off, e.comp_terms, e.r, e.f,
                   (float)e.cfg.bond_k, (float)e.cfg.bond_r0, (float)e.cfg.angle_k, (float)e.cfg.angle_theta0);
        return;
    }
    if (e.n_bonds > 0)
        k_bonds<<<nblk(e.n_bonds, 256), 256, 0, st>>>((int)e.n_bonds, e.bonds, e.r, e.f, (float)e.cfg.bond_k,
                                                        (float)e.cfg.bond_r0, acc, measure ? 1 : 0);
    if (e.n_angles > 0)
        k_angles<<<nblk(e.n_angles, 256), 256, 0, st>>>((int)e.n_angles, e.angles, e.r, e.f, (float)e.cfg.angle_k,
                                                          (float)e.cfg.angle_theta0, acc, measure ? 1 : 0);
}

void launch_limit(Engine &e, cudaStream_t st) {
    const int b = site_block(e, e.n);
    launch_pdl(k_limit, nblk(e.n, b), b, 0, st, (int)e.n, e.eps, e.sig, e.cfg.limit, e.f);
}

size_t atm_smem(const Engine &e) {
    if (e.cfg.precision == KOMD_FP64) return (size_t)atm_warps(e) * e.nl_cap * (sizeof(AtmStageD) + sizeof(float4));
    return (size_t)kWarpsPerBlock * e.nl_cap * 2 * sizeof(float4);
}

// stage vertex i's neighbours above i (ballot compaction); returns their count
__device__ __forceinline__ int atm_stage(const AtmParams &p, int i, float4 *se, float4 *sq, int lane, unsigned lt) {
    const int ni = min(p.nl_count[i], p.nl_cap);
    int m = 0;
    for (int k0 = 0; k0 < ni; k0 += 32) {
        const int k = k0 + lane;
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
        bool up = false;
        if (k < ni) {
            e = p.nl[(size_t)i * p.nl_cap + k];
            up = (__float_as_int(e.w) >> 6) > i;
        }
        const unsigned bm = __ballot_sync(0xffffffffu, up);
        if (up) {
            const int pos = m + __popc(bm & lt);
            const float A = e.x * e.x + e.y * e.y + e.z * e.z;
            se[pos] = e;
            sq[pos] = atm_stage_q(A);
        }
        m += __popc(bm);
    }
    return m;
}

// one warp per vertex: stage its neighbours above it, then the sweep
__global__ void __launch_bounds__(kBlock) k_atm_s(AtmParams p) {
    pdl_wait();
    extern __shared__ float4 s_dyn[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cap = p.nl_cap;
    float4 *se = s_dyn + wib * 2 * cap, *sq = se + cap;
    const int i = blockIdx.x * kWarpsPerBlock + wib;
    if (i >= p.n) return;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    const int m = atm_stage(p, i, se, sq, lane, lt);
    __syncwarp();
    atm_vertex(p, i, se, sq, m, lane, p.rc2f);
}

// the same flush fused with Integrator::integrate1 of the step (ATM is the
// last force term): f[site] += ..., then v[site] += f[site] * dt/(2m) with
// k_step1's operations, its non-finite check and the rebuild-flag reset
__device__ __forceinline__ void flush_step1_body(const FlushArgs &a, int bid) {
    __shared__ double s_f[3 * kIoBlock], s_v[3 * kIoBlock];
    const int n = a.n;
    const int *__restrict__ site_slot = a.site_slot;
    unsigned long long *__restrict__ acc = a.acc;
    double *__restrict__ f = a.f, *__restrict__ v = a.v;
    const double scale_fix = a.scale_fix;
    const double *__restrict__ hdtm = a.hdtm;
    int *__restrict__ err = a.err, *__restrict__ rebuild = a.rebuild;
    double *f_out = a.f_out, *v_out = a.v_out;
    const int t = threadIdx.x;
    const int base = bid * blockDim.x, site = base + t;
    const int cnt = min((int)blockDim.x, n - base);
    if (rebuild && site == 0) *rebuild = 0;   // every consumer of this step's flag has run
    if (site < n) {
        // one thread per site (f, v, dt/2m coalesced, the accumulators
        // gathered); every load first, then the arithmetic
        const int slot = site_slot[site];
        long long q[3];
        double fo[3], vo[3];
        for (int d = 0; d < 3; d++) q[d] = (long long)acc[3 * slot + d];
        if (a.fown) {   // the half-list pass's FP32 force, widened exactly
            const float4 o = a.fown[slot];
            fo[0] = f2d(o.x);
            fo[1] = f2d(o.y);
            fo[2] = f2d(o.z);
        } else {
            for (int d = 0; d < 3; d++) fo[d] = f[3 * site + d];
        }
        for (int d = 0; d < 3; d++) vo[d] = v[3 * site + d];
        const double c = hdtm[site];
        bool bad = false;
        for (int d = 0; d < 3; d++) {
            acc[3 * slot + d] = 0ull;
            // scale_fix = scale / 2^32 exactly: the same product as scale * (q / 2^32)
            const double fd = fo[d] + scale_fix * (double)q[d];
            f[3 * site + d] = fd;
            const double vv = dadd(vo[d], dmul(fd, c));
            v[3 * site + d] = vv;
            bad |= not_finite(vv);
            s_f[3 * t + d] = fd;
            s_v[3 * t + d] = vv;
        }
        if (bad) atomicOr(&err[E_NONFINITE], 1);
    }
    if (f_out || v_out) {   // the caller's host buffers, in whole lines
        __syncthreads();
        if (f_out) rows_out(s_f, f_out, base, cnt);
        if (v_out) rows_out(s_v, v_out, base, cnt);
    }
}
__global__ void __launch_bounds__(kIoBlock) k_atm_flush_step1(FlushArgs a) {
    pdl_wait();
    flush_step1_body(a, blockIdx.x);
}

// The end of one step and the start of the next in one pass over the sites
// (several steps in one call): the last force term's sums into f (KICK_FLUSH:
// the triplets' fixed-point sums; KICK_LEARNED: the learned term's, from fsur;
// KICK_PLAIN: f is complete), integrate1 of the step and integrate0 of the next
// -- the half-kick f dt/2m is formed once for both -- and the drift.  The
// operations and their order are those of k_atm_flush_step1 / k_sur_apply_step1
// / k_step1 and k_step0_fused.  The rebuild flag is set here for the next step;
// the force pass has cleared it (PairParams::rebuild_done).  256,000 sites: 18 +
// 13.7 us for the two kernels, 22.9 us for this one (24.4 with the FP32 forces
// widened and finiteness tested on the FP64 pipe, which bounds it).
enum { KICK_PLAIN = 0, KICK_FLUSH = 1, KICK_LEARNED = 2 };
template <int MODE>
__device__ __forceinline__ void kick_drift_body(const FlushArgs &a, const Step0Args &dr, float4 *fsur, int bid) {
    const int s = bid * blockDim.x + threadIdx.x;
    if (s >= a.n) return;
    const int slot = a.site_slot[s];
    long long q[3];
    double fo[3], vo[3], ro[3], b[3];
    float4 fs = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE == KICK_FLUSH)
        for (int d = 0; d < 3; d++) q[d] = (long long)a.acc[3 * slot + d];
    if (MODE == KICK_LEARNED) fs = fsur[slot];
    if (MODE == KICK_FLUSH && a.fown) {   // the half-list pass's FP32 force, widened exactly
        const float4 o = a.fown[slot];
        fo[0] = f2d(o.x);
        fo[1] = f2d(o.y);
        fo[2] = f2d(o.z);
    } else {
        for (int d = 0; d < 3; d++) fo[d] = a.f[3 * s + d];
    }
    for (int d = 0; d < 3; d++) {
        vo[d] = a.v[3 * s + d];
        ro[d] = dr.r[3 * s + d];
        b[d] = dr.bias[3 * s + d];
    }
    const double c = a.hdtm[s];
    bool bad = false;
    double x[3];
    for (int d = 0; d < 3; d++) {
        double fd = fo[d];
        if (MODE == KICK_FLUSH) {
            a.acc[3 * slot + d] = 0ull;
            fd = fo[d] + a.scale_fix * (double)q[d];
            a.f[3 * s + d] = fd;
        }
        if (MODE == KICK_LEARNED) {
            fd = fo[d] + f2d(d == 0 ? fs.x : (d == 1 ? fs.y : fs.z));
            a.f[3 * s + d] = fd;
        }
        const double kick = dmul(fd, c), v1 = dadd(vo[d], kick);
        bad |= not_finite(v1);
        const double v2 = dadd(v1, kick);
        a.v[3 * s + d] = v2;
        x[d] = dadd(ro[d], dmul(v2, dr.dt));
    }
    if (MODE == KICK_LEARNED) fsur[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bad) atomicOr(&a.err[E_NONFINITE], 1);
    drift_finish(dr, s, slot, x, b);
}
template <int MODE>
__global__ void __launch_bounds__(kIoBlock) k_kick_drift(FlushArgs a, Step0Args dr, float4 *fsur) {
    pdl_trigger();
    pdl_wait();
    kick_drift_body<MODE>(a, dr, fsur, blockIdx.x);
}

// the same for systems outside the fused drift (per-step cells, molecules of
// several sites): k_step1's and k_step0's operations
__global__ void k_step10(int n, double *__restrict__ r, double *__restrict__ v, const double *__restrict__ f,
                         const double *__restrict__ hdtm, double dt, const double *__restrict__ bias,
                         const float4 *__restrict__ ref4, const int *__restrict__ site_slot,
                         float4 *__restrict__ pos4, float half_skin2, int *__restrict__ rebuild,
                         int *__restrict__ err) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double c = hdtm[s];
    double x[3], vo[3], fo[3];
    for (int d = 0; d < 3; d++) {
        vo[d] = v[3 * s + d];
        fo[d] = f[3 * s + d];
        x[d] = r[3 * s + d];
    }
    bool bad = false;
    for (int d = 0; d < 3; d++) {
        const double kick = dmul(fo[d], c), v1 = dadd(vo[d], kick);
        bad |= not_finite(v1);
        const double v2 = dadd(v1, kick);
        v[3 * s + d] = v2;
        x[d] = dadd(x[d], dmul(v2, dt));
        r[3 * s + d] = x[d];
    }
    if (bad) atomicOr(&err[E_NONFINITE], 1);
    if (bias) local_position(s, x, bias, ref4, site_slot, pos4, half_skin2, rebuild);
}

// f[site] += 2 sign nu g (fixed point -> FP64) and the accumulators back to 0
__global__ void k_atm_flush(int n, const int *__restrict__ slot_site, unsigned long long *__restrict__ acc,
                            double *__restrict__ f, double scale_fix, const float4 *__restrict__ own) {
    pdl_wait();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const int site = slot_site[slot];
    long long q[3];
    double fo[3];
    for (int d = 0; d < 3; d++) q[d] = (long long)acc[3 * slot + d];
    if (own) {   // the half-list pass's FP32 force, widened exactly
        const float4 o = own[slot];
        fo[0] = f2d(o.x);
        fo[1] = f2d(o.y);
        fo[2] = f2d(o.z);
    } else {
        for (int d = 0; d < 3; d++) fo[d] = f[3 * site + d];
    }
    for (int d = 0; d < 3; d++) {
        acc[3 * slot + d] = 0ull;
        f[3 * site + d] = fo[d] + scale_fix * (double)q[d];
    }
}

static void atm_dispatch_f(AtmParams &p, bool measure, bool compat, int grid, size_t sm, cudaStream_t st) {
    if (measure) {
        if (compat) launch_pdl(k_atm_q<true, true>, grid, kBlock, sm, st, p);
        else launch_pdl(k_atm_q<true, false>, grid, kBlock, sm, st, p);
    } else {
        if (compat) launch_pdl(k_atm_q<false, true>, grid, kBlock, sm, st, p);
        else launch_pdl(k_atm_q<false, false>, grid, kBlock, sm, st, p);
    }
}

static void atm_dispatch_d(AtmParams &p, bool measure, bool compat, int grid, int warps, size_t sm, cudaStream_t st) {
    if (measure) {
        if (compat) k_atm_d<true, true><<<grid, 32 * warps, sm, st>>>(p);
        else k_atm_d<true, false><<<grid, 32 * warps, sm, st>>>(p);
    } else {
        if (compat) k_atm_d<false, true><<<grid, 32 * warps, sm, st>>>(p);
        else k_atm_d<false, false><<<grid, 32 * warps, sm, st>>>(p);
    }
}

AtmParams atm_params(const Engine &e) {
    AtmParams p;
    p.n = (int)e.n;
    p.slot_site = e.slot_site;
    p.nl = e.nl;
    p.nl_count = e.nl_count;
    p.nl_cap = e.nl_cap;
    p.f = e.f;
    p.partials = e.partials;
    p.nu = e.cfg.nu;
    p.rc2 = e.cfg.cutoff_3b * e.cfg.cutoff_3b;
    p.sign = e.cfg.atm_sign == KOMD_ATM_SIGN_REFERENCE ? 1.0 : -1.0;
    p.share = 2.0 * p.sign * p.nu;
    p.rc2f = (float)p.rc2;
    p.virial_compat = e.cfg.virial_mode == KOMD_VIRIAL_COMPAT;
    p.atm_direct = e.cfg.atm_direct;
    p.e_site = e.atm_esite;
    p.acc = e.atm_acc;
    sw_params(e.cfg.cutoff_3b, e.cfg.switch_width, p.sw, p.sw_rc2, p.sw_iw);
    return p;
}

// the fixed-point sums of the once-per-triplet sweep into f and, where a kernel
// takes it along, the step's end; returns whether it did
bool launch_atm_flush(Engine &e, cudaStream_t st, StepEnd end, bool force_units) {
    const double sign = e.cfg.atm_sign == KOMD_ATM_SIGN_REFERENCE ? 1.0 : -1.0;
    const double scale_fix = force_units ? 1.0 / kAtmFix : 2.0 * sign * e.cfg.nu / kAtmFix;
    const float4 *own = force_units ? half_own(e) : nullptr;   // force_units: the half-list pass ran
    if (end == END_STEP1) {
        const int b = site_block(e, e.n);
        launch_pdl(k_atm_flush_step1, nblk(e.n, b), b, 0, st, flush_args(e, scale_fix, own));
        return true;
    }
    if (end == END_KICK_DRIFT && e.fused_drift) {
        const int b = site_block(e, e.n);
        launch_pdl(k_kick_drift<KICK_FLUSH>, nblk(e.n, b), b, 0, st, flush_args(e, scale_fix, own), step0_args(e),
                   (float4 *)nullptr);
        return true;
    }
    launch_pdl(k_atm_flush, nblk(e.n, 256), 256, 0, st, (int)e.n, e.slot_site, e.atm_acc, e.f, scale_fix, own);
    return false;
}

bool launch_atm(Engine &e, cudaStream_t st, bool measure, StepEnd end) {
    AtmParams p = atm_params(e);
    const bool compat = e.cfg.atm_enum == KOMD_ATM_ENUM_COMPAT;
    if (!measure && !compat && e.cfg.precision == KOMD_FP32 && e.atm_acc) {
        // every triplet once (lowest slot), fixed-point scatter, then the flush into f
        launch_pdl(k_atm_s, nblk(e.n, kWarpsPerBlock), kBlock, atm_smem(e), st, p);
        return launch_atm_flush(e, st, end, false);
    }
    if (e.cfg.precision == KOMD_FP64)
        atm_dispatch_d(p, measure, compat, atm_grid(e), atm_warps(e), atm_smem(e), st);
    else atm_dispatch_f(p, measure, compat, measure ? atm_grid(e) : nblk(e.n, kWarpsPerBlock), atm_smem(e), st);
    return false;
}

void launch_step0(Engine &e, cudaStream_t st, bool in_step) {
    const float hs = (float)(0.5 * e.cfg.skin);
    if (in_step && e.fused_drift) {
        const int b = site_block(e, e.n);
        launch_pdl(k_step0_fused, nblk(e.n, b), b, 0, st, step0_args(e));
        return;
    }
    const int b = site_block(e, e.n);
    launch_pdl(k_step0, nblk(e.n, b), b, 0, st, (int)e.n, e.r, e.v, e.f, e.hdtm, e.cfg.delta_t,
               e.verlet ? e.bias : nullptr, e.verlet ? e.ref4 : nullptr, e.site_slot, e.pos4, hs * hs, e.rebuild);
}

// integrate1 of a step and integrate0 of the next
void launch_kick_drift(Engine &e, cudaStream_t st) {
    const int b = site_block(e, e.n);
    if (e.fused_drift) {
        launch_pdl(k_kick_drift<KICK_PLAIN>, nblk(e.n, b), b, 0, st, flush_args(e, 0.0, nullptr), step0_args(e),
                   (float4 *)nullptr);
        return;
    }
    const float hs = (float)(0.5 * e.cfg.skin);
    launch_pdl(k_step10, nblk(e.n, b), b, 0, st, (int)e.n, e.r, e.v, e.f, e.hdtm, e.cfg.delta_t,
               e.verlet ? e.bias : nullptr, e.verlet ? e.ref4 : nullptr, e.site_slot, e.pos4, hs * hs, e.rebuild,
               e.err);
}

// the same with the learned term's forces (fsur, slot order) added first; needs the fused drift
void launch_learned_kick_drift(Engine &e, float *fsur, cudaStream_t st) {
    const int b = site_block(e, e.n);
    launch_pdl(k_kick_drift<KICK_LEARNED>, nblk(e.n, b), b, 0, st, flush_args(e, 0.0, nullptr), step0_args(e),
               reinterpret_cast<float4 *>(fsur));
}

void launch_step1(Engine &e, cudaStream_t st) {
    const int b = site_block(e, e.n);
    launch_pdl(k_step1, nblk(e.n, b), b, 0, st, (int)e.n, e.v, e.f, e.hdtm, e.err, e.verlet ? e.rebuild : nullptr);
}

int kinetic_grid(const Engine &e) { return std::min(nblk(e.n, kBlock), e.num_sms * 2); }

void launch_velocity_scale(Engine &e, cudaStream_t st, const double *acc, double beta) {
    const int b = site_block(e, 3 * e.n);
    launch_pdl(k_velocity_scale, std::min(nblk(3 * e.n, b), e.num_sms * 8), b, 0, st, (int)e.n, e.v, acc,
               e.cfg.temperature_target, sci_factor(), beta, e.err);
}

// the kinetic sums into acc (R_NSLOTS), whose other slots become zero
void launch_kinetic(Engine &e, cudaStream_t st, int n_terms, double *acc, bool step1) {
    auto k = step1 ? k_kinetic<false, true> : n_terms > 0 ? k_kinetic<true, false> : k_kinetic<false, false>;
    launch_pdl(k, kinetic_grid(e), kBlock, 0, st, e.g, (int)e.n, n_terms, e.r, e.v, e.m, e.partials, acc, e.kin_done,
               e.f, e.hdtm, e.err, e.verlet ? e.rebuild : nullptr);
}

void launch_sum_partials(cudaStream_t st, int nblocks, const double *partials, double *out) {
    launch_pdl(k_sum_partials, R_NSLOTS, kSumThreads, 0, st, nblocks, partials, out);
}

void launch_rdf(Engine &e, cudaStream_t st, double *bins, bool cells) {
    launch_rdf_bins(e, st, bins, cells, e.cfg.rdf_max, e.cfg.rdf_dr, e.rdf_bins);
}

void launch_rdf_bins(Engine &e, cudaStream_t st, double *bins, bool cells, double max_r, double dr, int64_t nbins) {
    if (cells) {
        const bool hist_smem = nbins <= kRdfSmemBins;
        // parts of a cell's molecules where there are few cells, as in pair_cell.cu
        const int most = std::max(1, (int)((double)e.n_mol / e.g.ncell / kRdfWarps + 0.999));
        const int split = std::max(1, std::min(most, (e.num_sms * 8 + e.g.ncell - 1) / e.g.ncell));
        RdfArgs a{max_r, dr, 1.0 / dr, pair_pre2(e.g, max_r * max_r), nbins, {0}, {0}, {0}};
        auto high = [](double x) {
            uint64_t b;
            std::memcpy(&b, &x, sizeof(b));
            return (int)(b >> 32);
        };
        for (int d = 0; d < 3; d++) {
            a.lo[d] = high(0.4 * e.g.L[d]);
            a.up[d] = high(0.6 * e.g.L[d]);
            a.top[d] = high(1.4 * e.g.L[d]);
        }
        k_rdf_cells<<<e.g.ncell * split, 32 * kRdfWarps, hist_smem ? sizeof(unsigned) * nbins : 0, st>>>(
            e.g, e.com, e.cell_mstart, e.cell_mols, a, hist_smem, split, bins);
    }
    else
        k_rdf_all<<<nblk(e.n_mol, 128), 128, 0, st>>>(e.g, (int)e.n_mol, e.com, max_r, dr, nbins, bins);
}

// Shared memory above the default 48 KB (static and dynamic together) has to be
// allowed kernel by kernel, and the limit is the process's, not the engine's: it is
// only ever raised, so that an engine with small lists does not take from one with
// larger ones what that one's launches need.
void allow_smem(const void *kernel, size_t bytes) {
    if (bytes <= 40 * 1024) return;   // the static arrays are below 8 KB
    static std::mutex mutex;
    std::lock_guard<std::mutex> lock(mutex);
    const int want = std::max((int)bytes, 49 * 1024);   // above the default, so that it reads as allowed
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, kernel) == cudaSuccess && a.maxDynamicSharedSizeBytes >= want) return;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, want);
}

// the ATM kernels' staging, whose size follows the list capacity
void set_kernel_attributes(Engine &e) {
    const size_t sm = atm_smem(e);
    if (e.cfg.precision == KOMD_FP64) {
        for (auto k : {k_atm_d<true, true>, k_atm_d<true, false>, k_atm_d<false, true>, k_atm_d<false, false>})
            allow_smem((const void *)k, sm);
    } else {
        for (auto k : {k_atm_s, k_atm_q<true, true>, k_atm_q<true, false>, k_atm_q<false, true>, k_atm_q<false, false>})
            allow_smem((const void *)k, sm);
    }
}

// ---- packed replicas (kernels.cuh): the container, drift and flush stages of
// every replica in one launch each
__device__ __forceinline__ int packed_rep(const int *__restrict__ start, int nrep, int b) {
    int lo = 0, hi = nrep;   // start[0] = 0 <= b < start[nrep]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}
// the packed per-site stages at 32 registers (eight blocks per SM): the
// groups' stages share the SMs, and the force pass of another group needs
// the register file (6.43 against 6.46 ms per step for 512 replicas)
__global__ void __launch_bounds__(kIoBlock, 8) k_step0_fused_p(const Step0Args *a, const int *start, int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    step0_fused_body(a[r], blockIdx.x - start[r]);
}
__global__ void k_com_wrap_bin_p(const BinArgs *a, const int *start, int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    com_wrap_bin_body(a[r], blockIdx.x - start[r], start[r + 1] - start[r]);
}
__global__ void __launch_bounds__(1024) k_scan2_p(const ScanArgs *a) { scan2_body(a[blockIdx.x]); }
__global__ void k_scatter_mol_p(const ScatterArgs *a, const int *start, int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    scatter_mol_body(a[r], blockIdx.x - start[r], start[r + 1] - start[r]);
}
__global__ void __launch_bounds__(kBlock, 4) k_cell_sort_p(const SortArgs *a, const int *start, int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    cell_sort_body(a[r], blockIdx.x - start[r], start[r + 1] - start[r]);
}
__global__ void __launch_bounds__(kIoBlock, 8) k_atm_flush_step1_p(const FlushArgs *a, const int *start, int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    flush_step1_body(a[r], blockIdx.x - start[r]);
}

__global__ void __launch_bounds__(kIoBlock, 5) k_kick_drift_p(const FlushArgs *a, const Step0Args *dr, const int *start,
                                                              int nrep) {
    const int r = packed_rep(start, nrep, blockIdx.x);
    kick_drift_body<KICK_FLUSH>(a[r], dr[r], nullptr, blockIdx.x - start[r]);
}

// blocks per replica of the container stages: on a step without a rebuild
// they exit at once; on a rebuild step a replica's blocks do its whole
// binning, so too few of them make a long tail for the launch
int packed_blocks_container(const Engine &e) { return std::max(1, std::min(nblk(e.n_mol, 256), 64)); }

// `steps` steps of every replica: the stages of enqueue_steps on the Verlet path
// with the fused drift and the half-list pass, each stage one launch; a step's
// flush takes the next one's drift along
void launch_packed_steps(const PackedStep &pk, int steps, cudaStream_t st) {
    const int nr = pk.nrep;
    const Step0Args *dr = (const Step0Args *)pk.step0.args;
    const FlushArgs *fl = (const FlushArgs *)pk.flush.args;
    k_step0_fused_p<<<pk.step0.blocks, kIoBlock, 0, st>>>(dr, pk.step0.start, nr);
    for (int k = 0; k < steps; k++) {
        k_com_wrap_bin_p<<<pk.bin.blocks, 256, 0, st>>>((const BinArgs *)pk.bin.args, pk.bin.start, nr);
        k_scan2_p<<<nr, 1024, 0, st>>>((const ScanArgs *)pk.scan.args);
        k_scatter_mol_p<<<pk.scatter.blocks, 256, 0, st>>>((const ScatterArgs *)pk.scatter.args, pk.scatter.start, nr);
        k_cell_sort_p<<<pk.sort.blocks, kBlock, 0, st>>>((const SortArgs *)pk.sort.args, pk.sort.start, nr);
        launch_packed_pair_stages(pk, st, true);
        launch_packed_pair_stages(pk, st, false);
        if (k + 1 < steps) k_kick_drift_p<<<pk.flush.blocks, kIoBlock, 0, st>>>(fl, dr, pk.flush.start, nr);
        else k_atm_flush_step1_p<<<pk.flush.blocks, kIoBlock, 0, st>>>(fl, pk.flush.start, nr);
    }
}


}  // namespace komd
