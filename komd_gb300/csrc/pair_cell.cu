// pair_cell.cu -- the pair kernel of the per-step cell lists: LJ 12-6
// (LJ12_6.cpp:15-43) and FENE (FENE.cpp:15-43) with the ATM neighbour list,
// energy, virial and histograms; the tabulated force of the IBI plugin
// (plugins/IBI/IBI_ForceFunctor.cpp:18-37); and the neighbour counts.
//
// Full shell (27 neighbour cells, periodic images by cell wrap), no atomics on
// forces.  A block of four warps takes part of a home cell's sites: it stages
// the 27-cell neighbourhood in shared memory in FP32 home-cell coordinates,
// and each warp walks home sites: 32 staged sites at a time are tested against
// the range, the hits queued by ballot, and the queue evaluated 32 pairs at a
// time on full warps.
//
// Real = double: the FP32 test keeps a margin over the coordinates' rounding
// (pre2), so it drops only pairs that are outside; the queued pairs take the
// reference's FP64 arithmetic from the absolute positions, with the exact
// range test.  GB300 issues FP64 at about 1/64 of its FP32 rate, so the FP64
// pipe bounds this form, and only pairs near or inside the range may reach
// it; comparisons are made on the doubles' bits (integer pipe), a division
// 1 / x is one correctly rounded reciprocal, r and 1 / r of the table's force
// come from one reciprocal root (rsqrt_d: 181 -> 145 us a launch at 32,000
// sites against a square root and a reciprocal), and the warp's sums split
// their components over the lanes (6 additions instead of 15).
// Real = float: the staged coordinates are the operands; issue-bound.
//
// Against one warp per home cell with every candidate in the result type, a launch:
// FP64 LJ on 4,000 sites 944 -> 30 us (with the sensors 1326 -> 50), on 32,000 with the
// ATM list 1344 -> 149, FP32 LJ + FENE on 1,536 sites of molecules 68 -> 11, and the
// tabulated force on 32,000 sites (a warp per cell that staged for itself) 347 -> 145.
#include <climits>
#include <cstdint>

#include "engine.cuh"
#include "kernels.cuh"

namespace komd {

constexpr int kPcWarps = 4;      // warps (home sites in flight) per block
constexpr int kPcStage = 640;    // staged sites per round (more rounds for a larger neighbourhood)

enum PairKind { PC_LJ = 0, PC_TABLE = 1, PC_COUNT = 2 };

__device__ __forceinline__ bool above(double a, double b) { return dabove(a, b); }
__device__ __forceinline__ bool above(float a, float b) { return a > b; }

// FunctionPL::evaluateAt (plugins/IBI/IBI_Math.h:30-44): the upper node is the
// first node >= r (by binary search on integer keys, the node the reference's
// linear scan finds), slope[k] = (y[k+1] - y[k]) / (x[k+1] - x[k]) is the
// reference's quotient, computed once with the same IEEE operations.  At
// r == x[0] the reference reads x[-1]; here the first segment is used.
__device__ __forceinline__ double table_eval(double r, const PairTable &t) {
    const long long kr = dkey(r);
    if (kr > dkey(t.xs[t.n - 1])) return t.hi;
    if (kr < dkey(t.xs[0])) return t.lo;
    int a = 0, b = t.n - 1;           // lower_bound: first index with xs[i] >= r
    while (a < b) {
        const int m = (a + b) >> 1;
        if (kr > dkey(t.xs[m])) a = m + 1;
        else b = m;
    }
    const int lb = (a < 1 ? 1 : a) - 1;
    return dadd(t.ys[lb], dmul(t.slope[lb], dsub(r, t.xs[lb])));
}

template <typename Real, int KIND, bool MEASURE, bool EMIT, bool FENE>
__global__ void __launch_bounds__(32 * kPcWarps) k_pair_cell(PairParams p, PairTable tab, int split) {
    constexpr bool FP64 = sizeof(Real) == 8;
    __shared__ float4 s_p[kPcStage];             // home-cell coordinates, sigma/2
    __shared__ int2 s_j[kPcStage];               // slot, neighbour cell | image << 5
    __shared__ int s_k[FENE ? kPcStage : 1];     // molecule key
    __shared__ double s_sh[27][3];
    __shared__ float s_o[27][3];
    __shared__ int s_st[27], s_pre[28], s_im[27];
    __shared__ int s_q[kPcWarps][64];
    __shared__ double s_part[MEASURE ? kPcWarps : 1][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int cell = blockIdx.x / split, part = blockIdx.x - cell * split;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (w == 0) {
        int cx, cy, cz;
        cell_coords(p.g, cell, cx, cy, cz);
        int cnt = 0;
        if (lane < 27) {
            const NbCell q = neighbour_cell(p.g, cx, cy, cz, lane);
            const int s0 = p.cell_start[q.cell];
            cnt = p.cell_start[q.cell + 1] - s0;
            s_st[lane] = s0;
            s_im[lane] = q.crosses ? 32 : 0;
            if (FP64)
                for (int d = 0; d < 3; d++) s_sh[lane][d] = q.shift[d];
            s_o[lane][0] = p.offtab[cx * 3 + lane % 3];
            s_o[lane][1] = p.offtab[p.g.nd[0] * 3 + cy * 3 + (lane / 3) % 3];
            s_o[lane][2] = p.offtab[(p.g.nd[0] + p.g.nd[1]) * 3 + cz * 3 + lane / 9];
        }
        int inc = cnt;   // inclusive prefix of the 27 counts
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane < 27) s_pre[lane] = inc - cnt;
        if (lane == 26) s_pre[27] = inc;
    }
    __syncthreads();
    const int hs = s_st[13], hn = s_pre[14] - s_pre[13];   // neighbour 13 is the home cell
    const int total = part * kPcWarps < hn ? s_pre[27] : 0;   // a part without home sites stages nothing
    const float pre2 = FP64 ? p.pre2 : (float)p.scan2;
    const Real rc2 = (Real)p.rc2, rc3sq = (Real)p.rc3sq;
    double a_u = 0.0, a_w[6] = {0, 0, 0, 0, 0, 0};
    int a_pairs = 0;

    for (int sb = 0; sb < total; sb += kPcStage) {
        const int ns = min(kPcStage, total - sb);
        if (sb > 0) __syncthreads();
        for (int t = threadIdx.x; t < ns; t += 32 * kPcWarps) {
            const int gi = sb + t;
            int a = 0, b = 27;   // the neighbour cell holding staged site gi
            while (b - a > 1) {
                const int mid = (a + b) >> 1;
                if (s_pre[mid] <= gi) a = mid;
                else b = mid;
            }
            const int j = s_st[a] + (gi - s_pre[a]);
            float4 q = p.pos4[j];
            q.x += s_o[a][0];
            q.y += s_o[a][1];
            q.z += s_o[a][2];
            s_p[t] = q;
            s_j[t] = make_int2(j, a | s_im[a]);
            if (FENE) s_k[t] = p.skey[j];
        }
        __syncthreads();
        for (int h = part * kPcWarps + w; h < hn; h += split * kPcWarps) {
            const int is = hs + h;
            const float4 hp = p.pos4[is];
            const int ki = p.skey[is], site_i = p.slot_site[is];
            const int self = s_pre[13] + h - sb;
            Real pix = 0, piy = 0, piz = 0, sgi = 0, epi = 0;
            if (FP64) {
                pix = (Real)p.posd[3 * (size_t)is];
                piy = (Real)p.posd[3 * (size_t)is + 1];
                piz = (Real)p.posd[3 * (size_t)is + 2];
                sgi = (Real)p.sig_d[is];
                epi = (Real)p.seps_d[is];
            } else {
                sgi = hp.w;
                epi = p.seps[is];
            }
            Real fx = 0, fy = 0, fz = 0;
            int cnt = EMIT && sb > 0 ? p.nl_count[is] : 0;   // counts run on over the rounds

            auto eval = [&](int c, bool valid) {   // every lane calls
                Real dx = 0, dy = 0, dz = 0, r2 = 0;
                int j = 0, code = 0;
                if (valid) {
                    const int2 jn = s_j[c];
                    j = jn.x;
                    code = jn.y;
                    if (FP64) {
                        const double *pj = p.posd + 3 * (size_t)j;
                        double x = pj[0], y = pj[1], z = pj[2];
                        if (code & 32) {   // the image's shift (zero otherwise)
                            const double *sh = s_sh[code & 31];
                            x = dadd(x, sh[0]);
                            y = dadd(y, sh[1]);
                            z = dadd(z, sh[2]);
                        }
                        dx = (Real)dsub((double)pix, x);
                        dy = (Real)dsub((double)piy, y);
                        dz = (Real)dsub((double)piz, z);
                        r2 = (Real)dadd(dadd(dmul((double)dx, (double)dx), dmul((double)dy, (double)dy)),
                                        dmul((double)dz, (double)dz));
                    } else {
                        const float4 pj = s_p[c];
                        dx = hp.x - pj.x;
                        dy = hp.y - pj.y;
                        dz = hp.z - pj.z;
                        r2 = dx * dx + dy * dy + dz * dz;
                    }
                }
                if constexpr (KIND == PC_TABLE) {
                    // (dr / r) * F as dr * (F / r), 1 / r and r from one reciprocal root
                    if (valid && !above(r2, rc2)) {
                        const double ir = rsqrt_d((double)r2);
                        const double Fr = dmul(ir, table_eval(sqrt_d((double)r2, ir), tab));
                        fx = (Real)__fma_rn((double)dx, Fr, (double)fx);
                        fy = (Real)__fma_rn((double)dy, Fr, (double)fy);
                        fz = (Real)__fma_rn((double)dz, Fr, (double)fz);
                    }
                    return;
                }
                const bool same = valid && p.multi_key && p.skey[j] == ki;
                if constexpr (KIND == PC_COUNT) {
                    if (valid && !above(r2, rc2) && !same) cnt++;
                    return;
                }
                if (FENE && same && !(code & 32)) {
                    // same-molecule pairs, no cutoff: force on i along (r_j - r_i),
                    // overstretch -> 1e30 / (r_j - r_i)  (FENE.cpp:28-33)
                    const Real sgj = FP64 ? (Real)p.sig_d[j] : (Real)(2.0f * s_p[c].w);
                    const Real sgm = FP64 ? (sgi + sgj) / (Real)2.0 : (sgi + (Real)0.5 * sgj);
                    const Real R0 = (Real)1.5 * sgm;
                    const Real R02 = R0 * R0;
                    if (R02 <= r2) {
                        fx += ((Real)1 / (-dx)) * (Real)1e30;
                        fy += ((Real)1 / (-dy)) * (Real)1e30;
                        fz += ((Real)1 / (-dz)) * (Real)1e30;
                    } else {
                        Real e;
                        if (FP64) e = (Real)sqrt((double)epi * (double)p.seps_d[j]);
                        else e = epi * (Real)p.seps[j];
                        const Real k = (Real)p.stiffness * e / (sgm * sgm);
                        const Real fac = k / ((Real)1 - (r2 / R02));
                        fx -= dx * fac; fy -= dy * fac; fz -= dz * fac;
                    }
                }
                if (EMIT) {   // r_i - r_j and the code, in queue order
                    const bool emit = valid && !above(r2, rc3sq);
                    const unsigned em = __ballot_sync(0xffffffffu, emit);
                    if (emit) {
                        const int c2 = cnt + __popc(em & lt);
                        if (c2 < p.nl_cap) {
                            const size_t at = (size_t)is * p.nl_cap + c2;
                            if constexpr (FP64) {
                                AtmEntryD en;
                                en.x = dx; en.y = dy; en.z = dz;
                                en.code = code | (j << 6);
                                reinterpret_cast<AtmEntryD *>(p.nl)[at] = en;
                            } else {
                                p.nl[at] = make_float4(dx, dy, dz, __int_as_float(code | (j << 6)));
                            }
                        }
                    }
                    cnt += __popc(em);
                }
                if (!p.use_lj || !valid || above(r2, rc2) || same) return;
                Real fac, u, ljd;
                if (FP64) {
                    // LJ12_6_Force arithmetic in FP64 (pow(x, 3.0), pow(lj6, 2.0) as
                    // products); for equal species (s + s) / 2 and sqrt(e e) are s and e exactly
                    const double inv = __drcp_rn((double)r2);
                    double sg2, e;
                    if (p.uniform) {
                        sg2 = (double)sgi * (double)sgi;
                        e = epi;
                    } else {
                        const double sgm = (p.sig_d[j] + (double)sgi) / 2.0;
                        sg2 = sgm * sgm;
                        e = sqrt((double)epi * p.seps_d[j]);
                    }
                    const double x = sg2 * inv;
                    const double lj6 = x * x * x, lj12 = lj6 * lj6;
                    ljd = (Real)(24.0 * e * (2.0 * lj12 - lj6));
                    fac = (Real)((double)ljd * inv);
                    u = (Real)(4.0 * e * (lj12 - lj6));
                } else {
                    const float inv = __frcp_rn((float)r2);
                    const float sgm = (float)sgi + s_p[c].w;
                    const float x = sgm * sgm * inv;
                    const float lj6 = x * x * x, lj12 = lj6 * lj6;
                    const float e = (float)epi * (p.uniform ? (float)epi : p.seps[j]);
                    ljd = 24.0f * e * (2.0f * lj12 - lj6);
                    fac = ljd * inv;
                    u = 4.0f * e * (lj12 - lj6);
                }
                if (!MEASURE) {
                    if (p.lj_scaled) fac *= (Real)p.lj_fscale;   // ATM2B; sensors stay unscaled
                    fx += dx * fac; fy += dy * fac; fz += dz * fac;
                } else {
                    fx += dx * fac; fy += dy * fac; fz += dz * fac;
                    // COMPAT: image pairs counted per list entry
                    const double wf = (p.virial_compat && (code & 32)) ? (double)fac : 0.5 * (double)fac;
                    const double gx = (double)dx * wf, gy = (double)dy * wf, gz = (double)dz * wf;
                    a_u += 0.5 * (double)u;
                    a_pairs++;
                    a_w[0] += (double)dx * gx;
                    a_w[1] += (double)dx * gy;
                    a_w[2] += (double)dy * gy;
                    a_w[3] += (double)dx * gz;
                    a_w[4] += (double)dy * gz;
                    a_w[5] += (double)dz * gz;
                    if (p.lj_hist) {
                        const int site_j = p.slot_site[j];
                        if (site_i < site_j) {
                            const double rp = sqrt((double)r2);
                            const double bw = 3.0 * p.max_sigma / (double)p.lj_bins;
                            unsigned long long bin = (unsigned long long)(rp / bw);
                            if (bin > (unsigned long long)(p.lj_bins - 1)) bin = p.lj_bins - 1;
                            atomicAdd(&p.lj_hist[bin], (double)u);
                            atomicAdd(&p.lj_hist[p.lj_bins + bin], (double)ljd / rp);
                            atomicAdd(&p.lj_hist[2 * p.lj_bins + bin], 1.0);
                            atomicAdd(&p.lj_hist[3 * p.lj_bins + bin], 1.0);
                        }
                    }
                }
            };

            int qn = 0;
            for (int c0 = 0; c0 < ns; c0 += 32) {
                const int c = c0 + lane;
                bool hit = false;
                if (c < ns && c != self) {
                    const float4 pj = s_p[c];
                    const float dx = hp.x - pj.x, dy = hp.y - pj.y, dz = hp.z - pj.z;
                    hit = !(dx * dx + dy * dy + dz * dz > pre2);
                    if (FENE) hit = hit || (s_k[c] == ki && !(s_j[c].y & 32));
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) s_q[w][qn + __popc(m & lt)] = c;
                qn += __popc(m);
                if (qn >= 32) {   // a full batch: one queued pair per lane
                    __syncwarp();
                    const int c1 = s_q[w][lane], c2 = s_q[w][32 + lane];
                    __syncwarp();
                    qn -= 32;
                    if (lane < qn) s_q[w][lane] = c2;
                    __syncwarp();
                    eval(c1, true);
                }
            }
            __syncwarp();
            if (qn > 0) {
                const int c1 = lane < qn ? s_q[w][lane] : 0;
                __syncwarp();
                eval(c1, lane < qn);
            }
            if constexpr (KIND == PC_COUNT) {
                const int c = __reduce_add_sync(0xffffffffu, cnt);
                if (lane == 0) p.counts[site_i] = (sb > 0 ? p.counts[site_i] : 0) + c;
            } else {
                const Real fs = warp_sum3(fx, fy, fz, lane);
                if ((lane & 7) == 0 && lane < 24) {
                    double *o = p.f + 3 * (size_t)site_i + (lane >> 3);
                    // the first writer of f in a step, but the table's force adds to it
                    *o = (KIND == PC_TABLE || sb > 0) ? dadd(*o, (double)fs) : (double)fs;
                }
                if (EMIT && lane == 0) {
                    const bool last = sb + kPcStage >= total;
                    p.nl_count[is] = last ? min(cnt, p.nl_cap) : cnt;
                    if (last && cnt > p.nl_cap) atomicOr(&p.err[E_ATM_OVERFLOW], 1);
                }
            }
            __syncwarp();
        }
    }
    if (MEASURE) {
        double vals[8] = {a_u, a_w[0], a_w[1], a_w[2], a_w[3], a_w[4], a_w[5], 0.0};
        for (int k = 0; k < 7; k++) {
            double x = vals[k];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            vals[k] = x;
        }
        const int np = __reduce_add_sync(0xffffffffu, a_pairs);
        if (lane == 0) {
            for (int k = 0; k < 7; k++) s_part[w][k] = vals[k];
            s_part[w][7] = 0.5 * (double)np;
        }
        __syncthreads();
        if (threadIdx.x < R_NSLOTS) {
            const int t = threadIdx.x;
            double s = 0.0;
            int src = -1;
            if (t == R_ULJ) src = 0;
            else if (t >= R_W0 && t <= R_W5) src = 1 + t - R_W0;
            else if (t == R_PAIRS) src = 7;
            if (src >= 0)
                for (int k = 0; k < kPcWarps; k++) s += s_part[k][src];
            p.partials[(size_t)blockIdx.x * R_NSLOTS + t] = s;
        }
    }
}

// blocks per home cell: enough blocks for about eight per SM when there are
// few cells, at most one warp per home site of a mean cell (a block stages the
// whole neighbourhood, so more parts than that only repeat the staging)
static int pair_cell_split(const Engine &e) {
    const double mean = (double)e.n / (double)e.g.ncell;
    const int most = std::max(1, (int)(mean / kPcWarps + 0.999));
    const int want = (e.num_sms * 8 + e.g.ncell - 1) / e.g.ncell;
    return std::max(1, std::min(most, want));
}
int pair_cell_grid(const Engine &e) { return e.g.ncell * pair_cell_split(e); }

template <typename Real, bool M, bool E>
static void dispatch_lj(const PairParams &p, bool fene, int grid, int split, cudaStream_t st) {
    if (fene) k_pair_cell<Real, PC_LJ, M, E, true><<<grid, 32 * kPcWarps, 0, st>>>(p, PairTable{}, split);
    else k_pair_cell<Real, PC_LJ, M, E, false><<<grid, 32 * kPcWarps, 0, st>>>(p, PairTable{}, split);
}

// returns the number of blocks (rows of partial sums when measuring)
int launch_pair_cell(Engine &e, const PairParams &p, bool measure, bool emit, bool fene, cudaStream_t st) {
    const int split = pair_cell_split(e), grid = pair_cell_grid(e);
    const bool d = e.cfg.precision == KOMD_FP64;
    if (measure) {
        if (emit) d ? dispatch_lj<double, true, true>(p, fene, grid, split, st) : dispatch_lj<float, true, true>(p, fene, grid, split, st);
        else d ? dispatch_lj<double, true, false>(p, fene, grid, split, st) : dispatch_lj<float, true, false>(p, fene, grid, split, st);
    } else {
        if (emit) d ? dispatch_lj<double, false, true>(p, fene, grid, split, st) : dispatch_lj<float, false, true>(p, fene, grid, split, st);
        else d ? dispatch_lj<double, false, false>(p, fene, grid, split, st) : dispatch_lj<float, false, false>(p, fene, grid, split, st);
    }
    return grid;
}

// per-site LJ partner counts (exact FP64 arithmetic)
void launch_counts(Engine &e, cudaStream_t st) {
    PairParams p = pair_params(e);
    p.scan2 = p.rc2;
    p.pre2 = pair_pre2(e.g, p.scan2);
    k_pair_cell<double, PC_COUNT, false, false, false><<<pair_cell_grid(e), 32 * kPcWarps, 0, st>>>(
        p, PairTable{}, pair_cell_split(e));
}

// the tabulated force of every pair inside the cutoff (no same-molecule exclusion), added to f
void launch_pair_table(Engine &e, cudaStream_t st) {
    if (!e.tab_x || !e.tab_s || e.tab_n < 2) return;
    PairParams p = pair_params(e);
    p.scan2 = p.rc2;
    p.pre2 = pair_pre2(e.g, p.scan2);
    const PairTable t{e.tab_n, e.tab_x, e.tab_y, e.tab_s, e.tab_lo, e.tab_hi};
    k_pair_cell<double, PC_TABLE, false, false, false><<<pair_cell_grid(e), 32 * kPcWarps, 0, st>>>(
        p, t, pair_cell_split(e));
}

}  // namespace komd
