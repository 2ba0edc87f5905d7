// pair_tile.cu -- the FP32 pair kernel of the hot path: LJ 12-6 forces
// (LJ12_6.cpp:15-43), energy and virial, and the ATM neighbour list inside
// cutoff_3b, for one home cell per CTA.
//
//   1. threads 0..26 resolve the 27 neighbour cells (periodic wrap) and their
//      home-relative offsets from a per-dimension FP32 table computed once in
//      FP64 on the host, so no FP64 instruction runs in this kernel;
//   2. the neighbourhood's sites are staged in shared memory in home-cell
//      coordinates (float4 position + slot, key, cell code, sqrt(eps));
//   3. every warp owns a subset of home sites; for a home site the 32 lanes
//      test 32 staged candidates at a time and ballot-compact the hits into a
//      per-warp queue, so the force arithmetic always runs on full warps;
//   4. each dequeued pair adds its LJ force to the home site's shared-memory
//      accumulator and, inside cutoff_3b, appends (r_i - r_j, code) to the
//      home site's ATM list in queue order (deterministic list order).
// The lanes of a site are found by a ballot of the places where the site changes, and
// the candidates of the last 32 that are not there are out of reach instead of
// masked: 32,000 sites of liquid argon 44 -> 34.5 us.  Emptying the queue at each site, its
// force in the lanes' registers, takes 33 us, but sums in another order: snapshots
// for training then differ in their last bits, which BF16 roundings amplify.
// Full shell: each site's force is summed by its own CTA, no global atomics.
//
// The Verlet path (skin > 0) has its own kernels here: the list build
// (k_vlist_build, rebuild steps only), the LJ pass over each site's list row
// (k_lj_vlist) and the LJ pass that sweeps each site's ATM triplets from
// shared memory (k_lj_atm).
#include "engine.cuh"
#include "kernels.cuh"
#include "atm_device.cuh"

namespace komd {

constexpr int kTileWarps = 4;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kStage = 640;   // staged neighbour sites per round (more rounds if a neighbourhood is larger)
constexpr int kHome = 64;     // home sites per round
constexpr int kQ = 64;        // per-warp hit queue

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// neighbour nb (dx fastest) of domain cell (cx, cy, cz), wrapped; integer only
__device__ __forceinline__ int nb_cell(const Grid &g, int cx, int cy, int cz, int nb, int &kx, int &ky, int &kz,
                                       bool &crosses) {
    kx = cx + nb % 3 - 1;
    ky = cy + (nb / 3) % 3 - 1;
    kz = cz + nb / 9 - 1;
    crosses = false;
    if (kx < 0) { kx += g.nd[0]; crosses = true; } else if (kx >= g.nd[0]) { kx -= g.nd[0]; crosses = true; }
    if (ky < 0) { ky += g.nd[1]; crosses = true; } else if (ky >= g.nd[1]) { ky -= g.nd[1]; crosses = true; }
    if (kz < 0) { kz += g.nd[2]; crosses = true; } else if (kz >= g.nd[2]) { kz -= g.nd[2]; crosses = true; }
    return kx + g.nd[0] * (ky + g.nd[1] * kz);
}

template <bool MEASURE, bool EMIT>
__global__ void __launch_bounds__(kTileThreads) k_pair_tile(PairParams p) {
    pdl_wait();
    __shared__ float4 s_pos[kStage];
    __shared__ int4 s_aux[kStage];        // slot, key, code (nb | crosses << 5), sqrt(eps) bits
    __shared__ float4 s_hpos[kHome];
    __shared__ int2 s_haux[kHome];        // key, sqrt(eps) bits
    __shared__ float s_f[kHome * 3];
    __shared__ int s_cnt[kHome];
    __shared__ unsigned s_q[kTileWarps][kQ];
    __shared__ int s_nbs[27], s_nbn[27], s_nbpre[28], s_nbc[27];
    __shared__ float s_nbo[27][3];
    __shared__ double s_part[kTileWarps][8];

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int cell = blockIdx.x;
    int cx, cy, cz;
    cell_coords(p.g, cell, cx, cy, cz);
    if (tid < 27) {
        int kx, ky, kz;
        bool cr;
        const int c = nb_cell(p.g, cx, cy, cz, tid, kx, ky, kz, cr);
        const int s0 = p.cell_start[c];
        s_nbs[tid] = s0;
        s_nbn[tid] = p.cell_start[c + 1] - s0;
        s_nbc[tid] = cr ? 32 : 0;
        // home-relative offset of the neighbour cell's centre (FP32 table, per dimension)
        s_nbo[tid][0] = p.offtab[cx * 3 + tid % 3];
        s_nbo[tid][1] = p.offtab[p.g.nd[0] * 3 + cy * 3 + (tid / 3) % 3];
        s_nbo[tid][2] = p.offtab[(p.g.nd[0] + p.g.nd[1]) * 3 + cz * 3 + tid / 9];
    }
    __syncthreads();
    if (tid == 0) {
        int acc = 0;
        for (int k = 0; k < 27; k++) { s_nbpre[k] = acc; acc += s_nbn[k]; }
        s_nbpre[27] = acc;
    }
    __syncthreads();
    const int Nn = s_nbpre[27];
    const int hs = s_nbs[13], hn = s_nbn[13];
    const float rc2 = (float)p.rc2, rc3sq = (float)p.rc3sq, scan2 = (float)p.scan2;
    float4 *nl = p.nl;
    float m_u = 0.f, m_pairs = 0.f, m_w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // per-lane partials (MEASURE)
    const unsigned lt = lanemask_lt();

    for (int hb = 0; hb < hn; hb += kHome) {
        const int hc = min(kHome, hn - hb);
        for (int t = tid; t < hc; t += kTileThreads) {
            s_hpos[t] = p.pos4[hs + hb + t];
            s_haux[t] = make_int2(p.skey[hs + hb + t], __float_as_int(p.seps[hs + hb + t]));
            s_f[3 * t] = 0.f; s_f[3 * t + 1] = 0.f; s_f[3 * t + 2] = 0.f;
            s_cnt[t] = 0;
        }
        const int self_base = s_nbpre[13] + hb;
        for (int sb = 0; sb < Nn; sb += kStage) {
            const int ns = min(kStage, Nn - sb);
            __syncthreads();
            for (int t = tid; t < ns; t += kTileThreads) {
                const int gi = sb + t;
                int lo = 0, hi = 27;            // largest nb with s_nbpre[nb] <= gi
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (s_nbpre[mid] <= gi) lo = mid; else hi = mid;
                }
                const int nb = lo;
                const int j = s_nbs[nb] + (gi - s_nbpre[nb]);
                float4 q = p.pos4[j];
                q.x += s_nbo[nb][0];
                q.y += s_nbo[nb][1];
                q.z += s_nbo[nb][2];
                s_pos[t] = q;
                s_aux[t] = make_int4(j, p.skey[j], nb | s_nbc[nb], __float_as_int(p.seps[j]));
            }
            if (ns + tid < ((ns + 31) & ~31)) s_pos[ns + tid] = make_float4(1e15f, 1e15f, 1e15f, 0.f);   // out of reach
            __syncthreads();

            // Process one queued pair per lane (valid = lane holds an entry).
            // Entries of one home site occupy contiguous lanes (the queue is
            // filled site by site), and a site belongs to exactly one warp:
            // its force is reduced over its lane group and added by the
            // group's first lane with a plain read-modify-write.
            auto process = [&](unsigned e, bool valid) {
                const int i = valid ? (int)(e >> 16) : 0;
                const int j = valid ? (int)(e & 0xffffu) : 0;
                const float4 pi = s_hpos[i];
                const float4 pj = s_pos[j];
                const int4 a = s_aux[j];
                const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                // the lane's group [first, last]: entries of a site are neighbours in the queue
                const int site = valid ? i : (0x10000 | lane);
                const int before = __shfl_up_sync(0xffffffffu, site, 1);
                const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != site);
                const unsigned upto = lt | (1u << lane), after = heads & ~upto;
                const int first = 31 - __clz(heads & upto), last = after ? __ffs(after) - 2 : 31;
                float fx = 0.f, fy = 0.f, fz = 0.f;
                if (p.use_lj && valid && r2 <= rc2 && s_haux[i].x != a.y) {
                    const float inv = rcp_approx(r2);
                    const float sg = pi.w + pj.w;
                    const float x = sg * sg * inv;
                    const float lj6 = x * x * x;
                    const float ee = __int_as_float(s_haux[i].y) * __int_as_float(a.w);
                    const float ljd = 24.0f * ee * (2.0f * lj6 * lj6 - lj6);
                    const float fac = MEASURE ? ljd * inv : ljd * inv * p.lj_fscalef;   // ATM2B factor
                    fx = dx * fac; fy = dy * fac; fz = dz * fac;
                    if (MEASURE) {
                        const float wt = (p.virial_compat && (a.z & 32)) ? 1.0f : 0.5f;
                        m_u += 2.0f * ee * (lj6 * lj6 - lj6);       // half of 4 eps (s12 - s6) per visit
                        m_pairs += 0.5f;
                        m_w[0] += wt * dx * fx;
                        m_w[1] += wt * 0.5f * (dx * fy + dy * fx);
                        m_w[2] += wt * dy * fy;
                        m_w[3] += wt * 0.5f * (dx * fz + dz * fx);
                        m_w[4] += wt * 0.5f * (dy * fz + dz * fy);
                        m_w[5] += wt * dz * fz;
                    }
                }
                for (int o = 1; o < 32; o <<= 1) {
                    const float yx = __shfl_down_sync(0xffffffffu, fx, o);
                    const float yy = __shfl_down_sync(0xffffffffu, fy, o);
                    const float yz = __shfl_down_sync(0xffffffffu, fz, o);
                    if (lane + o <= last) { fx += yx; fy += yy; fz += yz; }
                }
                const bool emit = EMIT && valid && r2 <= rc3sq;
                const unsigned em = __ballot_sync(0xffffffffu, emit) & (0xffffffffu << first) & (0xffffffffu >> (31 - last));
                int base = 0;
                if (EMIT && valid && lane == first) base = s_cnt[i];
                base = __shfl_sync(0xffffffffu, base, first);
                if (valid && lane == first) {
                    s_f[3 * i] += fx;
                    s_f[3 * i + 1] += fy;
                    s_f[3 * i + 2] += fz;
                    if (EMIT) s_cnt[i] = base + __popc(em);
                }
                if (emit) {
                    const int c = base + __popc(em & lt);
                    const int slot_i = hs + hb + i;
                    if (c < p.nl_cap)
                        nl[(size_t)slot_i * p.nl_cap + c] = make_float4(dx, dy, dz, __int_as_float(a.z | (a.x << 6)));
                }
                __syncwarp();
            };

            int qn = 0;
            for (int i = w; i < hc; i += kTileWarps) {
                const float4 pi = s_hpos[i];
                const int self = self_base + i - sb;
                for (int j0 = 0; j0 < ns; j0 += 32) {
                    const int j = j0 + lane;
                    const float4 pj = s_pos[j];
                    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                    const bool hit = dx * dx + dy * dy + dz * dz <= scan2 && j != self;
                    const unsigned m = __ballot_sync(0xffffffffu, hit);
                    if (hit) s_q[w][qn + __popc(m & lt)] = ((unsigned)i << 16) | (unsigned)j;
                    qn += __popc(m);
                    if (qn >= 32) {
                        __syncwarp();
                        const unsigned e = s_q[w][lane];
                        const unsigned tail = (lane < qn - 32) ? s_q[w][lane + 32] : 0u;
                        __syncwarp();
                        if (lane < qn - 32) s_q[w][lane] = tail;
                        __syncwarp();
                        qn -= 32;
                        process(e, true);
                    }
                }
            }
            __syncwarp();
            if (qn > 0) {
                const unsigned e = (lane < qn) ? s_q[w][lane] : 0u;
                __syncwarp();
                process(e, lane < qn);
            }
        }
        __syncthreads();
        for (int t = tid; t < hc; t += kTileThreads) {
            const int slot = hs + hb + t;
            const int site = p.slot_site[slot];
            p.f[3 * site] = (double)s_f[3 * t];
            p.f[3 * site + 1] = (double)s_f[3 * t + 1];
            p.f[3 * site + 2] = (double)s_f[3 * t + 2];
            if (EMIT) {
                const int c = s_cnt[t];
                p.nl_count[slot] = min(c, p.nl_cap);
                if (c > p.nl_cap) atomicOr(&p.err[E_ATM_OVERFLOW], 1);
            }
        }
        __syncthreads();
    }
    if (MEASURE) {
        // the lanes' FP32 partials summed over the warp in FP32 (a fixed tree:
        // GB300's FP64 pipe made an FP64 tree the bulk of this pass), FP64 from
        // the warp sums on
        float vals[8] = {m_u, m_w[0], m_w[1], m_w[2], m_w[3], m_w[4], m_w[5], m_pairs};
        for (int k = 0; k < 8; k++) {
            float x = vals[k];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            vals[k] = x;
        }
        if (lane == 0) for (int k = 0; k < 8; k++) s_part[w][k] = (double)vals[k];
        __syncthreads();
        if (tid < R_NSLOTS) {
            double s = 0.0;
            int src = -1;
            if (tid == R_ULJ) src = 0;
            else if (tid >= R_W0 && tid <= R_W5) src = 1 + tid - R_W0;
            else if (tid == R_PAIRS) src = 7;
            if (src >= 0)
                for (int k = 0; k < kTileWarps; k++) s += s_part[k][src];
            p.partials[(size_t)blockIdx.x * R_NSLOTS + tid] = s;
        }
    }
}

// ---------------------------------------------------------------------------
// Verlet list build (rebuild steps only).  Blocks of a resident grid take units
// -- part of a home cell's sites -- from a counter the scan resets (cells
// differ in cost, and steps without a rebuild launch few blocks).  A block
// stages the cell's 27-cell neighbourhood in shared memory, by neighbour cell
// then slot (1024 sites a round); each warp then tests the staged sites, 32 at
// a time, against up to four home sites at once (one shared read serves the
// four).  Lane t keeps the ballot of batch t, so the test loop is 9
// instructions a home and batch; the hits are then expanded from the lanes'
// words in order and appended 32 at a time, so that the append (order key,
// molecule key, row write) runs on full warps and row writes are contiguous.
// Rows hold the pairs inside cutoff + skin in
// staging order (deterministic); bit 31 marks a same-molecule pair (no LJ).
// A row has two regions: the neighbours above the site (vl_above: larger z
// at the rebuild, ties by slot) from the front, the others from the back
// (row[cap-1] downwards); the count word holds both (above | below << 16).
// The half-list force pass reads the front region alone, full-row readers
// both (vl_entry).
// Issue-bound (79 % issue activity, 232M instructions at 256k sites).  Against a
// warp per home cell with a lane per home site, a launch takes 247 us (320) at
// 256,000 sites and skin 0.6, 16 us (118; 216 cells left most SMs idle) at
// 4,000, and 565 us (1157) on 300,000 sites of molecules in cells of 4.8.
// Per-lane shares of the staged sites without ballots, and classifying the hits
// in the test loop, took 254 and 375 us at 256,000.
// ---------------------------------------------------------------------------
// the count word of a row (both regions clamped so that they never overlap)
__device__ __forceinline__ int vl_count_word(int chi, int clo, int cap) {
    const int a = min(chi, cap), b = min(clo, cap - a);
    return a | (b << 16);
}

// logical entry k of a full row (the front region, then the back region)
__device__ __forceinline__ int vl_entry(int k, int chi, int cap) { return k < chi ? k : cap - 1 - (k - chi); }

constexpr int kVbMaxWarps = 8;
constexpr int kVbRound = 1024;   // staged sites a round: a ballot word per lane and 32 sites
constexpr int kVbQueue = 256;    // hits expanded at a time per warp

// H home sites h0, h0 + 1, ... (those below h1) of one warp against the ns
// staged sites, and their rows
template <int H>
__device__ __forceinline__ void vb_homes(const PairParams &p, const float4 *s_p, const unsigned *s_w, short *s_q, int hs,
                                         int h0, int h1, int ns, int self0, bool first, bool last, float rl2, int lane,
                                         unsigned lt) {
    float hx[H], hy[H], hz[H];
    unsigned word[H];
#pragma unroll
    for (int k = 0; k < H; k++) {
        const float4 q = p.pos4[hs + min(h0 + k, h1 - 1)];
        hx[k] = q.x; hy[k] = q.y; hz[k] = q.z;
        word[k] = 0u;
    }
    const int nb = (ns + 31) >> 5;   // the staging is padded to whole batches with sites out of range
    for (int t = 0; t < nb; t++) {
        const float4 pj = s_p[32 * t + lane];
#pragma unroll
        for (int k = 0; k < H; k++) {
            const float ax = hx[k] - pj.x, ay = hy[k] - pj.y, az = hz[k] - pj.z;
            const unsigned m = __ballot_sync(0xffffffffu, ax * ax + ay * ay + az * az <= rl2);
            if (lane == t) word[k] = m;
        }
    }
#pragma unroll
    for (int k = 0; k < H; k++) {
        if (h0 + k >= h1) break;
        const int hslot = hs + h0 + k;
        const int self = self0 + h0 + k;   // the site itself, if it is staged in this round
        unsigned m = word[k];
        if ((self >> 5) == lane && self >= 0) m &= ~(1u << (self & 31));
        const int zi = p.zkey[hslot], hkey = p.skey[hslot];
        unsigned *row = p.vl + (size_t)hslot * p.vl_cap;
        int chi = 0, clo = 0;   // run on over the rounds
        if (!first) {
            const int cw = p.vl_count[hslot];
            chi = cw & 0xffff;
            clo = cw >> 16;
        }
        const int mine = __popc(m);
        int off = mine;   // exclusive prefix of the lanes' hits
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += y;
        }
        const int hits = __shfl_sync(0xffffffffu, off, 31);
        off -= mine;
        for (int q0 = 0; q0 < hits; q0 += kVbQueue) {   // one trip unless a round holds more hits
            const int qe = min(hits, q0 + kVbQueue);
            __syncwarp();
            while (m && off < qe) {
                s_q[off - q0] = (short)(32 * lane + __ffs(m) - 1);
                m &= m - 1;
                off++;
            }
            __syncwarp();
            for (int c0 = q0; c0 < qe; c0 += 32) {
                const bool valid = c0 + lane < qe;
                unsigned wd = 0;
                bool up = false;
                if (valid) {
                    const int c = s_q[c0 - q0 + lane];
                    wd = s_w[c];
                    const unsigned j = wd & 0x3ffffffu;
                    up = vl_above(zi, __float_as_int(s_p[c].w), (unsigned)hslot, j);
                    if (p.multi_key && p.skey[j] == hkey) wd |= 0x80000000u;
                }
                const unsigned mu = __ballot_sync(0xffffffffu, valid && up);
                const unsigned md = __ballot_sync(0xffffffffu, valid && !up);
                // a full row drops hits and the counts still grow: flagged below
                const int at = up ? chi + __popc(mu & lt) : clo + __popc(md & lt);
                if (valid && at < p.vl_cap) row[up ? at : p.vl_cap - 1 - at] = wd;
                chi += __popc(mu);
                clo += __popc(md);
            }
        }
        if (lane == 0) {
            if (last) {
                p.vl_count[hslot] = vl_count_word(chi, clo, p.vl_cap);
                if (chi + clo > p.vl_cap) atomicOr(&p.err[E_VL_OVERFLOW], 1);
            } else {   // past 0x7fff the row has overflowed already
                p.vl_count[hslot] = min(chi, 0x7fff) | (min(clo, 0x7fff) << 16);
            }
        }
    }
    __syncwarp();
}

__device__ __forceinline__ void vlist_build_body(const PairParams &p, const VbShape &shape, int bid) {
    extern __shared__ float4 s_dyn[];
    __shared__ int s_st[27], s_pre[28];
    __shared__ short s_q[kVbMaxWarps][kVbQueue];
    __shared__ int s_unit;
    if (!*p.rebuild) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const unsigned lt = lanemask_lt();
    if (bid == 0 && threadIdx.x == 0 && p.rebuild_count) atomicAdd(p.rebuild_count, 1);
    const float rl2 = (float)p.rl2;
    const int stage = shape.stage, split = shape.split;
    float4 *s_p = s_dyn;                                            // position in the home cell's frame, order key
    unsigned *s_w = reinterpret_cast<unsigned *>(s_dyn + stage);    // list word without the same-molecule bit
    for (;;) {
        __syncthreads();   // the previous unit's shared data is read to the end
        if (threadIdx.x == 0) s_unit = atomicAdd(p.vb_next, 1);
        __syncthreads();
        const int unit = s_unit;
        if (unit < 0 || unit >= p.g.ncell * split) break;
        const int cell = unit / split, part = unit - cell * split;
        if (w == 0) {
            int cx, cy, cz, cnt = 0;
            cell_coords(p.g, cell, cx, cy, cz);
            if (lane < 27) {
                int kx, ky, kz;
                bool cr;
                const int q = nb_cell(p.g, cx, cy, cz, lane, kx, ky, kz, cr);
                const int s0 = p.cell_start[q];
                cnt = p.cell_start[q + 1] - s0;
                s_st[lane] = s0;
            }
            int inc = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane < 27) s_pre[lane] = inc - cnt;
            if (lane == 26) s_pre[27] = inc;
        }
        __syncthreads();
        const int hs = s_st[13], hn = s_pre[14] - s_pre[13];   // neighbour 13 is the home cell
        // this unit's homes, in contiguous shares of the warps
        const int u0 = (int)((long long)hn * part / split), u1 = (int)((long long)hn * (part + 1) / split);
        const int w0 = u0 + (u1 - u0) * w / warps, w1 = u0 + (u1 - u0) * (w + 1) / warps;
        const int total = u1 > u0 ? s_pre[27] : 0;
        for (int sb = 0; sb < total; sb += stage) {
            const int ns = min(stage, total - sb);
            if (sb > 0) __syncthreads();
            for (int nb = w; nb < 27; nb += warps) {   // a neighbour cell per warp
                const int s0 = s_st[nb], t0 = s_pre[nb] - sb;
                const int k0 = max(0, -t0), k1 = min(s_pre[nb + 1] - s_pre[nb], ns - t0);
                if (k0 >= k1) continue;
                const float4 o = p.nboff[(size_t)cell * 27 + nb];
                for (int k = k0 + lane; k < k1; k += 32) {
                    const int j = s0 + k;
                    const float4 q = p.pos4[j];
                    s_p[t0 + k] = make_float4(q.x + o.x, q.y + o.y, q.z + o.z, __int_as_float(p.zkey[j]));
                    s_w[t0 + k] = ((unsigned)nb << 26) | (unsigned)j;
                }
            }
            for (int t = ns + threadIdx.x; t < ((ns + 31) & ~31); t += blockDim.x)   // out of range of every home
                s_p[t] = make_float4(1e30f, 1e30f, 1e30f, 0.f);
            __syncthreads();
            const bool first = sb == 0, last = sb + stage >= total;
            const int self0 = s_pre[13] - sb;
            for (int h = w0; h < w1;) {
                const int rem = w1 - h;
                if (rem >= 3) {
                    vb_homes<4>(p, s_p, s_w, s_q[w], hs, h, w1, ns, self0, first, last, rl2, lane, lt);
                    h += 4;
                } else {
                    vb_homes<2>(p, s_p, s_w, s_q[w], hs, h, w1, ns, self0, first, last, rl2, lane, lt);
                    h += 2;
                }
            }
        }
    }
}
__global__ void __launch_bounds__(32 * kVbMaxWarps) k_vlist_build(PairParams p, VbShape shape) {
    pdl_trigger();
    pdl_wait();
    vlist_build_body(p, shape, blockIdx.x);
}

// ---------------------------------------------------------------------------
// LJ forces from the Verlet list (every step of the Verlet path): one warp
// per site, one list entry per lane; the neighbour's position is its FP32
// cell-local position plus the build-cell offset of the entry's neighbour
// cell.  Inside cutoff_3b the pair is appended to the ATM list in list
// order.  No atomics: the warp owns its site.
// ---------------------------------------------------------------------------
// The LJ pass over site i's Verlet row (one warp, lanes over the entries):
// the site's LJ force to f, and inside cutoff_3b the pair appended to the ATM
// list in list order -- to the global list, or (TO_SMEM) staged in shared
// memory (se, sq) for the sweep that follows in the same warp.  Returns the
// number of ATM neighbours kept.
// U = list entries per lane in flight (independent loads for latency hiding)
// W = lanes of the site: with 16 the warp holds two sites (live: this one is there), and
// odd entries have sums of their own, (hx, hy, hz): those of lanes 16 to 31 with W = 32
template <bool MEASURE, bool EMIT, bool UNIFORM, int U, bool TO_SMEM, int W = 32>
__device__ __forceinline__ int lj_site(const PairParams &p, int i, bool live, int lane, unsigned lt, float rc2,
                                       float rc3sq, float4 *se, float4 *sq, float &m_u, float &m_pairs,
                                       float (&m_w)[6]) {
    static_assert(W == 32 || (W == 16 && !MEASURE && !TO_SMEM && U % 2 == 0), "");
    const int sub = lane & (W - 1);
    const int cw = live ? p.vl_count[i] : 0;
    const int chi = cw & 0xffff, cnt = chi + (cw >> 16);   // both regions of the row
    const int cmax = W == 32 ? cnt : max(cnt, __shfl_xor_sync(0xffffffffu, cnt, 16));
    const float4 pi = p.pos4[i];
    const float sei = UNIFORM ? 0.f : p.seps[i];
    const float4 *off = p.nboff + (size_t)p.slot_cell[i] * 27;
    const unsigned *row = p.vl + (size_t)i * p.vl_cap;
    const float sg2u = p.sig0 * p.sig0, eeu = p.eps0;
    float fx = 0.f, fy = 0.f, fz = 0.f, hx = 0.f, hy = 0.f, hz = 0.f;
    int c_atm = 0;
    const unsigned half = W == 32 ? 0xffffffffu : (lane < 16 ? 0xffffu : 0xffff0000u);
    constexpr bool kAhead = W == 16;   // list entries read one pass ahead
    unsigned en[U];
    if (kAhead) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = u * W + sub;
            en[u] = k < cnt ? __ldcs(row + vl_entry(k, chi, p.vl_cap)) : 0xffffffffu;
        }
    }
    for (int k0 = 0; k0 < cmax; k0 += W * U) {
        unsigned e[U];
        float4 o[U], pj[U];
        float sej[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + (kAhead ? W * U : 0) + u * W + sub;
            if (kAhead) e[u] = en[u];
            // read once per step: evict first
            (kAhead ? en[u] : e[u]) = k < cnt ? __ldcs(row + vl_entry(k, chi, p.vl_cap)) : 0xffffffffu;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned x = e[u] != 0xffffffffu ? e[u] : 0u;   // slot 0 and its site's own cell: read, not used
            o[u] = off[(x >> 26) & 31u];
            pj[u] = p.pos4[x & 0x3ffffffu];
            if (!UNIFORM) sej[u] = p.seps[x & 0x3ffffffu];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool valid = e[u] != 0xffffffffu;
            const float dx = pi.x - (pj[u].x + o[u].x), dy = pi.y - (pj[u].y + o[u].y), dz = pi.z - (pj[u].z + o[u].z);
            // the roundings written out: left to the compiler they differ between the forms
            const float r2 = valid ? fmaf(dz, dz, fmaf(dx, dx, dy * dy)) : 1e30f;
            const bool lj = p.use_lj && r2 <= rc2 && !(e[u] >> 31);
            const float inv = rcp_approx(r2);
            float x, ee;
            if (UNIFORM) {
                x = sg2u * inv;
                ee = eeu;
            } else {
                const float sg = pi.w + pj[u].w;
                x = sg * sg * inv;
                ee = sei * sej[u];
            }
            const float lj6 = x * x * x;
            float fac0 = 24.0f * ee * fmaf(2.0f * lj6, lj6, -lj6) * inv;
            float usw = 1.0f;
            if (p.sw) {   // switched cutoff: U S, force fac S - 2 U dS/dx
                float dS;
                sw_eval(r2, p.sw_rc2, p.sw_iw, usw, dS);
                fac0 = fac0 * usw - 8.0f * ee * (lj6 * lj6 - lj6) * dS;
            }
            if (!MEASURE) fac0 *= p.lj_fscalef;   // ATM2B factor
            // no branch around a dozen instructions; both factors are dropped, so that a
            // position that is not finite reaches nobody else
            const float fac = lj ? fac0 : 0.f;
            const float ex = lj ? dx : 0.f, ey = lj ? dy : 0.f, ez = lj ? dz : 0.f;
            if (W == 32 || (u & 1) == 0) {
                fx = fmaf(ex, fac, fx); fy = fmaf(ey, fac, fy); fz = fmaf(ez, fac, fz);
            } else {
                hx = fmaf(ex, fac, hx); hy = fmaf(ey, fac, hy); hz = fmaf(ez, fac, hz);
            }
            if (MEASURE && lj) {
                const float gx = dx * fac, gy = dy * fac, gz = dz * fac;
                m_u += 2.0f * ee * (lj6 * lj6 - lj6) * usw;
                m_pairs += 0.5f;
                m_w[0] += 0.5f * dx * gx;
                m_w[1] += 0.25f * (dx * gy + dy * gx);
                m_w[2] += 0.5f * dy * gy;
                m_w[3] += 0.25f * (dx * gz + dz * gx);
                m_w[4] += 0.25f * (dy * gz + dz * gy);
                m_w[5] += 0.5f * dz * gz;
            }
            if (EMIT) {
                // staged for the once-per-triplet sweep: neighbours above i only
                const bool emit = valid && r2 <= rc3sq && (!TO_SMEM || (int)(e[u] & 0x3ffffffu) > i);
                const unsigned m = __ballot_sync(0xffffffffu, emit) & half;
                if (emit) {
                    const int pos = c_atm + __popc(m & lt);
                    const int nb = (int)((e[u] >> 26) & 31u), j = (int)(e[u] & 0x3ffffffu);
                    const int code = nb | (o[u].w != 0.f ? 32 : 0) | (j << 6);
                    if (pos < p.nl_cap) {
                        const float4 entry = make_float4(dx, dy, dz, __int_as_float(code));
                        if (TO_SMEM) {   // staged as the sweep wants it: e and (A, 1/A, 1/sqrt A)
                            se[pos] = entry;
                            sq[pos] = atm_stage_q(r2);
                        } else {
                            p.nl[(size_t)i * p.nl_cap + pos] = entry;
                        }
                    }
                }
                c_atm += __popc(m);
            }
        }
    }
    // lanes 0, W/4 and W/2 of a site hold x, y and z: one FP32 -> FP64 conversion for
    // the three (a conversion takes the FP64 pipe for a whole warp, whatever the active lanes)
    if (W == 16) { fx += hx; fy += hy; fz += hz; }
    const float fs = warp_sum3<float, W>(fx, fy, fz, lane);
    if ((sub & (W / 4 - 1)) == 0 && sub < 3 * W / 4 && live)
        p.f[3 * (size_t)p.slot_site[i] + sub / (W / 4)] = (double)fs;
    if (EMIT && sub == 0 && live) {
        if (!TO_SMEM) p.nl_count[i] = min(c_atm, p.nl_cap);
        if (c_atm > p.nl_cap) atomicOr(&p.err[E_ATM_OVERFLOW], 1);
    }
    return min(c_atm, p.nl_cap);
}

template <bool MEASURE, bool EMIT, bool UNIFORM, int U>
__global__ void __launch_bounds__(256, U == 3 ? 4 : 5) k_lj_vlist(PairParams p, int n, int per) {
    pdl_wait();
    __shared__ double s_part[8][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float rc2 = p.rc2f, rc3sq = p.rc3sqf;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.rebuild_done) *p.rebuild_done = 0;
    float m_u = 0.f, m_pairs = 0.f, m_w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // each block walks `per` consecutive groups of 8 slots: neighbouring slots share
    // most of their neighbours, so the gathers of one group hit L1 lines of the last
    for (int it = 0; it < per; it++) {
        const int i = (blockIdx.x * per + it) * 8 + w;
        if (i < n)
            lj_site<MEASURE, EMIT, UNIFORM, U, false>(p, i, true, lane, lt, rc2, rc3sq, nullptr, nullptr, m_u, m_pairs,
                                                      m_w);
    }
    if (MEASURE) {
        // the lanes' FP32 partials summed over the warp in FP32 (a fixed tree:
        // GB300's FP64 pipe made an FP64 tree the bulk of this pass), FP64 from
        // the warp sums on
        float vals[8] = {m_u, m_w[0], m_w[1], m_w[2], m_w[3], m_w[4], m_w[5], m_pairs};
        for (int k = 0; k < 8; k++) {
            float x = vals[k];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            vals[k] = x;
        }
        if (lane == 0) for (int k = 0; k < 8; k++) s_part[w][k] = (double)vals[k];
        __syncthreads();
        const int tid = threadIdx.x;
        if (tid < R_NSLOTS) {
            double s = 0.0;
            int src = -1;
            if (tid == R_ULJ) src = 0;
            else if (tid >= R_W0 && tid <= R_W5) src = 1 + tid - R_W0;
            else if (tid == R_PAIRS) src = 7;
            if (src >= 0)
                for (int k = 0; k < 8; k++) s += s_part[k][src];
            p.partials[(size_t)blockIdx.x * R_NSLOTS + tid] = s;
        }
    }
}

// The same with two sites a warp, sixteen lanes each.  The pass waits on its gathers
// (with one site a warp and three entries a lane in flight: half of the issue slots, 40 %
// of the L1 wavefronts), so what counts is how many sites are in flight and how little
// each costs: a row of 74 entries takes five passes of 16 lanes where 32 lanes take 96
// entries' worth, the reduction and the conversion to FP64 serve two sites, two entries
// a lane in flight with the next two list entries read ahead fit in 48 registers (five
// blocks an SM, not four).  A lane sums entries of equal place modulo 32 apart, so
// every force is that of the kernel above bit for bit.  300,000 sites of three-site
// molecules: 135 -> 90 us, and 86 with selects for the branches around a pair's
// arithmetic; 32,000 sites of liquid argon with the ATM list 25.4 -> 18.8 -> 17.6.
// Without the read-ahead 99, four entries in flight 119, six 132 us.
template <bool EMIT, bool UNIFORM>
__global__ void __launch_bounds__(256, 5) k_lj_vlist2(PairParams p, int n, int per) {
    pdl_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float rc2 = p.rc2f, rc3sq = p.rc3sqf;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.rebuild_done) *p.rebuild_done = 0;
    float m_u, m_pairs, m_w[6];   // no sensors
    for (int it = 0; it < per; it++) {
        const int i0 = ((blockIdx.x * per + it) * 8 + w) * 2, i = i0 + (lane >> 4);
        if (i0 >= n) return;
        lj_site<false, EMIT, UNIFORM, 2, false, 16>(p, min(i, n - 1), i < n, lane, lt, rc2, rc3sq, nullptr, nullptr,
                                                    m_u, m_pairs, m_w);
    }
}

// LJ and ATM in one pass (FP32 forces, FULL triplets, Verlet path): each warp
// runs the LJ pass of its site, stages the site's ATM neighbours above it in
// shared memory instead of the global list, and sweeps its triplets at once.
// Warps in their latency-bound LJ phase and warps in their issue-bound sweep
// share each SM, and the ATM list never goes to memory.  The arithmetic and
// the order of every sum are those of k_lj_vlist + k_atm_s.
template <bool UNIFORM, int U>
__global__ void __launch_bounds__(256, 4) k_lj_atm(PairParams p, AtmParams a, int n, int per) {
    pdl_wait();
    extern __shared__ float4 s_dyn[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float4 *se = s_dyn + w * 2 * p.nl_cap, *sq = se + p.nl_cap;
    const float rc2 = p.rc2f, rc3sq = p.rc3sqf, rc3f = a.rc2f;
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.rebuild_done) *p.rebuild_done = 0;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    float m_u = 0.f, m_pairs = 0.f, m_w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int it = 0; it < per; it++) {
        const int i = (blockIdx.x * per + it) * 8 + w;
        if (i < n) {
            const int m = lj_site<false, true, UNIFORM, U, true>(p, i, true, lane, lt, rc2, rc3sq, se, sq, m_u, m_pairs, m_w);
            __syncwarp();
            atm_vertex(a, i, se, sq, m, lane, rc3f);
            __syncwarp();   // se / sq are refilled by the next site
        }
    }
}

// ---------------------------------------------------------------------------
// The half-list LJ + ATM pass (FP32 forces, FULL triplets, Verlet path, no
// Limit): each pair and each triplet is evaluated once, from its lowest
// member in the order vl_above.  One warp per site i walks the front region
// of i's row only (the neighbours above i, about half the row):
//   1. LJ: the force on i stays in the lanes' registers; the reaction on the
//      partner j is staged in shared memory (sr) beside the partner's slot;
//      partners inside cutoff_3b are staged for the triplet sweep as well
//      (se, sq, at the front of their arrays), LJ-only partners fill sr from
//      the back;
//   2. the triplet sweep of atm_vertex_shares leaves each ATM partner's share
//      in its owner lane;
//   3. each partner gets its LJ reaction plus its ATM share (in force units)
//      through ONE 64-bit fixed-point add per component -- integer sums, so
//      the result does not depend on the order in which warps add;
//   4. i's own force (its LJ sum plus its ATM share) is written to f; the
//      flush adds the fixed-point sums of the partners' contributions.
// Against the full-row pass this reads half the list, evaluates each LJ
// pair once instead of twice, and converts one FP32 partial per partner.
// Bound by instruction issue (81 % of the slots, 740 a site, 44 % of them the
// sweep): 256,000 sites of liquid argon at skin 0.6, 221 -> 195 us, from branches
// around a dozen instructions replaced by selects, reciprocal roots by PTX
// rsqrt.approx.ftz, a shorter fixed-point conversion and the cutoffs' FP32 values in
// the parameters (812 a site, 78 % before).  Five blocks an SM were slower (39 against
// 35 us at 31,000 sites), two sites a warp gained nothing.
// ---------------------------------------------------------------------------
// what the half-list pass reads of a site before its arithmetic: the count
// of its front region, the region's first 64 entries (rows hold vl_cap >= 64
// entries, so both reads stay inside the row; the count masks them, and the
// entries are read without waiting for it), its position and its cell.
// (Loading this one site ahead, during the previous site's sweep, was
// measured slower: the extra live registers spill at the 64-register bound.)
struct HalfRow {
    int cnt, cell;
    unsigned e0, e1;
    float4 pi;
};

__device__ __forceinline__ void half_row_load(const PairParams &p, int i, int lane, HalfRow &h) {
    const unsigned *row = p.vl + (size_t)i * p.vl_cap;
    h.cnt = p.vl_count[i] & 0xffff;   // the neighbours above i
    h.e0 = __ldcs(row + lane);        // read once per step: evict first
    h.e1 = __ldcs(row + 32 + lane);
    h.pi = p.pos4[i];
    h.cell = p.slot_cell[i];
}

// PLAIN: the LJ term is on with no ATM2B factor (use_lj = 1, lj_fscalef = 1),
// so neither is read per pair (the products are the same: a factor of 1 is exact)
template <bool UNIFORM, bool SW, bool PLAIN>
__device__ __forceinline__ void lj_half(const PairParams &p, int i, const HalfRow &h, int lane, unsigned lt, float rc2,
                                        float rc3sq, float4 *se, float4 *sq, float4 *sr, int capa, int capr,
                                        int &m_out, int &k_out, float &fx, float &fy, float &fz) {
    const int cnt = h.cnt;
    const float4 pi = h.pi;
    const float sei = UNIFORM ? 0.f : p.seps[i];
    const float4 *off = p.nboff + (size_t)h.cell * 27;
    const unsigned *row = p.vl + (size_t)i * p.vl_cap;
    const float sg2u = p.sig0 * p.sig0, eeu = p.eps0;
    fx = fy = fz = 0.f;
    int m = 0, k = 0;
    for (int k0 = 0; k0 < cnt; k0 += 64) {
        unsigned e[2];
        float4 o[2], pj[2];
        float sej[2];
        if (k0 == 0) {   // the first 64 entries, read with the count
            e[0] = lane < cnt ? h.e0 : 0xffffffffu;
            e[1] = 32 + lane < cnt ? h.e1 : 0xffffffffu;
        } else {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int kk = k0 + u * 32 + lane;
                e[u] = kk < cnt ? __ldcs(row + kk) : 0xffffffffu;
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const unsigned x = e[u] != 0xffffffffu ? e[u] : 0u;   // slot 0 and its site's own cell: read, not used
            o[u] = off[(x >> 26) & 31u];
            pj[u] = p.pos4[x & 0x3ffffffu];
            if (!UNIFORM) sej[u] = p.seps[x & 0x3ffffffu];
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const bool valid = e[u] != 0xffffffffu;
            const float dx = pi.x - (pj[u].x + o[u].x), dy = pi.y - (pj[u].y + o[u].y), dz = pi.z - (pj[u].z + o[u].z);
            const float r2 = valid ? dx * dx + dy * dy + dz * dz : 1e30f;
            const bool lj = (PLAIN || p.use_lj) && r2 <= rc2 && !(e[u] >> 31);
            const float inv = rcp_approx(r2);
            float x, ee;
            if (UNIFORM) {
                x = sg2u * inv;
                ee = eeu;
            } else {
                const float sg = pi.w + pj[u].w;
                x = sg * sg * inv;
                ee = sei * sej[u];
            }
            const float lj6 = x * x * x;
            float fac = 24.0f * ee * (2.0f * lj6 * lj6 - lj6) * inv;
            if (!PLAIN) fac *= p.lj_fscalef;   // ATM2B factor
            if (SW) {   // switched cutoff (no ATM2B with it): U S, force fac S - 2 U dS/dx
                float S, dS;
                sw_eval(r2, p.sw_rc2, p.sw_iw, S, dS);
                fac = fac * S - 8.0f * ee * (lj6 * lj6 - lj6) * dS;
            }
            // no branch around a dozen instructions; what does not count is dropped last, so
            // that a position that is not finite reaches nobody else
            const float gx = lj ? dx * fac : 0.f, gy = lj ? dy * fac : 0.f, gz = lj ? dz * fac : 0.f;
            fx += gx; fy += gy; fz += gz;
            const bool at = valid && r2 <= rc3sq;   // a triplet partner (LJ or not)
            const bool lo = lj && !at;              // an LJ-only partner
            const unsigned ma = __ballot_sync(0xffffffffu, at), ml = __ballot_sync(0xffffffffu, lo);
            const int pos = (at ? m : k) + __popc((at ? ma : ml) & lt);
            if ((at && pos < capa) || lo) {
                // the partner's slot j at bits 6-30 (j < 2^25 with ATM on): the list word
                // shifted past its cell and molecule bits.  This pass reads only
                // code >> 6 (the cell bits of atm_code are for the COMPAT filter)
                const int code = (int)(e[u] << 6);
                sr[at ? pos : capr - 1 - pos] = make_float4(-gx, -gy, -gz, __int_as_float(code));
                if (at) {
                    se[pos] = make_float4(dx, dy, dz, __int_as_float(code));
                    sq[pos] = atm_stage_q(r2);
                }
            }
            m += __popc(ma);
            k += __popc(ml);
        }
    }
    if (lane == 0 && m > capa) atomicOr(&p.err[E_ATM_OVERFLOW], 1);
    m_out = min(m, capa);
    k_out = k;
}

template <bool UNIFORM, bool SW, bool PLAIN>
__device__ __forceinline__ void lj_atm_half_body(const PairParams &p, const AtmParams &a, float sa, int n, int per,
                                                 int bid) {
    extern __shared__ float4 s_dyn[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int capa = p.nl_cap, capr = p.vl_cap;
    float4 *se = s_dyn + (size_t)w * (2 * capa + capr), *sq = se + capa, *sr = sq + capa;
    const float rc2 = p.rc2f, rc3sq = p.rc3sqf, rc3f = a.rc2f;
    const unsigned lt = lanemask_lt();
    if (bid == 0 && threadIdx.x == 0 && p.rebuild_done) *p.rebuild_done = 0;
    for (int it = 0; it < per; it++) {
        const int i = (bid * per + it) * 8 + w;
        if (i >= n) break;   // warp-uniform; later groups of this block are past n too
        HalfRow cur;
        half_row_load(p, i, lane, cur);
        int m, k;
        float fx, fy, fz;
        lj_half<UNIFORM, SW, PLAIN>(p, i, cur, lane, lt, rc2, rc3sq, se, sq, sr, capa, capr, m, k, fx, fy, fz);
        __syncwarp();
        float ax, ay, az, gx, gy, gz;
        atm_vertex_shares<SW>(a, se, sq, m, lane, rc3f, sa, ax, ay, az, gx, gy, gz);
        // every partner: LJ reaction + ATM share (force units), one fixed-point add per component
        const int tot = m + k;
        for (int L = lane; L < tot; L += 32) {
            const float4 rr = sr[L < m ? L : capr - 1 - (L - m)];
            float vx = rr.x, vy = rr.y, vz = rr.z;
            if (L == lane) {   // the first trip: lane L < 32 owns partner L's share (zero for m > 32)
                vx = fmaf(sa, ax, vx);
                vy = fmaf(sa, ay, vy);
                vz = fmaf(sa, az, vz);
            }
            unsigned long long *acc = a.acc + 3 * (size_t)(__float_as_int(rr.w) >> 6);
            // hardly a zero among them: added without a look
            atomicAdd(acc, (unsigned long long)fix32_rn(vx));
            atomicAdd(acc + 1, (unsigned long long)fix32_rn(vy));
            atomicAdd(acc + 2, (unsigned long long)fix32_rn(vz));
        }
        // the site's own force: its LJ sum and its ATM share
        fx = fmaf(sa, gx, fx);
        fy = fmaf(sa, gy, fy);
        fz = fmaf(sa, gz, fz);
        // the warp sums of (fx, fy, fz) by the butterfly over offsets 16, 8, 4, 2, 1,
        // the lanes splitting the components on the way: after offset 16 the lanes
        // below 16 carry x and y, the others z; after offset 8 lanes 0-7 carry x,
        // 8-15 y, 16-31 z.  Every sum pairs the same partial sums as a butterfly
        // per component (FP32 addition commutes), so the totals are bitwise those
        // of 15 shuffles, with 6.
        float c0;
        {
            const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
            const float r1 = __shfl_xor_sync(0xffffffffu, up16 ? fx : fz, 16);
            const float r2 = __shfl_xor_sync(0xffffffffu, fy, 16);
            c0 = (up16 ? fz : fx) + r1;   // z above 16, x below
            const float c1 = fy + r2;     // y below 16
            const float r3 = __shfl_xor_sync(0xffffffffu, (up16 || up8) ? c0 : c1, 8);
            c0 = ((up16 || !up8) ? c0 : c1) + r3;
            for (int o = 4; o > 0; o >>= 1) c0 += __shfl_xor_sync(0xffffffffu, c0, o);
        }
        if ((lane & 7) == 0) {   // lanes 0, 8, 16, 24: x, y, z and the slot's fourth word
            if (p.fown) {   // FP32 by slot, 16 bytes: the flush widens it (no FP64-pipe conversions here)
                reinterpret_cast<float *>(p.fown + i)[lane >> 3] = lane < 24 ? c0 : 0.f;
            } else if (lane < 24) {
                p.f[3 * (size_t)p.slot_site[i] + (lane >> 3)] = (double)c0;
            }
        }
        __syncwarp();   // se / sq / sr are refilled by the next site
    }
}
template <bool UNIFORM, bool SW, bool PLAIN>
__global__ void __launch_bounds__(256, 4) k_lj_atm_half(PairParams p, AtmParams a, float sa, int n, int per) {
    pdl_trigger();
    pdl_wait();
    lj_atm_half_body<UNIFORM, SW, PLAIN>(p, a, sa, n, per, blockIdx.x);
}

template <bool UNIFORM, bool SW, bool PLAIN = false>
static void launch_half(const PairParams &p, const AtmParams &a, float sa, int n, int per, int grid, size_t sm,
                        cudaStream_t st) {
    allow_smem((const void *)k_lj_atm_half<UNIFORM, SW, PLAIN>, sm);
    launch_pdl(k_lj_atm_half<UNIFORM, SW, PLAIN>, grid, 256, sm, st, p, a, sa, n, per);
}

// shared memory of the half-list pass: per warp nl_cap staged triplet
// partners (se, sq) and vl_cap partners' reactions (sr)
size_t lj_atm_half_smem(const Engine &e) {
    return (size_t)8 * sizeof(float4) * (2 * (size_t)e.nl_cap + (size_t)e.vl_cap);
}

// the half-list pass serves the step when nothing after the pair terms reads
// or clamps the force of a site before the flush (no Limit, no FENE, no
// tabulated term) and its staging fits the shared memory of four blocks
bool lj_atm_half(const Engine &e) {
    if (e.cfg.terms & (KOMD_TERM_LIMIT | KOMD_TERM_FENE | KOMD_TERM_TABULATED)) return false;
    return lj_atm_half_smem(e) <= 56 * 1024 || e.cfg.switch_width > 0;   // the switch runs here only
}

bool half_plain(const PairParams &p) { return p.use_lj && p.lj_fscalef == 1.0f; }

// the bonded terms add to f between the force pass and the flush, so with
// them the pass writes f itself
float4 *half_own(const Engine &e) { return (e.cfg.terms & KOMD_TERM_BONDED) ? nullptr : e.fown; }

int vlist_grid(const Engine &e) { return (int)((e.n + 7) / 8); }

// groups of 8 slots per block of the force pass: about eight resident waves of
// blocks (5 per SM), each over a contiguous range of slots
int vlist_per(const Engine &e) {
    const int groups = vlist_grid(e);
    const int target = e.num_sms * 5 * 8;
    return groups <= target ? 1 : (groups + target - 1) / target;
}

// blocks of the single-system passes over the slots (rows of partial sums when measuring)
int vlist_blocks(const Engine &e) {
    const int per = vlist_per(e);
    return (vlist_grid(e) + per - 1) / per;
}

// ---- packed replicas (kernels.cuh): the list build and the half-list pass of
// every replica in one launch each
__device__ __forceinline__ int packed_replica(const int *__restrict__ start, int nrep, int b) {
    int lo = 0, hi = nrep;   // start[0] = 0 <= b < start[nrep]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(32 * kVbMaxWarps) k_vlist_build_p(const PairParams *__restrict__ p, VbShape shape,
                                                                   const int *__restrict__ start, int nrep) {
    const int r = packed_replica(start, nrep, blockIdx.x);
    vlist_build_body(p[r], shape, blockIdx.x - start[r]);
}

template <bool UNIFORM, bool SW, bool PLAIN>
__global__ void __launch_bounds__(256, 4) k_lj_atm_half_p(const PairParams *__restrict__ p,
                                                          const AtmParams *__restrict__ a,
                                                          const float *__restrict__ sa, const int *__restrict__ n,
                                                          const int *__restrict__ per, const int *__restrict__ start,
                                                          int nrep) {
    const int r = packed_replica(start, nrep, blockIdx.x);
    lj_atm_half_body<UNIFORM, SW, PLAIN>(p[r], a[r], sa[r], n[r], per[r], blockIdx.x - start[r]);
}

template <bool UNIFORM, bool SW, bool PLAIN = false>
static void launch_half_p(const PackedStep &pk, cudaStream_t st) {
    allow_smem((const void *)k_lj_atm_half_p<UNIFORM, SW, PLAIN>, pk.force_smem);
    k_lj_atm_half_p<UNIFORM, SW, PLAIN><<<pk.force.blocks, 256, pk.force_smem, st>>>(pk.pp, pk.ap, pk.sa, pk.n,
                                                                                     pk.per, pk.force.start, pk.nrep);
}

void launch_packed_pair_stages(const PackedStep &pk, cudaStream_t st, bool vbuild) {
    if (vbuild) {
        // the force pass's shared-memory carve-out: an SM that runs one group's
        // list build beside another group's force pass would otherwise have to
        // drain to change it (48 replicas: 21.1 against 20.1 ms a pass)
        cudaFuncSetAttribute(k_vlist_build_p, cudaFuncAttributePreferredSharedMemoryCarveout, 72);
        k_vlist_build_p<<<pk.vbuild.blocks, 32 * pk.vb.warps, vb_smem(pk.vb), st>>>(pk.pp, pk.vb, pk.vbuild.start,
                                                                                    pk.nrep);
        return;
    }
    if (pk.sw) {
        if (pk.uniform) launch_half_p<true, true>(pk, st);
        else launch_half_p<false, true>(pk, st);
    } else {
        if (pk.uniform && pk.plain) launch_half_p<true, false, true>(pk, st);   // the benchmark's form
        else if (pk.uniform) launch_half_p<true, false>(pk, st);
        else launch_half_p<false, false>(pk, st);
    }
}

// The list build's shape for systems of up to `sites` sites per cell on average
// and `cells` cells in all: the staging holds a mean neighbourhood and a
// quarter, up to a round's 1024; eight warps where a cell keeps them busy, and
// parts of a cell's homes where the cells alone give fewer than six blocks per SM.
VbShape vb_shape(double sites, int64_t cells, int num_sms) {
    VbShape v;
    v.warps = sites >= 48.0 ? 8 : 4;
    v.stage = std::min(kVbRound, std::max(256, ((int)(27.0 * sites * 1.25) + 127) / 128 * 128));
    const int most = std::max(1, (int)(sites / v.warps + 0.999));
    const int64_t want = ((int64_t)num_sms * 6 + cells - 1) / std::max<int64_t>(cells, 1);
    v.split = (int)std::max<int64_t>(1, std::min<int64_t>(most, want));
    return v;
}
size_t vb_smem(const VbShape &v) { return (size_t)v.stage * (sizeof(float4) + sizeof(unsigned)); }

int packed_blocks_vbuild(const Engine &e) {
    // up to 256 blocks for a rebuilding replica; those of replicas without a
    // rebuild exit at once
    return std::max(1, std::min(e.g.ncell, 256));
}

void launch_vlist_build(Engine &e, cudaStream_t st) {
    PairParams p = pair_params(e);
    const VbShape v = vb_shape((double)e.n / e.g.ncell, e.g.ncell, e.num_sms);
    const int blocks = std::min(e.g.ncell * v.split, e.num_sms * 48 / v.warps);   // resident
    launch_pdl(k_vlist_build, blocks, 32 * v.warps, vb_smem(v), st, p, v);
}

template <bool UNIFORM>
static void lj_vlist_dispatch(PairParams &p, int n, int grid, int per, bool measure, bool emit, bool u3,
                              cudaStream_t st) {
    if (measure) {
        if (emit) launch_pdl(k_lj_vlist<true, true, UNIFORM, 2>, grid, 256, 0, st, p, n, per);
        else launch_pdl(k_lj_vlist<true, false, UNIFORM, 2>, grid, 256, 0, st, p, n, per);
    } else if (u3) {
        if (emit) launch_pdl(k_lj_vlist<false, true, UNIFORM, 3>, grid, 256, 0, st, p, n, per);
        else launch_pdl(k_lj_vlist<false, false, UNIFORM, 3>, grid, 256, 0, st, p, n, per);
    } else {
        if (emit) launch_pdl(k_lj_vlist<false, true, UNIFORM, 2>, grid, 256, 0, st, p, n, per);
        else launch_pdl(k_lj_vlist<false, false, UNIFORM, 2>, grid, 256, 0, st, p, n, per);
    }
}

// rows of at most 96 entries on average: one pass of 3 entries per lane
// instead of two of 2 (the row length is the number of sites within the
// list range, about density * 4/3 pi (cutoff + skin)^3)
bool vlist_u3(const Engine &e) {
    const double reach = std::max(e.cfg.cutoff, (e.cfg.terms & KOMD_TERM_ATM) ? e.cfg.cutoff_3b : 0.0) + e.cfg.skin;
    const double rho = (double)e.n / (e.g.L[0] * e.g.L[1] * e.g.L[2]);
    return rho * 4.18879020478639 * reach * reach * reach <= 88.0;
}

int launch_lj_vlist(Engine &e, PairParams &p, bool measure, bool emit, cudaStream_t st) {
    // two sites a warp once one site a warp (at most 32 warps an SM) takes more than one
    // wave: 4000 sites 11.4 us a step either way, 2048 10.9 against 11.4, 5324 14.0 against
    // 12.9, 16,384 19.5 against 16.9
    if (!measure && e.n > 32 * (int64_t)e.num_sms) {
        const int per2 = (vlist_per(e) + 1) / 2, grid2 = (int)((e.n + 16 * per2 - 1) / (16 * per2));
        auto k = e.uniform ? (emit ? k_lj_vlist2<true, true> : k_lj_vlist2<false, true>)
                           : (emit ? k_lj_vlist2<true, false> : k_lj_vlist2<false, false>);
        launch_pdl(k, grid2, 256, 0, st, p, (int)e.n, per2);
        return grid2;
    }
    // a block's partial sums cover all its groups (the lanes' sums run across them)
    const int per = vlist_per(e);
    const int grid = vlist_blocks(e);
    const bool u3 = vlist_u3(e);
    if (e.uniform) lj_vlist_dispatch<true>(p, (int)e.n, grid, per, measure, emit, u3, st);
    else lj_vlist_dispatch<false>(p, (int)e.n, grid, per, measure, emit, u3, st);
    return grid;
}

void launch_lj_atm(Engine &e, cudaStream_t st) {
    PairParams p = pair_params(e);
    const AtmParams a = atm_params(e);
    const int per = vlist_per(e);
    const int grid = vlist_blocks(e);
    if (lj_atm_half(e)) {
        const size_t sm = lj_atm_half_smem(e);
        const float sa = (float)(2.0 * a.sign * a.nu);   // share units (2 sign nu) to force units
        p.fown = half_own(e);
        if (p.sw) {
            if (e.uniform) launch_half<true, true>(p, a, sa, (int)e.n, per, grid, sm, st);
            else launch_half<false, true>(p, a, sa, (int)e.n, per, grid, sm, st);
        } else {
            if (e.uniform && half_plain(p)) launch_half<true, false, true>(p, a, sa, (int)e.n, per, grid, sm, st);
            else if (e.uniform) launch_half<true, false>(p, a, sa, (int)e.n, per, grid, sm, st);
            else launch_half<false, false>(p, a, sa, (int)e.n, per, grid, sm, st);
        }
        return;
    }
    const size_t sm = (size_t)8 * 2 * sizeof(float4) * (size_t)e.nl_cap;
    const bool u3 = vlist_u3(e);
    if (e.uniform) {
        if (u3) {
            allow_smem((const void *)k_lj_atm<true, 3>, sm);
            launch_pdl(k_lj_atm<true, 3>, grid, 256, sm, st, p, a, (int)e.n, per);
        } else {
            allow_smem((const void *)k_lj_atm<true, 2>, sm);
            launch_pdl(k_lj_atm<true, 2>, grid, 256, sm, st, p, a, (int)e.n, per);
        }
    } else {
        if (u3) {
            allow_smem((const void *)k_lj_atm<false, 3>, sm);
            launch_pdl(k_lj_atm<false, 3>, grid, 256, sm, st, p, a, (int)e.n, per);
        } else {
            allow_smem((const void *)k_lj_atm<false, 2>, sm);
            launch_pdl(k_lj_atm<false, 2>, grid, 256, sm, st, p, a, (int)e.n, per);
        }
    }
}

void launch_pair_tile(PairParams &p, int ncell, bool measure, bool emit, cudaStream_t st) {
    if (measure) {
        if (emit) launch_pdl(k_pair_tile<true, true>, ncell, kTileThreads, 0, st, p);
        else launch_pdl(k_pair_tile<true, false>, ncell, kTileThreads, 0, st, p);
    } else {
        if (emit) launch_pdl(k_pair_tile<false, true>, ncell, kTileThreads, 0, st, p);
        else launch_pdl(k_pair_tile<false, false>, ncell, kTileThreads, 0, st, p);
    }
}

}  // namespace komd
