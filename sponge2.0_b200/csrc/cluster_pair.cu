// Short-range force over the cluster lists: the per-step slot pack, the
// pruning of the neighbour tables into per-cluster partner lists, the
// cluster-pair force kernel and its finishing pass.  Together they are the
// B200 form of Lennard_Jones_And_Direct_Coulomb_Device and its dispatcher
// (SPONGE/Lennard_Jones_force/Lennard_Jones_force.cpp:43-136, 359-417) and of
// the solvent kernel (solvent_LJ.cpp:25-145), which evaluate the same pairs.
//
// List layout.  A cluster is 8 slots.  Each cluster I has one partner list:
// 32-bit words {partner slot - system's first slot (22 bits) | mask of the
// cluster's atoms the partner pairs with (8 bits) << 22 | image flag << 30}.
// A word's partner is evaluated against all eight atoms of I at once, so the
// partner's gathers and the word's decoding are paid once per eight pairs.
// The list holds partners in clusters J > I, and in I itself the pairs
// a < b: every pair once (a half list), the partner's share of each pair
// scattered by int64 atomics.  Words are kept when the partner lies within
// rc + buffer of one of the atoms at the last pruning, and a pruning is
// redone when an atom has moved half the buffer since, so no pair within rc
// is ever missing.
#include <math.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "pairfn.cuh"

namespace spgnb
{
namespace
{

constexpr int kPruneWarps = 4;
constexpr int kPruneAhead = 8;                      // pruning steps whose partners are loaded together
constexpr int kPruneStage = 384;                   // words a team's warp holds until they are joined
constexpr int kWindow = 32;                        // list parts are padded to whole 32-word windows
constexpr unsigned kWordSlotMask = (1u << 22) - 1u; // partner slot field of a list word
constexpr int kWordMaskShift = 22;                  // the 8-bit atom mask
constexpr unsigned kWordImage = 1u << 30;           // the pair needs its own periodic image
constexpr int kListImage = 1 << 30;                 // in a list's length: some word has its image flag set
constexpr int kPairResident[3] = {28, 20, 12};      // resident warps per SM of the force kernel's modes (registers)

// Per-step slot pack: each slot's offset from the build-time cluster centre
// moved by the displacement since the build (minimum image in the system's
// box, so a caller that wraps coordinates between builds is fine), with the
// charge; and the slot's aux record {cluster centre x | LJ type << 22, centre
// y, centre z, global index}, the 22-bit centre the force kernel takes
// differences of (its high bits are masked off there).  Slot slots_cap is a
// null slot: 10^4 A away from everything, charge 0.  With pruning on (pref
// set) the kernel also flags a re-pruning when some atom moved more than half
// the prune buffer since the last one.  It also clears the outputs the force
// call must start from zero (totals, module-owned per-atom energies).  With
// a gate it runs only when *gate is non-zero (after a rebuild, in the
// batched step).
__global__ void k_pack_slots(int slots_cap, int* counters, const int* __restrict__ slot_atom,
                             const int* __restrict__ slot_gid, const int* __restrict__ cl_sys,
                             const SysDesc* __restrict__ sys, const int4* __restrict__ cl_q,
                             const float4* __restrict__ x0, const float4* __restrict__ d0,
                             const float3* __restrict__ crd, const float* __restrict__ charge,
                             const int* __restrict__ local_type, SlotRec* __restrict__ rec,
                             const float4* __restrict__ pref, float half_buffer2, int* __restrict__ prune,
                             long long* __restrict__ clear_totals, long long* __restrict__ clear_one,
                             float* __restrict__ clear_a, float* __restrict__ clear_b, int clear_n,
                             const int* __restrict__ gate)
{
    grid_dep_wait();
    if (gate && *gate == 0) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    bool moved = false;
    // the outputs the force call zeroes first
    if (clear_totals && s < 8) clear_totals[s] = 0;
    if (clear_one && s == 0) *clear_one = 0;
    for (int k = s; k < clear_n; k += gridDim.x * blockDim.x)
    {
        if (clear_a) clear_a[k] = 0.0f;
        if (clear_b) clear_b[k] = 0.0f;
    }
    if (s == slots_cap)
    {
        rec[s].pos = make_float4(1.0e4f, 1.0e4f, 1.0e4f, 0.0f);
        rec[s].aux = make_int4(0, 0, 0, -1);
    }
    else if (s < slots_cap)
    {
        const int a = slot_atom[s];
        const float4 d = d0[s];
        const int4 q = cl_q[s >> 3];
        float4 p = make_float4(d.x, d.y, d.z, 0.0f);
        int t = 0;
        if (a >= 0)
        {
            const SysDesc& D = sys[cl_sys[s >> 3]];
            const float3 c = crd[a];
            const float4 o = x0[s];
            float dx = c.x - o.x, dy = c.y - o.y, dz = c.z - o.z;
            const float sx = rintf(dx * D.rcell.a11 + dy * D.rcell.a21 + dz * D.rcell.a31);
            const float sy = rintf(dy * D.rcell.a22 + dz * D.rcell.a32);
            const float sz = rintf(dz * D.rcell.a33);
            dx -= sx * D.cell.a11 + sy * D.cell.a21 + sz * D.cell.a31;
            dy -= sy * D.cell.a22 + sz * D.cell.a32;
            dz -= sz * D.cell.a33;
            p = make_float4(d.x + dx, d.y + dy, d.z + dz, charge[a]);
            t = local_type[a];
            if (pref)
            {
                const float4 r = pref[s];
                const float ex = p.x - r.x, ey = p.y - r.y, ez = p.z - r.z;
                moved = ex * ex + ey * ey + ez * ez > half_buffer2;
                if (moved) prune[cl_sys[s >> 3]] = 1;
            }
        }
        rec[s].pos = p;
        rec[s].aux = make_int4((q.x & 0x3fffff) | (t << 22), q.y, q.z, a >= 0 ? slot_gid[s] : -1);
    }
    if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) counters[kCntPrune] = 1;
}

// Pruning (no reference counterpart; results unchanged).  Runs after every
// rebuild and whenever some atom of a system moved more than buffer/2 since
// its last one (the pack kernel checks).  For cluster I it walks the
// elements of its neighbour table with J >= I (a table built one-sided holds
// no others), four at a time, one neighbour atom a lane: its own-atom mask
// bits come from the element's mask by a bit gather, it is tested against all
// eight atoms without branches (packed FP32x2, two atoms an instruction), and
// one word per partner within cutoff + buffer of any of them is written, in
// table order, padded to a whole window with words whose mask is empty.
// A chunk of 32 elements is loaded while the one before it is worked on, and
// its partners all together: with one step's loads in flight at a time the
// kernel waited for them (76 us on the 96,000-atom box against 57 now; four
// steps' partners together 58).  The form before, which first compacted each
// chunk's partners in shared memory, took 58 there, and 40 against 8 now on
// the 1,944-atom box, where a team works on each cluster.
// TEAM = 1: a warp takes a cluster; TEAM = 4: a block of four warps, each a
// share of the table, their words joined in order (few clusters: one warp's
// walk would be the kernel's time).  The last block to finish clears the
// flags.
template <int TEAM>
__global__ void __launch_bounds__(kPruneWarps * 32)
    k_prune8(ForceParams p0, const ForceParams* __restrict__ fps, float buffer, int* counters, int clusters_cap,
             int table_cap, int list_cap, const int* __restrict__ cl_sys, const SysDesc* __restrict__ sys,
             const int* __restrict__ tcount, const float4* __restrict__ tab, const uint2* __restrict__ tmask,
             const SlotRec* __restrict__ rec, float4* __restrict__ pref, int* __restrict__ lcount,
             unsigned* __restrict__ words, int n_sys, int* __restrict__ prune)
{
    grid_dep_wait();
    if (counters[kCntPrune] == 0) return;
    // the cluster's atoms negated, per coordinate, as four {even, odd} float2
    __shared__ __align__(16) float nown_all[kPruneWarps][3][kClusterSize];
    __shared__ float4 ent_all[kPruneWarps][32];  // a chunk's table elements
    __shared__ uint2 msk_all[kPruneWarps][32];
    __shared__ unsigned stage_all[TEAM > 1 ? kPruneWarps : 1][TEAM > 1 ? kPruneStage : 1];
    __shared__ int team_next, team_count[kPruneWarps], team_image[kPruneWarps];
    __shared__ unsigned long long kept_total;
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    if (threadIdx.x == 0) kept_total = 0;
    __syncthreads();
    float(&own)[3][kClusterSize] = nown_all[w];
    const float2* __restrict__ nown = reinterpret_cast<const float2*>(&own[0][0]);
    float4* ent = ent_all[w];
    uint2* msk = msk_all[w];
    const unsigned below = (1u << lane) - 1u;
    const int e_lane = lane >> 3, b_lane = lane & 7;
    for (;;)
    {
        int c = 0;
        if (TEAM == 1)
        {
            if (lane == 0) c = atomicAdd(&counters[kCntPruneNext], 1);
            c = __shfl_sync(0xffffffffu, c, 0);
        }
        else
        {
            __syncthreads();  // the previous cluster is done with
            if (threadIdx.x == 0) team_next = atomicAdd(&counters[kCntPruneNext], 1);
            __syncthreads();
            c = team_next;
        }
        if (c >= clusters_cap) break;
        const int sy = cl_sys[c];
        if (!prune[sy]) continue;
        const int s0 = c * kClusterSize;
        __syncwarp();
        if (lane < kClusterSize)
        {
            const float4 pl = rec[s0 + lane].pos;
            own[0][lane] = -pl.x;
            own[1][lane] = -pl.y;
            own[2][lane] = -pl.z;
            if (TEAM == 1 || w == 0) pref[s0 + lane] = pl;
        }
        __syncwarp();
        const SysDesc& D = sys[sy];
        const unsigned slot0 = (unsigned)D.cl_begin * kClusterSize;
        const ForceParams P = fps ? fps[sy] : p0;
        const float rp = sqrtf(P.rc2) + buffer + 1e-3f;
        const float rp2 = buffer > 0.0f ? rp * rp : 3.0e38f;
        const float2 nrp2 = f2(-rp2);
        const float4* __restrict__ tb = tab + (size_t)c * table_cap;
        const uint2* __restrict__ tm = tmask + (size_t)c * table_cap;
        unsigned* __restrict__ wc = words + (size_t)c * list_cap;
        const int usable = list_cap - kWindow;  // room left for the padding
        unsigned any_image = 0;

        // The words of table elements [lo, hi), to `out` (room of them);
        // returns their number.
        auto walk = [&](int lo, int hi, unsigned* out, int room) -> int {
            int kept = 0;
            auto element = [&](int t, float4& e, uint2& m) {
                e = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(s0));
                m = make_uint2(0u, 0u);
                if (t < hi)
                {
                    e = tb[t];
                    m = tm[t];
                    // clusters below I hold the other side of its pairs
                    if ((__float_as_int(e.w) & 0x3fffffff) < s0) m = make_uint2(0u, 0u);
                }
            };
            float4 en;
            uint2 mn;
            element(lo + lane, en, mn);
            for (int t0 = lo; t0 < hi; t0 += 32)
            {
                __syncwarp();
                ent[lane] = en;
                msk[lane] = mn;
                __syncwarp();
                element(t0 + 32 + lane, en, mn);
                const int quads = min(8, (hi - t0 + 3) / 4);
#pragma unroll 1
                for (int g = 0; g < quads; g += kPruneAhead)
                {
                    float4 pjs[kPruneAhead];
#pragma unroll
                    for (int k = 0; k < kPruneAhead; k++)
                        pjs[k] = rec[(__float_as_int(ent[4 * (g + k) + e_lane].w) & 0x3fffffff) + b_lane].pos;
#pragma unroll
                    for (int k = 0; k < kPruneAhead; k++)
                    {
                        if (g + k >= quads) break;
                        const float4 e = ent[4 * (g + k) + e_lane], pj = pjs[k];
                        const uint2 m = msk[4 * (g + k) + e_lane];
                        // the partner's own-atom bits: bit 8a + b of the element's
                        // mask for a = 0..7 (a multiplication gathers four bits)
                        const unsigned am = (((m.x >> b_lane) & 0x01010101u) * 0x01020408u) >> 24 |
                                            ((((m.y >> b_lane) & 0x01010101u) * 0x01020408u) >> 24) << 4;
                        const int eb = __float_as_int(e.w);
                        const unsigned js = (unsigned)(eb & 0x3fffffff) + b_lane;
                        const bool img = (eb & (1 << 30)) != 0;
                        // bit a: own atom a lies within the pruning radius of
                        // the partner; the minimum-image path (small boxes)
                        // only when a lane needs it
                        unsigned hit = 0;
                        if (!__any_sync(0xffffffffu, img && am != 0u))
                        {
                            const float2 cx = make_float2(e.x + pj.x, e.x + pj.x),
                                         cy = make_float2(e.y + pj.y, e.y + pj.y),
                                         cz = make_float2(e.z + pj.z, e.z + pj.z);
#pragma unroll
                            for (int p = 3; p >= 0; p--)
                            {
                                // r^2 - rp^2: its sign bits are shifted into hit
                                const float2 dx = __fadd2_rn(cx, nown[p]), dy = __fadd2_rn(cy, nown[4 + p]),
                                             dz = __fadd2_rn(cz, nown[8 + p]);
                                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nrp2)));
                                hit = __funnelshift_l(__float_as_uint(r2.y), hit, 1);
                                hit = __funnelshift_l(__float_as_uint(r2.x), hit, 1);
                            }
                        }
                        else
                        {
#pragma unroll 1
                            for (int a = 0; a < kClusterSize; a++)
                            {
                                const float4 pi = make_float4(-own[0][a], -own[1][a], -own[2][a], 0.0f);
                                const float3 d = pair_offset(e.x, e.y, e.z, pi, pj, img, D);
                                if (__fmaf_rn(d.z, d.z, __fmaf_rn(d.y, d.y, d.x * d.x)) < rp2) hit |= 1u << a;
                            }
                        }
                        hit &= am;
                        // partners in later clusters pair with every atom they
                        // reach; within the cluster only the pairs a < b
                        if ((js >> 3) == (unsigned)c) hit &= (1u << b_lane) - 1u;
                        const unsigned mh = __ballot_sync(0xffffffffu, hit != 0u);
                        const int at = kept + __popc(mh & below);
                        if (hit && at < room)
                            out[at] = (js - slot0) | (img ? kWordImage : 0u) | (hit << kWordMaskShift);
                        any_image |= img && hit != 0u ? 1u : 0u;
                        kept += __popc(mh);
                    }
                }
            }
            return kept;
        };

        const int T = tcount[c];
        int kh;
        if (TEAM == 1)
        {
            kh = walk(0, T, wc, usable);
            any_image = __any_sync(0xffffffffu, any_image);
        }
        else
        {
            unsigned* stage = stage_all[TEAM > 1 ? w : 0];
            const int quads = (T + 3) / 4;
            const int kept = walk(4 * (quads * w / TEAM), min(T, 4 * (quads * (w + 1) / TEAM)), stage, kPruneStage);
            any_image = __any_sync(0xffffffffu, any_image);
            if (lane == 0)
            {
                team_count[w] = kept;
                team_image[w] = (int)any_image;
            }
            __syncthreads();
            int start = 0, most = 0;
            kh = 0;
            any_image = 0;
#pragma unroll
            for (int v = 0; v < TEAM; v++)
            {
                const int k = team_count[v];
                if (v < w) start += k;
                kh += k;
                most = max(most, k);
                any_image |= (unsigned)team_image[v];
            }
            if (most > kPruneStage)
            {
                // a share that does not fit its staging: one warp for all
                if (w == 0) kh = walk(0, T, wc, usable);
            }
            else
                for (int k = lane; k < kept; k += 32)
                    if (start + k < usable) wc[start + k] = stage[k];
            if (w != 0) continue;
        }
        // an overflowed cluster keeps no list (the flag makes the caller regrow
        // and rebuild); otherwise pad it to a whole window
        if (kh > usable)
        {
            if (lane == 0) atomicOr(&counters[kCntOverflow], kOvfWords);
            kh = 0;
        }
        const int hp = (kh + kWindow - 1) & ~(kWindow - 1);
        const unsigned null_word = (unsigned)s0 - slot0;
        for (int k2 = kh + lane; k2 < hp; k2 += 32) wc[k2] = null_word;
        if (lane == 0)
        {
            lcount[s0] = hp | (any_image && hp ? kListImage : 0);
            atomicAdd(&kept_total, (unsigned long long)kh);
        }
        __syncwarp();
    }
    __shared__ int is_last;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        atomicAdd((unsigned long long*)&counters[kCntPWords], kept_total);
        __threadfence();
        is_last = atomicAdd(&counters[kCntPruneDone], 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    for (int q = threadIdx.x; q < n_sys; q += blockDim.x) prune[q] = 0;
    if (threadIdx.x == 0)
    {
        unsigned long long* wp = (unsigned long long*)&counters[kCntPWords];
        *(unsigned long long*)&counters[kCntPWordsLast] = atomicExch(wp, 0ull);
        counters[kCntPruneDone] = 0;
        counters[kCntPruneNext] = 0;
        counters[kCntPrune] = 0;
        counters[kCntPrunes] += 1;
    }
}

// Cluster-pair force kernel, one warp a block and one item a warp: a
// cluster's list, or a part of it.  The warp walks the item's words, one per
// lane per iteration; the partner's offset
// {delta + displacement, q} and aux record {22-bit centre, LJ type, global
// index} load once for all of the cluster's atoms the lane holds, and
//   dr = (c_J - c_I) * cell / 2^22 + p_j - p_i
// is formed with the exact integer centre difference.  The cluster's atoms
// are staged in shared memory as packed pairs, so every instruction of the
// pair function serves two pairs (FP32x2).  The LJ coefficients of a pair of
// cluster atoms against the partner's type come as one float4
// {-A_a, -A_b, B_a, B_b} of the T^3 table.  Words are loaded two iterations
// ahead of their use and partner records one, in registers.
//
// What bounds it, and why this shape: a packed FP32x2 instruction holds the
// FMA pipe for two cycles, and the kernel's time follows the instructions per
// word, of which only half are the pair arithmetic.  One-warp blocks leave
// the distribution of the items to the hardware: no counter (an atomic on one
// address per item), no barrier of unequal warps, no state kept live over the
// clusters (which spilled), and little shared memory, so that the L1 keeps
// partner records.  The same kernel as persistent blocks of four warps taking
// clusters from a counter took 89 us instead of 78 on the 96,000-atom box and
// 1,317 instead of 1,254 on the 1.0 M-atom box (with the partner records in
// shared memory rings 91 and 1,364).  Partner sums go out by RED (red_add):
// the ATOMG that atomicAdd becomes here waits for an answer, and with it and
// a test per component instead of one per word the two boxes took 103 and
// 1,548, the per-atom mode 217 instead of 151.  With 32-byte records and the
// fits as they are now (pairfn.cuh) the three take 71.5, 1,131 and 146.
//
// Each pair is evaluated once; a lane holds all 8 atoms, the partner's force
// (summed over the 8 in a fixed order) goes to its int64 fixed-point
// accumulator by one atomic add per component and word, and the cluster's
// forces are summed over the lanes in FP64 in a fixed order and added the same
// way.  Integer addition does not depend on order, so the forces are bitwise
// reproducible; the finishing pass converts them.  A lane's FP32 share depends
// on the parts a list is split into, and those, for one system, on the SM
// count, the mode and the list's capacity in clusters (launch_pair): one
// system's last bits can differ between chips, several systems' not.
//
// MODE 0: forces.  MODE 1: + energy and virial totals.  MODE 2: + per-atom
// energy and virial: a pair's terms belong to its owner, the atom with the
// lower global index, as the reference's half list credits them (water
// sites hand theirs to the residue's first atom, as SOLVENT_LENNARD_JONES
// does).  Cluster-owned sums stay in registers over the list; a word's
// partner-owned sums go to the partner's int64 staging, 8 atomic adds; the
// finishing pass turns the staging into the per-atom arrays and totals.
template <int MODE, int FIT, bool TRI>
__global__ void __launch_bounds__(32, kPairResident[MODE])
    k_pair8(ForceParams p0, const EwaldPoly ep, const ForceParams* __restrict__ fps, const SysDesc* __restrict__ sys, int n_clusters,
            int shift, int list_cap, const int* __restrict__ cl_sys, const int* __restrict__ lcount,
            const unsigned* __restrict__ words, const int4* __restrict__ cl_q, const SlotRec* __restrict__ rec,
            const float4* __restrict__ t4, long long* __restrict__ facc,
            long long* __restrict__ oacc, long long* __restrict__ totals, const int* __restrict__ only)
{
    grid_dep_wait();
    constexpr bool EN = MODE >= 1;
    constexpr bool PA = MODE >= 2;
    constexpr int NP = 4;        // the cluster's 8 atoms as packed pairs
    extern __shared__ float4 rows[];  // 4 x types coefficient rows (at least 8 x kSumRow floats)
    float* sums = reinterpret_cast<float*>(rows);  // after the list, the lanes' sums
    __shared__ float4 iat[4][2];  // the cluster's atom pairs {-x, -y | -z, -q}
    __shared__ int2 igid[4];      // and their global indices
    const int lane = threadIdx.x;
    // the item: part blockIdx.x mod 2^shift of the windows of its cluster's list
    const int c = blockIdx.x >> shift, part = blockIdx.x & ((1 << shift) - 1);
    const int s0 = c * kClusterSize;
    const int head = lcount[s0];
    const int windows = (head & ~kListImage) / kWindow;
    const int it0 = (windows * part) >> shift;
    const int iters = ((windows * (part + 1)) >> shift) - it0;
    if (iters <= 0) return;
    const int sy = cl_sys[c];
    if (only && !only[sy]) return;
    const ForceParams P = fps ? fps[sy] : p0;
    const PairParams2 pp = pack_params(P);
    const float2 lead = fit_lead<EN, FIT>(ep);
    const SysDesc& D = sys[sy];
    const Cell qc = D.qcell;
    const int slot0 = D.cl_begin * kClusterSize;
    const int4 ci = cl_q[c];
    const int nt = P.n_types;
    // the cluster's atoms, negated, as packed pairs, and the coefficient
    // rows of its four atom pairs against every partner type,
    // {-A_a, -A_b, B_a, B_b}, staged in shared memory
    {
        const float4 u = rec[s0 + (lane & 7)].pos;
        const int4 x = rec[s0 + (lane & 7)].aux;
        if (lane < 8)
        {
            float* f = reinterpret_cast<float*>(&iat[lane >> 1][0]) + (lane & 1);
            f[0] = -u.x;
            f[2] = -u.y;
            f[4] = -u.z;
            f[6] = -u.w;
            if (PA) reinterpret_cast<int*>(&igid[lane >> 1])[lane & 1] = x.w;
        }
        const int ti = (x.x >> 22) & 0x7f;
        const int row = (ti * nt + __shfl_down_sync(0xffffffffu, ti, 1)) * nt;  // of lanes 0, 2, 4, 6
        const float4* __restrict__ r = t4 + P.t4_begin;
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const int first = __shfl_sync(0xffffffffu, row, 2 * q);
            for (int e = lane; e < nt; e += 32) rows[q * nt + e] = __ldg(r + first + e);
        }
    }
    __syncwarp();
    float2 fx[NP], fy[NP], fz[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) fx[p] = fy[p] = fz[p] = f2(0.0f);
    float2 acc[(EN && !PA) ? 8 : 1];
#pragma unroll
    for (int q = 0; q < ((EN && !PA) ? 8 : 1); q++) acc[q] = f2(0.0f);
    float2 own[PA ? NP : 1][PA ? 8 : 1];
#pragma unroll
    for (int p = 0; p < (PA ? NP : 1); p++)
#pragma unroll
        for (int q = 0; q < (PA ? 8 : 1); q++) own[p][q] = f2(0.0f);

    const unsigned* __restrict__ wb = words + (size_t)c * list_cap + kWindow * it0;
    // the list's words; IMG: some of them need their pairs' own images
    auto walk = [&](auto image) {
        constexpr bool IMG = decltype(image)::value;
        // list words are loaded two iterations ahead of their use and
        // partner records one ahead, in registers
        const unsigned* __restrict__ wl = wb + lane;
        unsigned wc = wl[0];
        unsigned wn = iters > 1 ? wl[32] : 0u;
        float4 pjn;
        int4 xjn;
        load_rec(rec + (slot0 + (int)(wc & kWordSlotMask)), pjn, xjn);
#pragma unroll 1
        for (int it = 0; it < iters; it++)
        {
            const int jc = slot0 + (int)(wc & kWordSlotMask);
            const float ux = centre_step(xjn.x, ci.x), uy = centre_step(xjn.y, ci.y), uz = centre_step(xjn.z, ci.z);
            // the partner in the frame of the cluster's centre
            float sx = __fmaf_rn(ux, qc.a11, pjn.x);
            float sy2 = __fmaf_rn(uy, qc.a22, pjn.y);
            const float sz = __fmaf_rn(uz, qc.a33, pjn.z);
            if (TRI)
            {
                sx = __fmaf_rn(uy, qc.a21, sx);
                sx = __fmaf_rn(uz, qc.a31, sx);
                sy2 = __fmaf_rn(uz, qc.a32, sy2);
            }
            const int tj = (xjn.x >> 22) & 0x7f;
            const int gj = xjn.w;
            const float2 qj = f2(pjn.w);
            // the record is used up: the next one takes its registers
            unsigned wnn = 0u;
            if (it + 1 < iters)
            {
                const int jn = slot0 + (int)(wn & kWordSlotMask);
                load_rec(rec + jn, pjn, xjn);
                if (it + 2 < iters) wnn = wl[32 * (it + 2)];
            }
            float2 hx, hy, hz;     // the partner's force, negated
            float2 jo[PA ? 8 : 1];                                  // the partner's owned sums
#pragma unroll
            for (int q = 0; q < (PA ? 8 : 1); q++) jo[q] = f2(0.0f);
#pragma unroll
            for (int p = 0; p < NP; p++)
            {
                const float4 A = iat[p][0], B = iat[p][1];
                const float2 pnx = make_float2(A.x, A.y), pny = make_float2(A.z, A.w), pnz = make_float2(B.x, B.y),
                             pq = make_float2(B.z, B.w);
                float2 dx = __fadd2_rn(f2(sx), pnx), dy = __fadd2_rn(f2(sy2), pny), dz = __fadd2_rn(f2(sz), pnz);
                if (IMG && (wc & kWordImage))
                {
                    // small box: the pair takes its own minimum image
                    float ddx[2] = {dx.x, dx.y}, ddy[2] = {dy.x, dy.y}, ddz[2] = {dz.x, dz.y};
#pragma unroll
                    for (int h = 0; h < 2; h++)
                    {
                        const float tx = rintf(ddx[h] * D.rcell.a11 + ddy[h] * D.rcell.a21 + ddz[h] * D.rcell.a31);
                        const float ty = rintf(ddy[h] * D.rcell.a22 + ddz[h] * D.rcell.a32);
                        const float tz = rintf(ddz[h] * D.rcell.a33);
                        ddx[h] -= tx * D.cell.a11 + ty * D.cell.a21 + tz * D.cell.a31;
                        ddy[h] -= ty * D.cell.a22 + tz * D.cell.a32;
                        ddz[h] -= tz * D.cell.a33;
                    }
                    dx = make_float2(ddx[0], ddx[1]);
                    dy = make_float2(ddy[0], ddy[1]);
                    dz = make_float2(ddz[0], ddz[1]);
                }
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                const float4 ab = rows[p * nt + tj];
                float2 elj, ec;
                float2 f = pair_scalar2<EN, FIT>(r2, __fmul2_rn(qj, pq), make_float2(ab.x, ab.y),
                                                 make_float2(ab.z, ab.w), pp, ep, lead, elj, ec);
                const unsigned bitA = 1u << (kWordMaskShift + 2 * p), bitB = 2u << (kWordMaskShift + 2 * p);
                auto inside = [&](float2 v) {
                    return make_float2(inside_or_zero(v.x, r2.x, pp.rc2, wc, bitA),
                                       inside_or_zero(v.y, r2.y, pp.rc2, wc, bitB));
                };
                f = inside(f);
                fx[p] = __ffma2_rn(f, dx, fx[p]);
                fy[p] = __ffma2_rn(f, dy, fy[p]);
                fz[p] = __ffma2_rn(f, dz, fz[p]);
                hx = p == 0 ? __fmul2_rn(f, dx) : __ffma2_rn(f, dx, hx);
                hy = p == 0 ? __fmul2_rn(f, dy) : __ffma2_rn(f, dy, hy);
                hz = p == 0 ? __fmul2_rn(f, dz) : __ffma2_rn(f, dz, hz);
                const float2 gx = __fmul2_rn(f, dx), gy = __fmul2_rn(f, dy), gz = __fmul2_rn(f, dz);  // the virial's
                if (EN && !PA)
                {
                    acc[0] = __fadd2_rn(acc[0], inside(elj));
                    acc[1] = __fadd2_rn(acc[1], inside(ec));
                    acc[2] = __ffma2_rn(gx, dx, acc[2]);
                    acc[3] = __ffma2_rn(gx, dy, acc[3]);
                    acc[4] = __ffma2_rn(gy, dy, acc[4]);
                    acc[5] = __ffma2_rn(gx, dz, acc[5]);
                    acc[6] = __ffma2_rn(gy, dz, acc[6]);
                    acc[7] = __ffma2_rn(gz, dz, acc[7]);
                }
                if (PA)
                {
                    // the pair's owner is the lower global index: this lane's
                    // atom (kept over the list) or the partner (summed over
                    // the word's atoms)
                    const int2 pg = igid[p];
                    const float2 wi = make_float2(pg.x < gj ? 1.0f : 0.0f, pg.y < gj ? 1.0f : 0.0f);
                    const float2 v[8] = {inside(elj), inside(ec),
                                         __fmul2_rn(gx, dx), __fmul2_rn(gx, dy), __fmul2_rn(gy, dy),
                                         __fmul2_rn(gx, dz), __fmul2_rn(gy, dz), __fmul2_rn(gz, dz)};
#pragma unroll
                    for (int q = 0; q < 8; q++) own[p][q] = __ffma2_rn(v[q], wi, own[p][q]);
                    const float2 wj = __fadd2_rn(f2(1.0f), __fmul2_rn(wi, kPk[kPkMinusOne]));
#pragma unroll
                    for (int q = 0; q < 8; q++) jo[q] = __ffma2_rn(v[q], wj, jo[q]);
                }
            }
            if (PA)
            {
                // the partner's owned sums over this word: raw fixed point to
                // its staging (scaled in the finishing pass), one quantity
                // after another so that a warp's adds fall on few lines
                float js[8];
                bool any = false;
#pragma unroll
                for (int q = 0; q < 8; q++)
                {
                    js[q] = jo[q].x + jo[q].y;
                    any |= js[q] != 0.0f;
                }
                if (any)
                {
                    long long* oa = oacc + jc;
                    const size_t ostride = (size_t)n_clusters * kClusterSize;
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        red_add(oa + q * ostride, __float2ll_rn(js[q] * kTwoPow32));
                }
            }
            {
                // the partner's force: minus the sum over the cluster's atoms
                // (all zero when the word has no pair inside the cutoff)
                const float jx = hx.x + hx.y, jy = hy.x + hy.y, jz = hz.x + hz.y;
                if ((__float_as_uint(jx) | __float_as_uint(jy) | __float_as_uint(jz)) & 0x7fffffffu)
                {
                    long long* fa = facc + 3 * (size_t)jc;
                    red_add(fa + 0, __float2ll_rn(jx * -kTwoPow32));
                    red_add(fa + 1, __float2ll_rn(jy * -kTwoPow32));
                    red_add(fa + 2, __float2ll_rn(jz * -kTwoPow32));
                }
            }
            wc = wn;
            wn = wnn;
        }
    };
    if (head & kListImage)
        walk(std::true_type{});
    else
        walk(std::false_type{});

    // the cluster's sums over the lanes, eight at a time: lane 4a + d takes
    // component d of atom a's force; in the totals mode lane 4q + 3 the
    // energy or virial q
    double sum = 0.0;
#pragma unroll
    for (int d = 0; d < (EN && !PA ? 4 : 3); d++)
    {
        float v[8];
#pragma unroll
        for (int a = 0; a < 8; a++)
        {
            const float2 u = d == 0 ? fx[a / 2] : (d == 1 ? fy[a / 2] : fz[a / 2]);
            v[a] = d == 3 ? acc[a % ((EN && !PA) ? 8 : 1)].x + acc[a % ((EN && !PA) ? 8 : 1)].y : ((a & 1) ? u.y : u.x);
        }
        const double s = lane_totals8(sums, v, lane);
        if ((lane & 3) == d) sum = s;
    }
    if ((lane & 3) < 3)
        red_add(facc + 3 * (size_t)(s0 + (lane >> 2)) + (lane & 3), __double2ll_rn(sum * kForceScale));
    else if (EN && !PA)
    {
        // each pair once; the virial is -g (x) d, its symmetric
        // off-diagonal terms (xy + yx etc.) twice the one accumulated.  Eight
        // adds a list on one line: on the 1.0 M-atom box, where 137,000 lists
        // meet there, a force call with totals takes 1,682 us (2,065 with the
        // persistent warps that added theirs once at the end)
        const int q = lane >> 2;
        const double sc = q == 0 ? (double)kLjEnergyScale
                                 : (q == 1 ? (double)kCoulombEnergyScale
                                           : ((q == 3 || q == 5 || q == 6) ? -2.0 : -1.0));
        red_add(totals + 8 * (size_t)sy + q, __double2ll_rn(sum * sc * kEnergyScale));
    }
    if (PA)
    {
        // the cluster's owned sums: raw fixed point to each atom's
        // staging (scaled in the finishing pass), lane 4a + k quantity
        // q0 + k of atom a
#pragma unroll
        for (int q0 = 0; q0 < 8; q0 += 4)
        {
            double o = 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                float v[8];
#pragma unroll
                for (int a = 0; a < 8; a++) v[a] = (a & 1) ? own[a / 2][q0 + k].y : own[a / 2][q0 + k].x;
                const double s = lane_totals8(sums, v, lane);
                if ((lane & 3) == k) o = s;
            }
            red_add(oacc + (size_t)(q0 + (lane & 3)) * n_clusters * kClusterSize + s0 + (lane >> 2),
                    __double2ll_rn(o * kForceScale));
        }
    }
}

// The fused PME excluded-pair correction of atom a
// (Particle_Mesh::PME_Excluded_Force_With_Atom_Energy, PM_force.cpp:918-997):
// its symmetric exclusion list holds both sides of every pair, so each atom
// computes its own share, F_a += q_a q_x beta^3 h(beta r) dr with dr = the
// reference's minimum image of r_x - r_a, and the pair's owner (lower global
// index) adds -q_a q_x erf(beta r)/r to the energy and -F (x) dr to its
// virial (wv: xx, xy, yy, xz, yz, zz).
template <bool EN>
__device__ __forceinline__ void excl_terms(int a, const SysDesc& D, const ExclFuse& xf, float& fx, float& fy,
                                           float& fz, float& eown, float (&wv)[6])
{
    const int2 sn = xf.sn[a];
    const float3 ri = xf.crd[a];
    const float qa = xf.charge[a];
    const int ga = xf.atom_local[a];
    for (int k = 0; k < sn.y; k++)
    {
        const int jx = xf.list[sn.x + k];
        const float3 rj = xf.crd[jx];
        float ex = rj.x - ri.x, ey = rj.y - ri.y, ez = rj.z - ri.z;
        const float tx = floorf(ex * D.rcell.a11 + ey * D.rcell.a21 + ez * D.rcell.a31 + 0.5f);
        const float ty = floorf(ey * D.rcell.a22 + ez * D.rcell.a32 + 0.5f);
        const float tz = floorf(ez * D.rcell.a33 + 0.5f);
        ex -= tx * D.cell.a11 + ty * D.cell.a21 + tz * D.cell.a31;
        ey -= ty * D.cell.a22 + tz * D.cell.a32;
        ez -= tz * D.cell.a33;
        const float er = sqrtf(ex * ex + ey * ey + ez * ez);
        const float xb = xf.beta * er;
        const float qq = qa * xf.charge[jx];
        const float fa = qq * xf.beta3 * excl_h(xb);
        const float gx = fa * ex, gy = fa * ey, gz = fa * ez;
        fx += gx;
        fy += gy;
        fz += gz;
        if (EN && ga < xf.atom_local[jx])
        {
            eown -= qq * erff(xb) / er;
            wv[0] -= gx * ex;
            wv[1] -= gx * ey + gy * ex;
            wv[2] -= gy * ey;
            wv[3] -= gx * ez + gz * ex;
            wv[4] -= gy * ez + gz * ey;
            wv[5] -= gz * ez;
        }
    }
}

// Finishing pass of the force and totals modes, one thread per slot: the
// half-list kernel's int64 force sums go to the caller's float array, the
// staging cleared for the next call; with EXCL each atom also adds its
// excluded pairs' correction (and, with EN, its owned energy to the total).
// A thread touches only its own atom's force.
template <bool EXCL, bool EN>
__global__ void k_fin8(int slots, const int* __restrict__ slot_atom, const int* __restrict__ cl_sys,
                       const SysDesc* __restrict__ sys, long long* __restrict__ facc, float3* __restrict__ frc,
                       ExclFuse xf)
{
    grid_dep_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    float ene = 0.0f;
    if (s < slots)
    {
        const int a = slot_atom[s];
        long long* q = facc + 3 * (size_t)s;
        const long long x = q[0], y = q[1], z = q[2];
        if (x | y | z)
        {
            q[0] = 0;
            q[1] = 0;
            q[2] = 0;
        }
        if (a >= 0)
        {
            float fx = (float)((double)x * kForceUnscale), fy = (float)((double)y * kForceUnscale),
                  fz = (float)((double)z * kForceUnscale);
            if (EXCL)
            {
                float wv[6] = {0, 0, 0, 0, 0, 0};
                excl_terms<EN>(a, sys[cl_sys[s >> 3]], xf, fx, fy, fz, ene, wv);
            }
            if (fx != 0.0f || fy != 0.0f || fz != 0.0f)
            {
                float3 f = frc[a];
                f.x += fx;
                f.y += fy;
                f.z += fz;
                frc[a] = f;
            }
        }
    }
    if (EXCL && EN)
    {
        // the correction's energy total: one atomic per warp
        long long qe = __double2ll_rn((double)ene * kEnergyScale);
        for (int o = 16; o > 0; o >>= 1) qe += __shfl_xor_sync(0xffffffffu, qe, o);
        if ((threadIdx.x & 31) == 0 && qe) atomicAdd((unsigned long long*)xf.total, (unsigned long long)qe);
    }
}

// Finishing pass of the per-atom mode (one system), one thread per local
// atom a: its force from its slot's staging; the owned energy and virial of
// a itself, or, for the first atom of a water of the solvent tail, of every
// site of the residue (SOLVENT_LENNARD_JONES credits the residue's first
// atom; three or four sites), summed exactly in int64 from the sites'
// slots, go to the per-atom arrays by plain read-modify-writes (each element
// has one writer, so the result does not depend on thread order) and to the
// totals; the staging read is cleared for the next call.  With EXCL the
// atom's excluded-pair correction is added as in k_fin8.
//
// A block takes kFinAtoms atoms, a multiple of three and of four, counted so
// that the solvent tail starts at a block's first thread (lead): a residue
// lies within one block.  Each thread loads its own atom's eight sums and
// the residue's first adds the others' from shared memory, so no thread waits
// for more than its own loads (with the first atom's thread loading all of
// its residue's, 24 scattered values while the others idled, the kernel took
// 19 us on the 96,000-atom box; 12 now).
constexpr int kFinAtoms = 252;
template <bool EXCL>
__global__ void __launch_bounds__(256)
    k_fin8_atoms(int n, int slots, int lead, const int* __restrict__ atom_slot, const int* __restrict__ cl_sys,
                 const SysDesc* __restrict__ sys, long long* __restrict__ facc, long long* __restrict__ oacc,
                 float3* __restrict__ frc, long long* __restrict__ totals, OwnerMap om, PerAtomOut pa, ExclFuse xf)
{
    grid_dep_wait();
    __shared__ long long site[8][kFinAtoms];  // the block's atoms' owned sums
    const int a = (int)(blockIdx.x * kFinAtoms + threadIdx.x) - lead;
    const bool active = threadIdx.x < kFinAtoms && a >= 0 && a < n;
    float ene = 0.0f;
    long long tq[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // this atom's share of the totals
    int slot = 0, sites = 0;  // the sites whose owned sums a receives
    long long x = 0, y = 0, z = 0;
    long long r[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (active)
    {
        // every load first (they do not depend on each other beyond the
        // slot), then the arithmetic, then the stores: a thread waits for
        // memory about twice
        sites = 1;
        if (a >= om.solvent_start)
            sites = (a - om.solvent_start) % om.water_points ? 0 : min(min(om.water_points, n - a), 4);
        slot = atom_slot[a];
        const long long* q = facc + 3 * (size_t)slot;
        x = q[0];
        y = q[1];
        z = q[2];
#pragma unroll
        for (int u = 0; u < 8; u++) r[u] = oacc[(size_t)u * slots + slot];
#pragma unroll
        for (int u = 0; u < 8; u++) site[u][threadIdx.x] = r[u];
    }
    __syncthreads();
    if (active)
    {
        for (int k = 1; k < sites; k++)
#pragma unroll
            for (int u = 0; u < 8; u++) r[u] += site[u][threadIdx.x + k];
        if (sites == 0)  // its sums are its residue's first atom's
        {
#pragma unroll
            for (int u = 0; u < 8; u++) r[u] = 0;
        }
        long long* q = facc + 3 * (size_t)slot;
        const float3 f0 = frc[a];
        const bool own = sites > 0;
        const float e0 = own && pa.energy ? pa.energy[a] : 0.0f;
        const float l0 = own && pa.lj_energy ? pa.lj_energy[a] : 0.0f;
        const float d0 = own && pa.direct ? pa.direct[a] : 0.0f;
        float w0[6] = {0, 0, 0, 0, 0, 0};
        if (own && pa.virial)
        {
#pragma unroll
            for (int u = 0; u < 6; u++) w0[u] = pa.virial[6 * (size_t)a + u];
        }
        // the staging read is cleared for the next call
        if (x | y | z)
        {
            q[0] = 0;
            q[1] = 0;
            q[2] = 0;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) oacc[(size_t)u * slots + slot] = 0;
        // raw sums: -12 E_lj, -E_c, and +g (x) d; the virial is -g (x) d with
        // the symmetric off-diagonal terms twice the one summed
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
        {
            const double sg = u == 0 ? (double)kLjEnergyScale
                                     : (u == 1 ? (double)kCoulombEnergyScale : ((u == 3 || u == 5 || u == 6) ? -2.0 : -1.0));
            v[u] = (double)r[u] * sg;
            tq[u] = __double2ll_rn(v[u]);
        }
        const float elj = (float)(v[0] * kForceUnscale), ec = (float)(v[1] * kForceUnscale);
        float fx = (float)((double)x * kForceUnscale), fy = (float)((double)y * kForceUnscale),
              fz = (float)((double)z * kForceUnscale);
        float xe = 0.0f;
        float xw[6] = {0, 0, 0, 0, 0, 0};
        if (EXCL) excl_terms<true>(a, sys[cl_sys[slot >> 3]], xf, fx, fy, fz, xe, xw);
        ene = xe;
        if (fx != 0.0f || fy != 0.0f || fz != 0.0f) frc[a] = make_float3(f0.x + fx, f0.y + fy, f0.z + fz);
        if (own)
        {
            if (pa.energy) pa.energy[a] = e0 + (elj + ec);
            if (pa.lj_energy) pa.lj_energy[a] = l0 + elj;
            if (pa.direct) pa.direct[a] = d0 + ec;
            if (pa.virial)
            {
#pragma unroll
                for (int u = 0; u < 6; u++) pa.virial[6 * (size_t)a + u] = w0[u] + (float)(v[2 + u] * kForceUnscale);
            }
        }
        if (EXCL)
        {
            // the correction's own adds (its arrays may be the same ones)
            if (xf.energy && xe != 0.0f) xf.energy[a] += xe;
            if (xf.virial && xf.sn[a].y > 0)
            {
                float* w = xf.virial + 6 * (size_t)a;
#pragma unroll
                for (int u = 0; u < 6; u++) w[u] += xw[u];
            }
        }
    }
    // the totals: summed over the warp by shuffles, over the block in shared
    // memory, one atomic per value and block
    __shared__ long long bsum[8];
    if (threadIdx.x < 8) bsum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++)
    {
        long long v = tq[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd((unsigned long long*)&bsum[k], (unsigned long long)v);
    }
    __syncthreads();
    if (threadIdx.x < 8 && bsum[threadIdx.x])
        atomicAdd((unsigned long long*)&totals[threadIdx.x], (unsigned long long)bsum[threadIdx.x]);
    if (EXCL)
    {
        // the correction's energy total: one atomic per warp
        long long qe = __double2ll_rn((double)ene * kEnergyScale);
        for (int o = 16; o > 0; o >>= 1) qe += __shfl_xor_sync(0xffffffffu, qe, o);
        if ((threadIdx.x & 31) == 0 && qe) atomicAdd((unsigned long long*)xf.total, (unsigned long long)qe);
    }
}

// The K (forces) or M (energies) fit in r^2 for this Ewald parameter.
EwaldPoly scaled_fit(const ForceParams& f, bool energy)
{
    EwaldPoly e;
    const double b = f.beta, w = b * b / (double)SPGNB_EWALD_W_MAX;
    double nq = 1.0 / (w * w * w * w * w), np = (energy ? -b : -b * b * b) * nq;
    for (int k = 0; k < 6; k++, np *= w, nq *= w)
    {
        // divided by w^5: the denominator stays monic
        const float p = (float)((energy ? kEwaldMPHost[k] : kEwaldKPHost[k]) * np);
        const float q = (float)((energy ? kEwaldMQHost[k] : kEwaldKQHost[k]) * nq);
        e.p[k] = make_float2(p, p);
        e.q[k] = make_float2(q, q);
    }
    return e;
}

// The dynamic shared memory that leaves `blocks` blocks of this kernel
// resident on an SM: an equal share of the SM's, less the kernel's static
// memory and what the runtime reserves for each block.  0 when they fit
// anyhow.
size_t smem_for_resident(const void* kernel, long long blocks)
{
    int dev = 0, per_sm = 0, reserved = 0;
    cudaFuncAttributes attr{};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&attr, kernel) != cudaSuccess)
    {
        cudaGetLastError();
        return 0;
    }
    const long long own = (long long)attr.sharedSizeBytes + reserved;
    return (size_t)std::max(0LL, (per_sm / blocks & ~127LL) - own);  // allocated in units of 128 bytes
}

template <int M, int F, bool T>
int launch_pair(const ForceInputs& in, cudaStream_t s)
{
    const spgnb_nl* nl = in.nl;
    const EwaldPoly ep = F == 2 ? scaled_fit(in.p0, M >= 1) : EwaldPoly{};
    const int mt = in.max_types > 0 ? in.max_types : in.p0.n_types;
    size_t smem = sizeof(float4) * std::max(4 * mt, 2 * kSumRow);
    // the setting counts groups of four one-warp blocks: it holds the resident
    // ones down by the shared memory each asks for
    if (in.pair_blocks_per_sm > 0)
        smem = std::max(smem, smem_for_resident((const void*)k_pair8<M, F, T>, 4LL * in.pair_blocks_per_sm));
    // Each cluster's list in 2^shift parts, as many as keep the items within
    // one and a half times the warps the chip holds.  With fewer clusters than
    // warps the kernel's time is one warp's walk over a list: the 6,480-atom
    // box takes 39 us with whole lists and 14 with four parts, the 1,944-atom
    // one 26 and 7.  An item costs about one and a half windows of its own
    // (the 96,000-atom box takes 80 us with whole lists, 82 with halves, 101
    // with quarters).  Several systems: whole lists, since a system's sums, and
    // with them its trajectory's bits, must not depend on the systems around it.
    int shift = 0;
    if (!in.d_fps)
        while (shift < 4 && ((long long)nl->clusters_cap << (shift + 1)) <= 3LL * kPairResident[M] * num_sms() / 2) shift++;
    const unsigned grid = (unsigned)nl->clusters_cap << shift;
    if (smem > 48 * 1024)
        SPGNB_CUDA(cudaFuncSetAttribute(k_pair8<M, F, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    launch_dependent(k_pair8<M, F, T>, grid, 32, smem, s,
        in.p0, ep, in.d_fps, nl->d_sys, nl->clusters_cap, shift, nl->list_cap, nl->d_cl_sys, nl->d_pcount, nl->d_pwords,
        nl->d_cl_q, in.slots, in.t4, nl->d_facc, nl->d_oacc, in.totals, in.only);
    SPGNB_CHECK_LAUNCH("k_pair8");
    return SPGNB_OK;
}

template <int M, int F>
int launch_pair_t(const ForceInputs& in, bool tri, cudaStream_t s)
{
    return tri ? launch_pair<M, F, true>(in, s) : launch_pair<M, F, false>(in, s);
}

// FIT 2, the fits scaled to the call's one system, or 1 for several systems
// and for an Ewald parameter so small (beta below 0.0035 / A, or none) that the
// scaled coefficients, up to beta^-10, would leave FP32's range (at a w_scale
// of 1e-6 the denominator reaches 7.3e30 and its flushed reciprocal 1.4e-31:
// lowered by a factor of 20 or more it would leave the normal range); 0 outside the fits'
// range.
template <int M>
int launch_pair_ft(const ForceInputs& in, bool tri, cudaStream_t s)
{
    if (!in.fit) return launch_pair_t<M, 0>(in, tri, s);
    return in.d_fps || in.p0.w_scale < 1e-6f ? launch_pair_t<M, 1>(in, tri, s) : launch_pair_t<M, 2>(in, tri, s);
}

}  // namespace

std::vector<float4> coefficient_table(const float2* table, int T)
{
    std::vector<float4> t4((size_t)T * T * T);
    for (int a = 0; a < T; a++)
        for (int b = 0; b < T; b++)
            for (int j = 0; j < T; j++)
            {
                const float2 ga = table[(size_t)a * T + j], gb = table[(size_t)b * T + j];
                t4[((size_t)a * T + b) * T + j] = make_float4(-ga.x, -gb.x, ga.y, gb.y);
            }
    return t4;
}

int build_t4(const float2* table, int T, float4** d_t4)
{
    const std::vector<float4> t4 = coefficient_table(table, T);
    dfree(*d_t4);
    int st = dalloc(d_t4, t4.size());
    if (st) return st;
    SPGNB_CUDA(cudaMemcpy(*d_t4, t4.data(), sizeof(float4) * t4.size(), cudaMemcpyHostToDevice));
    return SPGNB_OK;
}

int force_check(const ForceInputs& in)
{
    if (!in.t4) return fail(SPGNB_E_STATE, "force: the LJ module has no pair table");
    if (in.mode == 2 && in.nl->S != 1)
        return fail(SPGNB_E_UNSUPPORTED, "force: per-atom energy/virial outputs are for a one-system list");
    if (in.p0.n_types <= 0 || in.p0.n_types > kMaxTypes)
        return fail(SPGNB_E_UNSUPPORTED, "force: %d LJ types (at most %d)", in.p0.n_types, kMaxTypes);
    return SPGNB_OK;
}

int launch_pack(const ForceInputs& in, cudaStream_t s, const int* gate)
{
    spgnb_nl* nl = in.nl;
    const int slots = nl->clusters_cap * kClusterSize;
    const bool track = nl->opt.prune_buffer > 0.0f;
    const float half = 0.5f * nl->opt.prune_buffer;
    launch_dependent(k_pack_slots, (slots + 256) / 256, 256, 0, s, slots, nl->d_counters, nl->d_slot_atom, nl->d_slot_gid,
                                                     nl->d_cl_sys, nl->d_sys, nl->d_cl_q, nl->d_slot_x0,
                                                     nl->d_slot_d0, in.crd, in.charge, in.atom_type, in.slots,
                                                     track ? nl->d_pref : nullptr, half * half,
                                                     nl->d_prune, in.clear.totals, in.clear.one, in.clear.a, in.clear.b,
                                                     in.clear.n, gate);
    SPGNB_CHECK_LAUNCH("k_pack_slots");
    return SPGNB_OK;
}

int launch_prune(const ForceInputs& in, cudaStream_t s)
{
    spgnb_nl* nl = in.nl;
    // the blocks-per-SM setting counts blocks of eight warps
    const int prune_bps = 2 * (in.prune_blocks_per_sm > 0 ? in.prune_blocks_per_sm : 5);
    // a block of four warps per cluster up to 36 clusters an SM (24,000 atoms:
    // 24 us a pruning, 27 with a warp each)
    const bool team = nl->clusters_cap <= num_sms() * 36;
    const int grid = std::max(1, std::min(num_sms() * prune_bps, team ? nl->clusters_cap :
                                                                 (nl->clusters_cap + kPruneWarps - 1) / kPruneWarps));
    launch_dependent(team ? k_prune8<4> : k_prune8<1>, grid, kPruneWarps * 32, 0, s, in.p0, in.d_fps, nl->opt.prune_buffer, nl->d_counters,
                                               nl->clusters_cap, nl->table_cap, nl->list_cap,
                                               nl->d_cl_sys, nl->d_sys, nl->d_tcount, nl->d_tab, nl->d_tmask,
                                               in.slots, nl->d_pref, nl->d_pcount, nl->d_pwords, nl->S,
                                               nl->d_prune);
    SPGNB_CHECK_LAUNCH("k_prune8");
    return SPGNB_OK;
}

int launch_pair_kernel(const ForceInputs& in, cudaStream_t s)
{
    spgnb_nl* nl = in.nl;
    cudaEvent_t ev0, ev1;
    pair_events(&ev0, &ev1);
    if (ev0) SPGNB_CUDA(cudaEventRecord(ev0, s));
    int st;
    if (in.mode == 0)
        st = launch_pair_ft<0>(in, nl->triclinic, s);
    else if (in.mode == 1)
        st = launch_pair_ft<1>(in, nl->triclinic, s);
    else
        st = launch_pair_ft<2>(in, nl->triclinic, s);
    if (st) return st;
    if (ev1) SPGNB_CUDA(cudaEventRecord(ev1, s));
    return SPGNB_OK;
}

int force_pipeline(const ForceInputs& in, cudaStream_t s)
{
    spgnb_nl* nl = in.nl;
    const int slots = nl->clusters_cap * kClusterSize;
    int st = force_check(in);
    if (!st) st = launch_pack(in, s, nullptr);
    if (!st) st = launch_prune(in, s);
    if (!st) st = launch_pair_kernel(in, s);
    if (st) return st;
    const bool excl = in.xf.list != nullptr;
    const int blocks = (slots + 255) / 256;
    if (in.mode == 2)
    {
        const int n = nl->local_atoms;
        const int lead = (kFinAtoms - in.om.solvent_start % kFinAtoms) % kFinAtoms;
        const int ab = (n + lead + kFinAtoms - 1) / kFinAtoms;
        launch_dependent(excl ? k_fin8_atoms<true> : k_fin8_atoms<false>, ab, 256, 0, s, n, slots, lead, nl->d_atom_slot,
                         nl->d_cl_sys, nl->d_sys, nl->d_facc, nl->d_oacc, in.frc, in.totals, in.om, in.pa, in.xf);
    }
    else if (excl && in.mode == 1)
        launch_dependent(k_fin8<true, true>, blocks, 256, 0, s, slots, nl->d_slot_atom, nl->d_cl_sys, nl->d_sys, nl->d_facc, in.frc,
                                                  in.xf);
    else if (excl)
        launch_dependent(k_fin8<true, false>, blocks, 256, 0, s, slots, nl->d_slot_atom, nl->d_cl_sys, nl->d_sys, nl->d_facc,
                                                   in.frc, in.xf);
    else
        launch_dependent(k_fin8<false, false>, blocks, 256, 0, s, slots, nl->d_slot_atom, nl->d_cl_sys, nl->d_sys, nl->d_facc,
                                                    in.frc, in.xf);
    SPGNB_CHECK_LAUNCH("k_fin8");
    return SPGNB_OK;
}

}  // namespace spgnb
