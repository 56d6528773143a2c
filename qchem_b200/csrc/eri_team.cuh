// eri_team.cuh -- warp-specialised ERI-batch kernel for the high-L classes (team form).
//
// A CTA takes 32 contracted quartets of one contraction pattern at a time (a "group": batch_plan.h), one per lane
// -- or, where a batch is too small to hide a long primitive loop, fewer quartets with the bra primitive pairs of
// each split over several lanes, whose [e0|f0] are added -- and works through them in three phases.
//
//  1. Stage tables.  For every primitive quartet x of the group (bra primitive pair outer, ket inner) and
//     every lane, a "stage" holds R^0_{tuv} scaled by the prefactor lambda and the single-centre Hermite
//     tables E^{i0}_t of the ket pair (and, after the last ket primitive of a bra primitive pair, of the bra
//     pair) -- generated code, team_produce_<k>.  All warps compute stages, warp w taking x = w, w + nwarps,
//     ..., and write them once to the CTA's slots of the R cache in global memory (entry-major, lane-minor).
//     Two variants were measured slower on a B200 and dropped: rebuilding the Hermite tables in the
//     consumers to halve the stage (1.4x slower on (dd|dd): the contraction is bound by instruction issue),
//     and walking the group one bra primitive pair at a time so that the cache stays in L2 (1.3x slower: a
//     barrier, a pipeline restart and an accumulator save per window cost more than the HBM traffic saved).
//  2. Contraction.  A warp works on one component f of the ket range of the horizontal-recurrence form (f over
//     L = LC..LC+LD on centre C) per pass.  Components that are cyclic rotations of one another run the same
//     code in rotated frames (gen_md.py, team form): warp 3 g + r takes piece pass * kNG + g of the ket code in
//     rotation r, so the three warps of a piece walk one instruction stream over one stage.  It keeps in
//     registers Y_f -- the ket step summed over the ket primitives of the current bra primitive pair -- and
//     acc_f = [e0|f] for every e, adding the bra step of Y_f to acc_f after the bra pair's last ket primitive
//     (team_ket_piece_<k>, team_bra_view_<k>).  The stages stream from the R cache into shared memory, three
//     deep, by bulk copies (cp.async.bulk, the Tensor Memory Accelerator's untiled form) on mbarriers, without a
//     gap between passes.  With more pieces than
//     a pass holds, each pass reads the stages again (from L2 or HBM) instead of recomputing them.
//  3. Recurrences.  acc_f goes to the CTA's scratch as [e0|f0] (lane-minor, so every access of a warp is
//     one coalesced line); the ket recurrence per e row gives [e0|cd] there, and the bra recurrence per
//     (c d) column writes (ab|cd) into the quartet's output block (generated team_hrr_ket_<k>,
//     team_hrr_bra_<k>).  No atomics: every output element is written once by one thread.
//
// This is the arithmetic of qchem's PrimGaussian::Repulsion4C (PG_Cart_MnD/Imp/GaussianRF.C:446-483) and
// its contraction (GaussianRF.C:726-752), with the bra and ket transfers done once per contracted quartet
// (horizontal recurrence) and the bra Hermite contraction once per bra primitive pair.
#pragma once
#include <cstdint>

#include "eri_team_iface.h"
#include "md_core.cuh"
#include "team_sync.cuh"

namespace qcg {

extern __shared__ __align__(128) double qcg_team_smem[];

// Shared memory of both kernels: three stages, whose space holds the group's primitive pairs while the stage
// tables are made (slot t of lane l: entry k at [(t * kTeamPairDoubles + k) * 32 + l]), then the Boys columns.
template <class Cls>
__device__ __forceinline__ BoysColumns team_boys(double* __restrict__ s, const double* __restrict__ table)
{
    for (int i = threadIdx.x; i < kBoysRows * kBoysColumns; i += blockDim.x)
    {
        const int k = i / kBoysRows, it = i - k * kBoysRows;
        const double f[kBoysColumns] = {1.0, 1.0, 0.5, 1.0 / 6.0, 1.0 / 24.0, 1.0 / 120.0, 1.0 / 720.0};
        double c = f[0];
#pragma unroll
        for (int j = 1; j < kBoysColumns; ++j) c = k == j ? f[j] : c;
        s[i] = table[it * 23 + Cls::LA + Cls::LB + Cls::LC + Cls::LD + k] * c;
    }
    return BoysColumns{s};
}
__device__ __forceinline__ void team_pair_store(int t, int lane, const TeamPair& d)
{
    double* const s = qcg_team_smem + t * kTeamPairDoubles * 32 + lane;
    s[0] = d.p; s[32] = d.Px; s[64] = d.Py; s[96] = d.Pz;
    s[128] = d.PAx; s[160] = d.PAy; s[192] = d.PAz; s[224] = d.kp; s[256] = d.h;
}
__device__ __forceinline__ TeamPair team_pair_load(int t, int lane)
{
    const double* const s = qcg_team_smem + t * kTeamPairDoubles * 32 + lane;
    return TeamPair{s[0], s[32], s[64], s[96], s[128], s[160], s[192], s[224], s[256]};
}

// Phase 1 of both kernels: the stage tables of the group's primitive quartets into rc.  bra(i) and ket(i) give
// this lane's primitive pairs; each is formed once, by the warps in turn, and read back from shared memory by the
// stages that use it (a contraction too long for that space forms them stage by stage).  A pair is two divisions and
// an exponential; formed by every stage they took half of a (ps|ps) stage's 2150 cycles.
template <class Cls, class Bra, class Ket>
__device__ __forceinline__ void team_stages(double* __restrict__ rc, const int Kab, const int Kcd, const int Kg,
                                            const BoysColumns& bt, Bra bra, Ket ket)
{
    constexpr int NW = Cls::kNW, STAGE = Cls::kStage * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int K = Kab * Kcd;
    const int npair = __reduce_max_sync(0xffffffffu, Kab + Kcd);
    const bool kept = npair <= Cls::kPairSlots;   // CTA-uniform: every warp sees the same lanes
    if (kept)
        for (int t = warp; t < npair; t += NW)
        {
            if (t < Kab) team_pair_store(t, lane, team_pair(bra(t)));
            else if (t < Kab + Kcd) team_pair_store(t, lane, team_pair(ket(t - Kab)));
        }
    __syncthreads();
    for (int x = warp; x < Kg; x += NW)
        if (x < K)
        {
            const int ij = x / Kcd, kl = x - ij * Kcd;
            const TeamPair ab = kept ? team_pair_load(ij, lane) : team_pair(bra(ij));
            const TeamPair cd = kept ? team_pair_load(Kab + kl, lane) : team_pair(ket(kl));
            Cls::produce(rc + (long long)x * STAGE + lane, ab, cd, bt, kl == Kcd - 1);
        }
    team::fence_async();   // the stages (global) and the pairs (shared) before the copies into the stage space
    __syncthreads();
}

// The ring of three slots in shared memory that the stages pass through, kUnroll stages to a slot: full[s] completes
// when slot s holds its stages, done[s] counts the warps that have finished with them.  slot, phase: the next step's
// slot and the parity its full[] completes with.
struct TeamRing
{
    uint64_t* full;
    int* done;
    int slot = 0;
    uint32_t phase = 0;
};

// Phase 2 of both kernels: [e0|f0] of the group (lane-minor, rows and columns in slot order) from the Kg stages
// in rc; K and Kcd are this lane's primitive-quartet and ket-pair counts (0 for an absent quartet).  Warps are not
// held together: each waits for a step's stages by itself, and the warp that leaves a slot last starts the copy of
// the step three later into it (a fixed warp that refilled slots as it came to them took 3.0 ms where this takes 2.6
// on (dd|pp)).  A step costs some hundred cycles of waits and barrier traffic beside its arithmetic (480 cycles
// for a (pp|pp) stage), so it takes as many stages as the shared memory gives three slots for.
// False, in every warp that sees it, when a bulk copy did not arrive.
template <class Cls>
__device__ __forceinline__ bool team_contract(const double* __restrict__ rc, double* __restrict__ hA, const int K,
                                              const int Kcd, const int Kg, TeamRing& ring, int* err)
{
    constexpr int NG = Cls::kNG, NE = Cls::kNE, NH = Cls::kNH, NC = Cls::kNCode, NW = Cls::kNW, U = Cls::kUnroll;
    constexpr int NPASS = (NC + NG - 1) / NG;
    constexpr int STAGE = Cls::kStage * 32;        // doubles per stage (entry-major, lane-minor)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int piece = warp / 3, rot = warp - 3 * piece;
    const int per = (Kg + U - 1) / U, nsteps = NPASS * per;   // steps of a pass, and in all
    // the copy of a pass's step c into slot, by one warp; a single stage goes without the bra tables where no lane's
    // bra step needs them
    auto issue = [&](int c, int slot) {
        const int x0 = c * U, n = Kg - x0 < U ? Kg - x0 : U;
        uint32_t bytes = (uint32_t)n * STAGE * sizeof(double);
        if (U == 1 && !__any_sync(0xffffffffu, x0 < K && (x0 + 1) % Kcd == 0))
            bytes = Cls::kKetStage * 32 * (uint32_t)sizeof(double);
        if (lane == 0)
            team::bulk_load(qcg_team_smem + slot * U * STAGE, rc + (long long)x0 * STAGE, bytes, &ring.full[slot]);
    };
    int ahead = 0;   // the step three later, within its pass
    for (int t = 0, slot = ring.slot; t < 3; ++t, slot = slot == 2 ? 0 : slot + 1)
    {
        if (warp == 0 && t < nsteps) issue(ahead, slot);
        if (++ahead == per) ahead = 0;
    }
    int t = 0;
    for (int pass = 0; pass < NPASS; ++pass)
    {
        const int jc = pass * NG + piece;
        const bool on = jc < NC && !(rot != 0 && Cls::fixed(jc));
        double Y[NH], acc[NE];
#pragma unroll
        for (int h = 0; h < NH; ++h) Y[h] = 0.0;
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.0;
        int kl = 0;
        for (int c = 0; c < per; ++c, ++t)
        {
            const int slot = ring.slot;
            if (!team::mbar_wait(&ring.full[slot], ring.phase))
            {
                // a copy did not arrive: record it, let the ones in flight land and leave
                if (lane == 0)
                {
                    atomicOr(err, 1);
                    team::drain(ring.full, slot, ring.phase, nsteps - t < 3 ? nsteps - t : 3);
                }
                __syncwarp();
                return false;
            }
            const int n = Kg - c * U < U ? Kg - c * U : U;
            for (int u = 0; u < n; ++u)
                if (on && c * U + u < K)
                {
                    const typename Cls::View v(qcg_team_smem + (slot * U + u) * STAGE + lane, rot);
                    Cls::ket(jc, v, Y);
                    if (kl == Kcd - 1)
                    {
                        Cls::bra(v, Y, acc);
#pragma unroll
                        for (int h = 0; h < NH; ++h) Y[h] = 0.0;
                        kl = 0;
                    }
                    else
                        ++kl;
                }
            __syncwarp();
            int last = 0;
            if (lane == 0) last = team::count_done(&ring.done[slot]) == NW - 1;
            if (__shfl_sync(0xffffffffu, last, 0))
            {
                if (lane == 0) ring.done[slot] = 0;
                if (t + 3 < nsteps) issue(ahead, slot);
            }
            if (++ahead == per) ahead = 0;
            ring.slot = slot == 2 ? 0 : slot + 1;
            if (slot == 2) ring.phase ^= 1;
        }
        if (on) Cls::store(acc, hA + (Cls::fslot(jc) + rot) * 32 + lane, rot);
    }
    __syncthreads();   // the stages are no longer read; [e0|f0] is written
    return true;
}

// OT: the output type.  Float output (the FP32 batches) is the FP64 evaluation rounded once.
template <class Cls, class OT>
__global__ void __launch_bounds__(Cls::kNW * 32, Cls::kMinBlocks)
    eri_batch_team_kernel(BasisDev bs, const int4* __restrict__ quartets, const int* __restrict__ order,
                          const int nq, OT* __restrict__ out, const double* __restrict__ boys_table, TeamScratchDev scr)
{
    constexpr int NW = Cls::kNW;
    constexpr int NF = Cls::kNF, NE = Cls::kNE;
    constexpr int STAGE = Cls::kStage * 32;        // doubles per stage (entry-major, lane-minor)
    constexpr int NCD = ncart(Cls::LC) * ncart(Cls::LD);
    constexpr long long BLK = (long long)ncart(Cls::LA) * ncart(Cls::LB) * NCD;
    static_assert(NE <= ncart(Cls::LA) * ncart(Cls::LB) && NF <= NCD, "[e0|f0] fits the output block");
    __shared__ uint64_t full[3];
    __shared__ int done[3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool leader = threadIdx.x == 0;
    if (leader)
    {
        for (int s = 0; s < 3; ++s)
        {
            team::mbar_init(&full[s]);
            done[s] = 0;
        }
        team::mbar_init_fence();
    }
    const BoysColumns bt = team_boys<Cls>(qcg_team_smem + Cls::kStageSpace, boys_table);
    __syncthreads();
    double* const rc = scr.rcache + (long long)blockIdx.x * scr.kmax * STAGE;   // this CTA's stage slots
    double* const hA = scr.hrr + (long long)blockIdx.x * (NE * NF + NE * NCD) * 32;
    double* const hB = hA + NE * NF * 32;
    TeamRing ring{full, done};
    __shared__ BatchPlanDev plan;
    __shared__ int lane_q[32];   // each lane's quartet, for the phases after the contraction; -1: none
    if (scr.plan)
        for (int k = threadIdx.x; k < (int)(sizeof(BatchPlanDev) / sizeof(int)); k += blockDim.x)
            reinterpret_cast<int*>(&plan)[k] = reinterpret_cast<const int*>(scr.plan)[k];
    else   // an uncontracted class: one pattern, groups of 32 quartets as they come
        for (int k = threadIdx.x; k < 257; k += blockDim.x)
        {
            plan.first[k] = k ? nq : 0;
            plan.group[k] = k ? (int)(((long long)nq + 31) >> 5) : 0;
            if (k < 256) plan.lanes[k] = 0;
        }
    __syncthreads();
    const int ngroups = plan.group[256];
    int b = -1;   // the group's bucket: the last one that starts no later, found by bisection (most are empty)
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x)
    {
        if (b < 0 || plan.group[b + 1] <= g)
        {
            b = 0;
            for (int hi = 256; hi - b > 1;)
            {
                const int mid = (b + hi) >> 1;
                if (plan.group[mid] <= g) b = mid;
                else hi = mid;
            }
        }
        // every warp reads the same quartets: lane l of every warp holds bra primitive pairs sub, sub + S, ... of its
        // quartet, S = 1 << lg
        const int lg = plan.lanes[b], sub = lane & ((1 << lg) - 1);
        // 64 bits: the last group of a batch of nearly 2^31 quartets reaches beyond it
        const long long gi = plan.first[b] + (long long)(g - plan.group[b]) * (32 >> lg) + (lane >> lg);
        const bool valid = gi < plan.first[b + 1];
        const long long q = valid ? (long long)(order ? order[gi] : gi) : 0;
        if (warp == 0) lane_q[lane] = valid && sub == 0 ? (int)q : -1;
        const int4 s = quartets[q];
        int ni = 0, nj = 0, nk = 0, nl = 0;
        if (valid)
        {
            ni = bs.nprim[s.x];
            nj = bs.nprim[s.y];
            nk = bs.nprim[s.z];
            nl = bs.nprim[s.w];
        }
        const int Kab = sub < ni * nj ? (ni * nj - sub - 1 >> lg) + 1 : 0;   // this lane's bra primitive pairs
        const int Kcd = nk * nl, K = Kab * Kcd;
        const int Kg = __reduce_max_sync(0xffffffffu, K);   // the group's longest primitive loop (CTA-uniform)
        if (Kg > scr.kmax)
        {
            if (leader) atomicOr(scr.err, 2);
            continue;
        }
        // 1. stage tables of every primitive quartet, written once to the R cache
        team_stages<Cls>(
            rc, Kab, Kcd, Kg, bt,
            [&](int m) {
                const int ij = (m << lg) + sub;
                return shell_prim_pair(bs, s.x, ij / nj, s.y, ij % nj);
            },
            [&](int kl) { return shell_prim_pair(bs, s.z, kl / nl, s.w, kl % nl); });
        // 2. contraction, the stages streamed back through shared memory three deep
        if (!team_contract<Cls>(rc, hA, K, Kcd, Kg, ring, scr.err)) return;
        // the lanes that share a quartet add their [e0|f0]
        if (const int share = plan.lanes[b]; share > 0)
        {
            for (int k = warp; k < NE * NF; k += NW)
            {
                double v = hA[k * 32 + lane];
                for (int o = 1; o < 1 << share; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                hA[k * 32 + lane] = v;
            }
            __syncthreads();
        }
        // 3. recurrences: ket per e row into [e0|cd], bra per (c d) column into the output block
        const int hq = lane_q[lane];
        const int4 hs = quartets[hq < 0 ? 0 : hq];
        if (hq >= 0)
        {
            const double* const C = bs.cen + 3 * hs.z;
            const double* const D = bs.cen + 3 * hs.w;
            const double CDx = C[0] - D[0], CDy = C[1] - D[1], CDz = C[2] - D[2];
            for (int e = warp; e < NE; e += NW)
                Cls::hrr_ket(hA + e * NF * 32 + lane, hB + e * NCD * 32 + lane, CDx, CDy, CDz);
        }
        __syncthreads();
        // the bra recurrence of W neighbouring columns at a time into the stage space, one column per warp and lane,
        // then out quartet by quartet: a quartet's runs of W values go out by neighbouring lanes.  (Each lane
        // storing its own column wrote 8 bytes at 32 places, on 32 pages, per instruction: 4.3k of 22k cycles per
        // primitive quartet of (dd|dd), 1.5k so.)
        constexpr int NAB = ncart(Cls::LA) * ncart(Cls::LB), W = NCD < NW ? NCD : NW;
        static_assert(NAB * W * 33 <= Cls::kStageSpace, "the columns fit the stage space");
        for (int c0 = 0; c0 < NCD; c0 += W)
        {
            const int width = c0 + W < NCD ? W : NCD - c0;
            if (hq >= 0 && warp < width)
            {
                const double* const A = bs.cen + 3 * hs.x;
                const double* const B = bs.cen + 3 * hs.y;
                const double ABx = A[0] - B[0], ABy = A[1] - B[1], ABz = A[2] - B[2];
                Cls::hrr_bra(hB + (c0 + warp) * 32 + lane, qcg_team_smem + warp * 33 + lane, W * 33, ABx, ABy, ABz);
            }
            __syncthreads();
            for (int l = warp; l < 32; l += NW)
            {
                const int lq = lane_q[l];
                if (lq < 0) continue;
                OT* const o = out + lq * BLK + c0;
                for (int k = lane; k < NAB * width; k += 32)
                {
                    const int ab = k / width, c = k - ab * width;
                    o[ab * NCD + c] = (OT)qcg_team_smem[(ab * W + c) * 33 + l];
                }
            }
            __syncthreads();
        }
    }
}

}   // namespace qcg

#include "jk_group.cuh"

namespace qcg {

// ------------------------------------------------------------------------------------------------
// The team form of the direct J/K build (contracted classes; uncontracted ones: jk_group.cuh).  The same stages
// and contraction on 32 quartets at a time, in the class's own order for this form (JKTeamListDev: quartets of equal
// primitive-loop length together, longest first, in a small build cut into runs of bra primitive pairs, each
// digested by itself, which the linearity of J and K allows) or in that of its screened work list; lane l takes
// item gbeg + 32 g + l, its entry found by binary search.  The stages are built from the primitive-pair table; then the digestion of [e0|f0] into J' and K' (team_digest), the (c d) columns split over the warps.
// This replaces qchem's MakeDirect/MakeExchange + ERI4::MatMul (Molecule/IrrepBasisSet.C:138-183,
// Internal/Imp/ERI4.C:10-17) without storing the integrals.
// ------------------------------------------------------------------------------------------------
template <class Cls, bool DET>
__global__ void __launch_bounds__(Cls::kNW * 32, Cls::kMinBlocks)
    jk_team_kernel(JKWorkDev w, PairListDev bra, PairListDev ket, PrimPairsDev P, const int* __restrict__ shell_f0,
                   const double* __restrict__ D, double* __restrict__ J, double* __restrict__ K, int n,
                   const double* __restrict__ boys_table, TeamScratchDev scr)
{
    constexpr int NW = Cls::kNW;
    constexpr int NF = Cls::kNF, NE = Cls::kNE;
    constexpr int STAGE = Cls::kStage * 32;
    constexpr int NCD = ncart(Cls::LC) * ncart(Cls::LD);
    __shared__ uint64_t full[3];
    __shared__ int done[3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool leader = threadIdx.x == 0;
    if (leader)
    {
        for (int s = 0; s < 3; ++s)
        {
            team::mbar_init(&full[s]);
            done[s] = 0;
        }
        team::mbar_init_fence();
    }
    const BoysColumns bt = team_boys<Cls>(qcg_team_smem + Cls::kStageSpace, boys_table);
    __syncthreads();
    double* const rc = scr.rcache + (long long)blockIdx.x * scr.kmax * STAGE;
    double* const hA = scr.hrr + (long long)blockIdx.x * NE * NF * 32;
    TeamRing ring{full, done};
    const JKTeamListDev& list = scr.list;
    const long long* const offs = list.n ? list.offs : w.offs;
    const long long gend = list.n ? list.total : w.gend, gbeg = list.n ? 0 : w.gbeg;
    const long long ngroups = (gend - gbeg + 31) >> 5;
    for (long long g = blockIdx.x; g < ngroups; g += gridDim.x)
    {
        const long long gq = gbeg + g * 32 + lane;
        bool valid = gq < gend;
        int i = 0, j = 0, p0 = 0, Kab = 0, Kcd = 0;
        if (valid)
        {
            int lo = 0, hi = list.n ? list.n : bra.n;   // entry or bra pair: offs[lo] <= gq < offs[lo + 1]
            while (hi - lo > 1)
            {
                const int mid = (lo + hi) >> 1;
                if (offs[mid] <= gq) lo = mid;
                else hi = mid;
            }
            const int pos = (int)(gq - offs[lo]);
            if (list.n)
            {
                const int4 e = list.entry[lo];
                i = e.x;
                p0 = e.y;
                Kab = e.z;
                j = list.kets[e.w + pos];
            }
            else
            {
                i = lo;
                Kab = bra.npp[i];
                j = (w.kbase ? w.kbase[i] : 0) + pos;
            }
            Kcd = ket.npp[j];
            if ((w.mol_active && bra.mol && !w.mol_active[bra.mol[i]]) ||
                jk_skip(w, bra, ket, i, j, bra.sa[i], bra.sb[i], ket.sa[j], ket.sb[j]))
            {
                valid = false;
                Kab = Kcd = 0;
            }
        }
        const int Kq = Kab * Kcd;
        const int Kg = __reduce_max_sync(0xffffffffu, Kq);   // CTA-uniform: every warp sees the same lanes
        if (Kg == 0) continue;                               // every quartet of the group skipped
        if (Kg > scr.kmax)
        {
            if (leader) atomicOr(scr.err, 2);
            continue;
        }
        // 1. stage tables, from the primitive-pair table
        team_stages<Cls>(
            rc, Kab, Kcd, Kg, bt, [&](int ij) { return load_pp(P, bra.ppo[i] + p0 + ij); },
            [&](int kl) { return load_pp(P, ket.ppo[j] + kl); });
        // 2. contraction (as in eri_batch_team_kernel)
        if (!team_contract<Cls>(rc, hA, Kq, Kcd, Kg, ring, scr.err)) return;
        // 3. recurrences and digestion, the (c d) columns in runs of neighbours over the warps
        constexpr int PER = (NCD + NW - 1) / NW;
        const int cd0 = warp * PER, cd1 = cd0 + PER < NCD ? cd0 + PER : NCD;
        if (cd0 < NCD)
            team_digest<Cls, DET>(w, bra, ket, P, shell_f0, D, J, K, n, hA + lane, valid, i, j, cd0, cd1, lane);
        __syncthreads();   // the scratch and the R cache are free for the next group
    }
}

}   // namespace qcg
