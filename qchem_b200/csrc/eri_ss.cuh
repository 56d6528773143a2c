// eri_ss.cuh -- ERI batches of the classes with an (ss) ket, (xx|ss): eri_ss_kernel.
//
// With an (ss) ket there is one ket component, so the team form has nothing to split over warps, and with at
// most 36 integrals a quartet fits one thread: Y[h], the Hermite integrals summed over the ket primitives of one
// bra primitive pair, and acc[e] = [e0|ss] stay in registers (70 + 62 for a (dd| bra), the bra contraction runs
// once per bra primitive pair and the bra recurrence once per quartet.  (The direct form evaluated (ab|ss) per
// primitive quartet and added it to the output block in memory: 250 000 quartets of (dd|ss), contractions of one to
// three, 1250 us where this takes 243, of (ss|ss) 334 and 143, sort included.)  What bounds it is the FP64 latency of the
// Boys function and the R recursion: issue 33%, FP64 pipe 37% and 22%, eight and thirteen warps per SM.
//
// A warp takes 32 / SPLIT quartets, SPLIT neighbouring lanes sharing one: lane s of a quartet takes the bra
// primitive pairs s, s + SPLIT, ..., and the lanes' acc are added by shuffles.  The ket primitive pairs of the
// warp's quartets are formed once per quartet into shared memory, by the lanes in turn.
#pragma once
#include "eri_kernels.cuh"
#include "eri_team.cuh"

namespace qcg {

constexpr int kSSThreads = 128, kSSKetSlots = 9;   // ket primitive pairs kept per quartet (contractions of three)
constexpr int kSSKetDoubles = 5;                   // p, P, K / p

template <class Cls, class OT, int SPLIT>
__global__ void __launch_bounds__(kSSThreads)
    eri_ss_kernel(BasisDev bs, const int4* __restrict__ quartets, const int* __restrict__ order, long long nq,
                  OT* __restrict__ out, const double* __restrict__ boys_table)
{
    constexpr int NE = Cls::kNE, NH = Cls::kNH, NAB = ncart(Cls::LA) * ncart(Cls::LB), QW = 32 / SPLIT;
    double* const smem = qcg_team_smem;
    const BoysColumns bt = team_boys<Cls>(smem, boys_table);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane % SPLIT;
    // slot t, field f of the lane's quartet: kets[(t * kSSKetDoubles + f) * QW]
    double* const kets = smem + kBoysRows * kBoysColumns + warp * (kSSKetSlots * kSSKetDoubles * QW) + lane / SPLIT;
    const long long nwarp = (long long)gridDim.x * (kSSThreads / 32);
    for (long long g = blockIdx.x * (long long)(kSSThreads / 32) + warp; g * QW < nq; g += nwarp)
    {
        const long long gi = g * QW + lane / SPLIT;
        const bool valid = gi < nq;
        const long long q = valid ? (order ? (long long)order[gi] : gi) : 0;
        const int4 s = quartets[q];
        const int nj = bs.nprim[s.y], nl = bs.nprim[s.w];
        const int Kab = valid ? bs.nprim[s.x] * nj : 0, Kcd = valid ? bs.nprim[s.z] * nl : 0;
        __syncwarp();   // the previous quartets' ket pairs are no longer read
        for (int t = sub; t < Kcd && t < kSSKetSlots; t += SPLIT)
        {
            const TeamPair d = team_pair(shell_prim_pair(bs, s.z, t / nl, s.w, t % nl));
            double* const k = kets + t * kSSKetDoubles * QW;
            k[0] = d.p; k[QW] = d.Px; k[2 * QW] = d.Py; k[3 * QW] = d.Pz; k[4 * QW] = d.kp;
        }
        __syncwarp();
        double acc[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.0;
        for (int ij = sub; ij < Kab; ij += SPLIT)
        {
            const TeamPair ab = team_pair(shell_prim_pair(bs, s.x, ij / nj, s.y, ij % nj));
            double Y[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) Y[h] = 0.0;
            for (int t = 0; t < Kcd; ++t)
            {
                TeamPair cd;
                if (t < kSSKetSlots)
                {
                    const double* const k = kets + t * kSSKetDoubles * QW;
                    cd = TeamPair{k[0], k[QW], k[2 * QW], k[3 * QW], 0.0, 0.0, 0.0, k[4 * QW], 0.0};
                }
                else
                    cd = team_pair(shell_prim_pair(bs, s.z, t / nl, s.w, t % nl));
                Cls::hermite_add(ab, cd, bt, Y);
            }
            Cls::bra_pair(ab, Y, acc);
        }
        if constexpr (SPLIT > 1)
        {
#pragma unroll
            for (int e = 0; e < NE; ++e)
#pragma unroll
                for (int o = SPLIT / 2; o >= 1; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
        }
        if (valid && sub == 0)
        {
            const double* const A = bs.cen + 3 * s.x;
            const double* const B = bs.cen + 3 * s.y;
            constexpr int NB = ncart(Cls::LB);
            OT* const o = out + q * NAB;
            Cls::bra_out(acc, A[0] - B[0], A[1] - B[1], A[2] - B[2],
                         [&](int ia, int ib, double x) { o[ia * NB + ib] = (OT)x; });
        }
    }
}

}   // namespace qcg
