// jk_group.cuh -- the team form of the direct J/K build for uncontracted classes (one primitive quartet per
// quartet): jk_group_kernel.
//
// With a single primitive quartet per lane there is no primitive loop to share: in jk_team_kernel one warp
// makes the only stage of a group of 32 quartets while the others wait, the stage travels through global
// memory, and every warp repeats the search for the lanes' bra pairs.  Here a CTA takes up to kGroups groups of 32
// quartets at a time, as many as their stages fit the shared memory, and its warps
//   make      (group)        the lanes' quartets and the stage tables, into shared memory;
//   contract  (piece, group, rotation)   Y_f and [e0|f], as in jk_team_kernel (gen_md.py, team form), to the
//                            CTA's scratch.  Tasks are drawn from a counter, piece by piece, so that warps at work
//                            side by side walk the same code;
//   digest    (group)        per (c d) column the ket recurrence as at most four terms of [e0|f0] rows (a table: one
//                            code for every row), the bra recurrence in registers, and its results straight into the
//                            J/K sums, without the [e0|cd] and (ab|cd) blocks in memory.  With fewer groups than
//                            warps a group's c components are split over several tasks.
// The 32 quartets of a group are neighbours in the work list and mostly share their bra pair: then J'(a b) is
// summed over the warp by shuffles and written once per warp instead of once per lane.
#pragma once
#include "eri_kernels.cuh"
#include "eri_team.cuh"

namespace qcg {

// Sum of V values over the 32 lanes, eight at a time: three exchange steps in which each lane keeps half of its
// values, two butterfly steps, then write(k, total of value k) on one lane per value.
template <int V, class Write>
__device__ __forceinline__ void warp_sums(const double (&v)[V], int lane, Write write)
{
#pragma unroll
    for (int k0 = 0; k0 < V; k0 += 8)
    {
        double t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = k0 + k < V ? v[k0 + k < V ? k0 + k : 0] : 0.0;
#pragma unroll
        for (int m = 8, o = 16; m > 1; m >>= 1, o >>= 1)
        {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < m / 2; ++k)
            {
                const double send = up ? t[k] : t[k + m / 2];
                const double keep = up ? t[k + m / 2] : t[k];
                t[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        double x = t[0];
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        const int k = k0 + (lane >> 2);
        if ((lane & 3) == 0 && k < V) write(k, x);
    }
}

// the factor of one term of the ket recurrence (the code in the upper byte of a Cls::column field)
__device__ __forceinline__ double column_factor(int code, const double (&d)[3])
{
    switch (code)
    {
    case 2: return d[0];
    case 3: return d[1];
    case 4: return d[2];
    case 5: return 2.0 * d[0];
    case 6: return 2.0 * d[1];
    case 7: return 2.0 * d[2];
    case 8: return d[0] * d[0];
    case 9: return d[1] * d[1];
    case 10: return d[2] * d[2];
    case 11: return d[0] * d[1];
    case 12: return d[1] * d[2];
    case 13: return d[0] * d[2];
    default: return 1.0;
    }
}

// Digestion of the (c d) columns [cd0, cd1) of this lane's quartet (bra pair i, ket pair j) into J' and K': h
// points at the lane's entry of row 0, column 0 of [e0|f0].  Per column the ket recurrence as at most four terms
// of [e0|f0] columns (Cls::column: warp-uniform, one code for every column), the bra recurrence in registers
// and its results straight into the sink.  Every lane of the warp calls it; lanes without a quartet (valid
// false) only take part in the sum of J'(a b), which goes over the warp by shuffles and is written once where
// its quartets share the bra pair (not in the deterministic mode, which rounds each quartet's contribution
// alone).
template <class Cls, bool DET>
__device__ __forceinline__ void team_digest(const JKWorkDev& w, const PairListDev& bra, const PairListDev& ket,
                                            const PrimPairsDev& P, const int* __restrict__ shell_f0,
                                            const double* __restrict__ D, double* __restrict__ J,
                                            double* __restrict__ K, int n, const double* h, bool valid,
                                            int i, int j, int cd0, int cd1, int lane)
{
    constexpr int NE = Cls::kNE, NF = Cls::kNF;
    constexpr int NB = ncart(Cls::LB), ND = ncart(Cls::LD), NAB = ncart(Cls::LA) * NB;
    JKSink<double, Cls::LA, Cls::LB, Cls::LC, Cls::LD, DET> sink;
    sink.D = D;
    sink.J = J;
    sink.K = K;
    sink.n = n;
    sink.set_bra(0, 0);
    if constexpr (DET) sink.det_lo = w.det_lo;
    if (valid)
    {
        const int sa = bra.sa[i], sb = bra.sb[i], sc = ket.sa[j], sd = ket.sb[j];
        if (bra.mol)
        {
            const int m = bra.mol[i];
            const long long o = w.mols.off[m];
            sink.D = D + o;
            sink.J = J + o;
            sink.K = K + o;
            sink.n = w.mols.n[m];
        }
        sink.fa = shell_f0[sa];
        sink.fb = shell_f0[sb];
        sink.fc = shell_f0[sc];
        sink.fd = shell_f0[sd];
        sink.s = (sa == sb ? 0.5 : 1.0) * (sc == sd ? 0.5 : 1.0) * ((w.same_class && i == j) ? 0.5 : 1.0);
        // C - D = (P - D) - (P - C) and A - B = (P - B) - (P - A), from the shell pairs' first primitive pairs
        const int kp = ket.ppo[j], bp = bra.ppo[i];
        const double CD[3] = {P.PBx[kp] - P.PAx[kp], P.PBy[kp] - P.PAy[kp], P.PBz[kp] - P.PAz[kp]};
        const double ABx = P.PBx[bp] - P.PAx[bp], ABy = P.PBy[bp] - P.PAy[bp], ABz = P.PBz[bp] - P.PAz[bp];
#pragma unroll 1
        for (int cd = cd0; cd < cd1; ++cd)
        {
            const int ic = cd / ND, id = cd - ic * ND;
            double y[NE];
            const unsigned long long col = Cls::column(cd);
            const double nrm = Cls::column_norm(cd);
            {
                const double c0 = nrm * column_factor((int)(col >> 8) & 255, CD);
                const double* const p = h + (int)(col & 255) * 32;
#pragma unroll
                for (int e = 0; e < NE; ++e) y[e] = c0 * p[e * NF * 32];
            }
            if constexpr (Cls::LD > 0)
#pragma unroll 1
                for (unsigned long long c = col >> 16; c & 0xff00; c >>= 16)
                {
                    const double ck = nrm * column_factor((int)(c >> 8) & 255, CD);
                    const double* const p = h + (int)(c & 255) * 32;
#pragma unroll
                    for (int e = 0; e < NE; ++e) y[e] = fma(ck, p[e * NF * 32], y[e]);
                }
            sink.ket_begin(ic, id);
            Cls::bra_out(y, ABx, ABy, ABz, [&](int ia, int ib, double x) { sink(ia, ib, ic, id, x); });
            sink.ket_end(ic, id);
        }
        sink.flush_k_row();
    }
    __syncwarp();
    if constexpr (!DET)
    {
        const unsigned m = __ballot_sync(0xffffffffu, valid);
        const int src = m ? __ffs(m) - 1 : 0;
        const int i0 = __shfl_sync(0xffffffffu, i, src);
        if (__all_sync(0xffffffffu, !valid || i == i0))
        {
            const int fa = __shfl_sync(0xffffffffu, sink.fa, src), fb = __shfl_sync(0xffffffffu, sink.fb, src);
            const int nn = __shfl_sync(0xffffffffu, sink.n, src);
            const long long o = __shfl_sync(0xffffffffu, (long long)(sink.J - J), src);
            warp_sums<NAB>(sink.jab, lane, [&](int k, double x) {
                const int ia = k / NB, ib = k - ia * NB;
                if (x != 0.0) atomicAdd(J + o + (size_t)(fa + ia) * nn + fb + ib, 2.0 * x);
            });
            return;
        }
    }
    if (valid) sink.flush_bra();
}

// The digestion of jk_group_kernel: rows [ic0, ic1) of c components of this lane's quartet, every d component of each.
// K'(a d) and K'(b d) stay in registers over the rows (kWholeRows: where they fit) and leave once per call, K'(a c)
// and K'(b c) once per row: (dp|pp) updates J' and K' 63 times per quartet and lane where a call per row and an update
// per column made 117.  What bounds it is latency: with eight warps of 255 registers an SM issues in one cycle of five,
// the warps waiting for loads of D and [e0|f0] (long scoreboard 3.7-4.3 cycles per issue) and, in (dp|ds), behind the
// queue of updates (1.9); the updates run at 0.6-1.2e11 per second, where (pp|pp) thread-per-quartet reaches 1.9e11.
template <class Cls, bool DET>
struct RowSink
{
    static constexpr int NA = ncart(Cls::LA), NB = ncart(Cls::LB), ND = ncart(Cls::LD), NAB = NA * NB;
    const double* __restrict__ D;
    double* __restrict__ J;
    double* __restrict__ K;
    int n, fa, fb, fc, fd;
    double s;
    long long det_lo = 0;
    double jab[NAB], kac[NA], kbc[NB], kad[NA * ND], kbd[NB * ND], jcd;
    double dls, das[NA], dal[NA], dbs[NB], dbl[NB];

    __device__ __forceinline__ void acc(double* M, size_t k, double v)
    {
        if constexpr (DET) fixed_add(M, k, det_lo, v);
        else atomicAdd(M + k, v);
    }
    __device__ __forceinline__ void row_begin(int la)
    {
#pragma unroll
        for (int k = 0; k < NA; ++k)
        {
            dal[k] = __ldg(D + (size_t)(fa + k) * n + la);
            kac[k] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < NB; ++k)
        {
            dbl[k] = __ldg(D + (size_t)(fb + k) * n + la);
            kbc[k] = 0.0;
        }
    }
    __device__ __forceinline__ void column_begin(int la, int id)
    {
        const int si = fd + id;
        dls = __ldg(D + (size_t)la * n + si);
        jcd = 0.0;
#pragma unroll
        for (int k = 0; k < NA; ++k) das[k] = __ldg(D + (size_t)(fa + k) * n + si);
#pragma unroll
        for (int k = 0; k < NB; ++k) dbs[k] = __ldg(D + (size_t)(fb + k) * n + si);
    }
    __device__ __forceinline__ void add(int ia, int ib, int id, double v)
    {
        const double w = s * v;
        jab[ia * NB + ib] += w * dls;
        jcd += w * __ldg(D + (size_t)(fa + ia) * n + fb + ib);
        kac[ia] += w * dbs[ib];
        kbc[ib] += w * das[ia];
        kad[ia * ND + id] += w * dbl[ib];
        kbd[ib * ND + id] += w * dal[ia];
    }
    __device__ __forceinline__ void flush_d(int id)
    {
#pragma unroll
        for (int k = 0; k < NA; ++k)
        {
            acc(K, (size_t)(fa + k) * n + fd + id, kad[k * ND + id]);
            kad[k * ND + id] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < NB; ++k)
        {
            acc(K, (size_t)(fb + k) * n + fd + id, kbd[k * ND + id]);
            kbd[k * ND + id] = 0.0;
        }
    }
    __device__ __forceinline__ void row_end(int la)
    {
#pragma unroll
        for (int k = 0; k < NA; ++k) acc(K, (size_t)(fa + k) * n + la, kac[k]);
#pragma unroll
        for (int k = 0; k < NB; ++k) acc(K, (size_t)(fb + k) * n + la, kbc[k]);
    }
};

template <class Cls, bool DET>
__device__ __forceinline__ void team_digest_rows(const JKWorkDev& w, const PairListDev& bra, const PairListDev& ket,
                                                 const PrimPairsDev& P, const int* __restrict__ shell_f0,
                                                 const double* __restrict__ D, double* __restrict__ J,
                                                 double* __restrict__ K, int n, const double* h, bool valid,
                                                 int i, int j, int ic0, int ic1, int lane)
{
    constexpr int NE = Cls::kNE, NF = Cls::kNF;
    constexpr int NA = ncart(Cls::LA), NB = ncart(Cls::LB), ND = ncart(Cls::LD), NAB = NA * NB;
    constexpr bool kWholeRows = (NA + NB) * ND <= 36;
    RowSink<Cls, DET> sink;
    sink.D = D;
    sink.J = J;
    sink.K = K;
    sink.n = n;
    sink.fa = sink.fb = 0;
#pragma unroll
    for (int k = 0; k < NAB; ++k) sink.jab[k] = 0.0;
    if constexpr (DET) sink.det_lo = w.det_lo;
    if (valid)
    {
        const int sa = bra.sa[i], sb = bra.sb[i], sc = ket.sa[j], sd = ket.sb[j];
        if (bra.mol)
        {
            const int m = bra.mol[i];
            const long long o = w.mols.off[m];
            sink.D = D + o;
            sink.J = J + o;
            sink.K = K + o;
            sink.n = w.mols.n[m];
        }
        sink.fa = shell_f0[sa];
        sink.fb = shell_f0[sb];
        sink.fc = shell_f0[sc];
        sink.fd = shell_f0[sd];
        sink.s = (sa == sb ? 0.5 : 1.0) * (sc == sd ? 0.5 : 1.0) * ((w.same_class && i == j) ? 0.5 : 1.0);
        // C - D = (P - D) - (P - C) and A - B = (P - B) - (P - A)
        const int kp = ket.ppo[j], bp = bra.ppo[i];
        const double CD[3] = {P.PBx[kp] - P.PAx[kp], P.PBy[kp] - P.PAy[kp], P.PBz[kp] - P.PAz[kp]};
        const double ABx = P.PBx[bp] - P.PAx[bp], ABy = P.PBy[bp] - P.PAy[bp], ABz = P.PBz[bp] - P.PAz[bp];
#pragma unroll
        for (int k = 0; k < NA * ND; ++k) sink.kad[k] = 0.0;
#pragma unroll
        for (int k = 0; k < NB * ND; ++k) sink.kbd[k] = 0.0;
#pragma unroll 1
        for (int ic = ic0; ic < ic1; ++ic)
        {
            const int la = sink.fc + ic;
            sink.row_begin(la);
#pragma unroll
            for (int id = 0; id < ND; ++id)
            {
                double y[NE];
                const unsigned long long col = Cls::column(ic * ND + id);
                const double nrm = Cls::column_norm(ic * ND + id);
                {
                    const double c0 = nrm * column_factor((int)(col >> 8) & 255, CD);
                    const double* const p = h + (int)(col & 255) * 32;
#pragma unroll
                    for (int e = 0; e < NE; ++e) y[e] = c0 * p[e * NF * 32];
                }
                if constexpr (Cls::LD > 0)
#pragma unroll 1
                    for (unsigned long long c = col >> 16; c & 0xff00; c >>= 16)
                    {
                        const double ck = nrm * column_factor((int)(c >> 8) & 255, CD);
                        const double* const p = h + (int)(c & 255) * 32;
#pragma unroll
                        for (int e = 0; e < NE; ++e) y[e] = fma(ck, p[e * NF * 32], y[e]);
                    }
                sink.column_begin(la, id);
                Cls::bra_out(y, ABx, ABy, ABz, [&](int ia, int ib, double x) { sink.add(ia, ib, id, x); });
                sink.acc(sink.J, (size_t)la * sink.n + sink.fd + id, 2.0 * sink.jcd);
                if constexpr (!kWholeRows) sink.flush_d(id);
            }
            sink.row_end(la);
        }
        if constexpr (kWholeRows)
        {
#pragma unroll
            for (int id = 0; id < ND; ++id) sink.flush_d(id);
        }
    }
    __syncwarp();
    // J'(a b): over the warp where its quartets share the bra pair (see team_digest)
    if constexpr (!DET)
    {
        const unsigned m = __ballot_sync(0xffffffffu, valid);
        const int src = m ? __ffs(m) - 1 : 0;
        const int i0 = __shfl_sync(0xffffffffu, i, src);
        if (__all_sync(0xffffffffu, !valid || i == i0))
        {
            const int fa = __shfl_sync(0xffffffffu, sink.fa, src), fb = __shfl_sync(0xffffffffu, sink.fb, src);
            const int nn = __shfl_sync(0xffffffffu, sink.n, src);
            const long long o = __shfl_sync(0xffffffffu, (long long)(sink.J - J), src);
            warp_sums<NAB>(sink.jab, lane, [&](int k, double x) {
                const int ia = k / NB, ib = k - ia * NB;
                if (x != 0.0) atomicAdd(J + o + (size_t)(fa + ia) * nn + fb + ib, 2.0 * x);
            });
            return;
        }
    }
    if (valid)
    {
#pragma unroll
        for (int k = 0; k < NAB; ++k)
            if (sink.jab[k] != 0.0) sink.acc(sink.J, (size_t)(sink.fa + k / NB) * sink.n + sink.fb + k % NB, 2.0 * sink.jab[k]);
    }
}

template <class Cls, bool DET>
__global__ void __launch_bounds__(Cls::kJKWarps * 32, Cls::kJKBlocks)
    jk_group_kernel(JKWorkDev w, PairListDev bra, PairListDev ket, PrimPairsDev P, const int* __restrict__ shell_f0,
                    const double* __restrict__ D, double* __restrict__ J, double* __restrict__ K, int n,
                    const double* __restrict__ boys_table, double* __restrict__ scratch, const int ngrp)
{
    constexpr int NGRP = Cls::kGroups, STAGE = Cls::kStage * 32;
    constexpr int NE = Cls::kNE, NF = Cls::kNF, NH = Cls::kNH, NC = Cls::kNCode;
    constexpr int NCc = ncart(Cls::LC);
    __shared__ int2 quartet[NGRP][32];   // (bra pair, ket pair) of each lane; bra -1: no quartet
    __shared__ int live[NGRP];           // whether a group has any quartet
    __shared__ int counter[2];
    const int lane = threadIdx.x & 31;
    const BoysColumns bt = team_boys<Cls>(qcg_team_smem + NGRP * STAGE, boys_table);
    if (threadIdx.x < 2) counter[threadIdx.x] = 0;
    __syncthreads();
    double* const hA = scratch + (long long)blockIdx.x * ngrp * NE * NF * 32;
    auto draw = [&](int c) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&counter[c], 1);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    const long long ngroups = (w.gend - w.gbeg + 31) >> 5;
    const long long nround = (ngroups + ngrp - 1) / ngrp;   // rounds of ngrp <= NGRP groups

    // the lanes' quartets and the stage of group s of round r
    auto make = [&](long long r, int s) {
        const long long gq = w.gbeg + (r * ngrp + s) * 32 + lane;
        bool valid = gq < w.gend;
        int i = 0, j = 0;
        if (valid)
        {
            int lo = 0, hi = bra.n;   // bra pair i: offs[i] <= gq < offs[i+1]
            while (hi - lo > 1)
            {
                const int mid = (lo + hi) >> 1;
                if (w.offs[mid] <= gq) lo = mid;
                else hi = mid;
            }
            i = lo;
            j = (w.kbase ? w.kbase[i] : 0) + (int)(gq - w.offs[i]);
            if (w.mol_active && bra.mol && !w.mol_active[bra.mol[i]]) valid = false;
            else if (jk_skip(w, bra, ket, i, j, bra.sa[i], bra.sb[i], ket.sa[j], ket.sb[j])) valid = false;
        }
        quartet[s][lane] = make_int2(valid ? i : -1, j);
        const bool any = __any_sync(0xffffffffu, valid);
        if (lane == 0) live[s] = any;
        if (valid)
            Cls::produce(qcg_team_smem + s * STAGE + lane, team_pair(load_pp(P, bra.ppo[i])),
                         team_pair(load_pp(P, ket.ppo[j])), bt, true);
    };

    // a digestion task is a group, or with fewer groups than warps a part of its rows; in the deterministic mode, which
    // rounds a task's K'(a d), K'(b d) and J'(a b), the parts are those of a full round whatever its groups
    const int parts = min(NCc, max(1, Cls::kJKWarps / (DET ? NGRP : ngrp))), rows = (NCc + parts - 1) / parts;
    for (long long r = blockIdx.x; r < nround; r += gridDim.x)
    {
        for (int s = threadIdx.x >> 5; s < ngrp; s += Cls::kJKWarps) make(r, s);
        if (threadIdx.x == 0) counter[1] = 0;   // last used before the barrier that ended the round
        __syncthreads();
        // contraction
        for (;;)
        {
            const int t = draw(0);
            if (t >= NC * ngrp * 3) break;
            const int jc = t / (ngrp * 3), u = t - jc * (ngrp * 3), s = u / 3, rot = u - 3 * s;
            if (!live[s] || (rot != 0 && Cls::fixed(jc))) continue;
            if (quartet[s][lane].x >= 0)
            {
                const typename Cls::View v(qcg_team_smem + s * STAGE + lane, rot);
                double Y[NH], acc[NE];
#pragma unroll
                for (int h = 0; h < NH; ++h) Y[h] = 0.0;
#pragma unroll
                for (int e = 0; e < NE; ++e) acc[e] = 0.0;
                Cls::ket(jc, v, Y);
                Cls::bra(v, Y, acc);
                Cls::store(acc, hA + (s * NE * NF + Cls::fslot(jc) + rot) * 32 + lane, rot);
            }
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x == 0) counter[0] = 0;
        // digestion
        for (;;)
        {
            const int t = draw(1);
            if (t >= ngrp * parts) break;
            const int s = t / parts, ic0 = (t - s * parts) * rows;
            if (!live[s] || ic0 >= NCc) continue;
            const int2 q = quartet[s][lane];
            team_digest_rows<Cls, DET>(w, bra, ket, P, shell_f0, D, J, K, n, hA + s * NE * NF * 32 + lane, q.x >= 0, q.x,
                                       q.y, ic0, min(ic0 + rows, NCc), lane);
        }
        __syncthreads();
    }
}

}   // namespace qcg
