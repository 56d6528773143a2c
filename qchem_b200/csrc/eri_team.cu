// eri_team.cu -- the team form of the FP64 ERI batches (eri_team.cuh) for ONE quartet class; compiled with
// -DQCG_CLASS=k for every class, defining launch_eri_team_k and team_shape_k.  The generated code comes from
// gen/md_team_<k>.cuh (stage tables, ket and bra steps, recurrences).
#include <algorithm>
#include <atomic>

#include "eri_kernels.cuh"
#include "eri_team.cuh"
#include "smem_attr.h"

#ifndef QCG_CLASS
#error "compile with -DQCG_CLASS=<0..20>"
#endif

#define QCG_STR2(x) #x
#define QCG_STR(x) QCG_STR2(x)
#define QCG_CAT2(a, b) a##b
#define QCG_CAT(a, b) QCG_CAT2(a, b)
#include QCG_STR(gen/QCG_CAT(md_team_, QCG_CLASS).cuh)

// the classes whose ket pair is (ss): X (X + 1) / 2
#define QCG_SS_KET (QCG_CLASS == 0 || QCG_CLASS == 1 || QCG_CLASS == 3 || QCG_CLASS == 6 || QCG_CLASS == 10 || QCG_CLASS == 15)
#if QCG_SS_KET
#include "eri_ss.cuh"
#endif

namespace qcg {

namespace {
constexpr int cls_X()
{
    int X = 0;
    while ((X + 1) * (X + 2) / 2 <= QCG_CLASS) ++X;
    return X;
}
constexpr int kX = cls_X();
constexpr int kY = QCG_CLASS - kX * (kX + 1) / 2;

// Pieces of ket code per pass (kNG; each runs on three warps, one per rotation).  With a piece per component, 31 for
// (dd|dd), four warps on four pieces outran eight on eight, because the code in flight has to fit the instruction
// cache: 8 passes, 19.2 ms for 250 000 quartets.  With a piece per orbit twelve warps run four pieces: 3 passes,
// 12.1 ms, and no_instruction fell from 24% of the stall samples to 2%.  A thread keeps Y_f and acc_f
// in registers, and the SM's 65 536 registers are split among four schedulers, so ceil(3 g / 4) warps per
// scheduler leave each thread 512 / ceil(3 g / 4) registers (255 at most): g is the largest for which Y_f, acc_f
// and kTemps further registers fit, and the pieces are then spread evenly over the passes.
constexpr int kTemps = 36;

constexpr int warp_regs(int g)
{
    const int per = (3 * g + 3) / 4, r = 512 / per / 8 * 8;
    return r > 255 ? 255 : r;
}
constexpr int team_pieces(int ncode, int nh, int ne)
{
    int g = 1;
    for (int x = 2; x <= 8 && x <= ncode; ++x)
        if (warp_regs(x) >= 2 * (nh + ne) + kTemps) g = x;
    const int npass = (ncode + g - 1) / g;
    return (ncode + npass - 1) / npass;
}
// CTAs per SM to compile for: twelve warps or more, as far as the registers go round and three stages each fit the
// shared memory, of which a CTA may then use kSmemPerSM / m bytes less what it holds beside the stages.  (Nine warps in
// one CTA, the (pp|pp) and (ds|pp) classes, wait together between the phases of a group: 250 000 quartets of
// contraction three 1068 and 1026 us, in two CTAs 853 and 799; of contraction two 612 and 562, 466 and 413.  With half the stages
// per slot a lone group of long loops is slower: 32 quartets of contraction eight 96 and 87, 123 and 112.)
constexpr int kSmemPerSM = 227 * 1024;
constexpr int kSmemBeside = 2048 + (int)sizeof(BatchPlanDev) + (int)(kBoysRows * kBoysColumns * sizeof(double));
constexpr int team_min_blocks(int ng, int stage, int regs)
{
    const int fit = kSmemPerSM / (3 * stage * 32 * 8 + kSmemBeside), want = (12 + 3 * ng - 1) / (3 * ng);
    int m = fit < want ? fit : want;
    while (m > 1 && warp_regs(ng * m) < regs) --m;
    return m < 1 ? 1 : m;
}
// stages per slot of the ring (team_contract): what three slots leave room for, eight at most
constexpr int team_unroll(int ng, int stage, int regs)
{
    const int u = (kSmemPerSM / team_min_blocks(ng, stage, regs) - kSmemBeside) / (3 * stage * 32 * 8);
    return u < 1 ? 1 : (u > 8 ? 8 : u);
}
// Doubles of the stage space: three slots, and at least 18 primitive pairs (contractions of three) and the columns
// of the bra recurrence that go out together.
constexpr int team_stage_space(int ng, int stage, int regs)
{
    const int ncd = ncart(kPairLA[kY]) * ncart(kPairLB[kY]), nab = ncart(kPairLA[kX]) * ncart(kPairLB[kX]);
    const int columns = nab * (ncd < 3 * ng ? ncd : 3 * ng) * 33, slots = 3 * team_unroll(ng, stage, regs) * stage * 32;
    int n = 18 * kTeamPairDoubles * 32;
    if (n < slots) n = slots;
    return n < columns ? columns : n;
}
constexpr size_t team_smem(int ng, int stage, int regs)
{
    return (size_t)(team_stage_space(ng, stage, regs) + kBoysRows * kBoysColumns) * sizeof(double);
}

struct Cls
{
    static constexpr int LA = kPairLA[kX], LB = kPairLB[kX], LC = kPairLA[kY], LD = kPairLB[kY];
    static constexpr int kNF = gen::QCG_CAT(kTeamNF, QCG_CLASS), kNE = gen::QCG_CAT(kTeamNE, QCG_CLASS);
    static constexpr int kNH = gen::QCG_CAT(kTeamNH, QCG_CLASS), kStage = gen::QCG_CAT(kTeamStage, QCG_CLASS);
    static constexpr int kNCode = gen::QCG_CAT(kTeamNCode, QCG_CLASS);
    static constexpr int kKetStage = gen::QCG_CAT(kTeamKetStage, QCG_CLASS);
    static constexpr int kNG = team_pieces(kNCode, kNH, kNE), kNW = 3 * kNG;
    static constexpr int kRegs = 2 * (kNH + kNE) + kTemps;
    static constexpr int kMinBlocks = team_min_blocks(kNG, kStage, kRegs), kUnroll = team_unroll(kNG, kStage, kRegs);
    // jk_group_kernel: eight warps (the digestion needs more registers than twelve leave), and up to eight groups of 32
    // quartets, one per warp, as far as their stages fit the shared memory
    static constexpr int kGroups = [] {
        const int g = (int)((227 * 1024 - 4096 - (int)(kBoysRows * kBoysColumns * sizeof(double))) /
                            (kStage * 32 * sizeof(double)));
        return g < 1 ? 1 : (g > 8 ? 8 : g);
    }();
    static constexpr int kJKWarps = 8, kJKBlocks = 1;
    static __device__ __forceinline__ unsigned long long column(int cd) { return gen::QCG_CAT(kTeamColumn, QCG_CLASS)[cd]; }
    static __device__ __forceinline__ double column_norm(int cd) { return gen::QCG_CAT(kTeamColumnNorm, QCG_CLASS)[cd]; }
    template <class Sink>
    static __device__ __forceinline__ void bra_out(const double (&y)[kNE], double ABx, double ABy, double ABz, Sink sink)
    {
        gen::QCG_CAT(team_bra_out_, QCG_CLASS)<double>(y, ABx, ABy, ABz, sink);
    }
    using View = gen::QCG_CAT(TeamView, QCG_CLASS)<double>;
    static __device__ __forceinline__ constexpr int fslot(int jc) { return gen::QCG_CAT(team_fslot_, QCG_CLASS)(jc); }
    static __device__ __forceinline__ constexpr bool fixed(int jc) { return gen::QCG_CAT(team_ffixed_, QCG_CLASS)(jc); }
    static constexpr int kStageSpace = team_stage_space(kNG, kStage, kRegs), kPairSlots = kStageSpace / (32 * kTeamPairDoubles);
    static __device__ __forceinline__ void produce(double* st, const TeamPair& ab, const TeamPair& cd,
                                                   const BoysColumns& bt, bool bra_e)
    {
        gen::QCG_CAT(team_produce_, QCG_CLASS)<double>(st, ab, cd, bt, bra_e);
    }
    static __device__ __forceinline__ void ket(int jc, const View& v, double (&Y)[kNH])
    {
        gen::QCG_CAT(team_ket_piece_, QCG_CLASS)<double>(jc, v, Y);
    }
    static __device__ __forceinline__ void bra(const View& v, const double (&Y)[kNH], double (&acc)[kNE])
    {
        gen::QCG_CAT(team_bra_view_, QCG_CLASS)<double>(v, Y, acc);
    }
    static __device__ __forceinline__ void store(const double (&acc)[kNE], double* hA, int rot)
    {
        gen::QCG_CAT(team_store_, QCG_CLASS)<double>(acc, hA, rot);
    }
    static __device__ __forceinline__ void hrr_ket(const double* p, double* y, double CDx, double CDy, double CDz)
    {
        gen::QCG_CAT(team_hrr_ket_, QCG_CLASS)<double>(p, y, CDx, CDy, CDz);
    }
    template <class OT>
    static __device__ __forceinline__ void hrr_bra(const double* y, OT* o, int os, double ABx, double ABy, double ABz)
    {
        gen::QCG_CAT(team_hrr_bra_, QCG_CLASS)<double, OT>(y, o, os, ABx, ABy, ABz);
    }
#if QCG_SS_KET
    static __device__ __forceinline__ void hermite_add(const TeamPair& ab, const TeamPair& cd, const BoysColumns& bt,
                                                       double (&Y)[kNH])
    {
        gen::QCG_CAT(team_hermite_add_, QCG_CLASS)<double>(ab, cd, bt, Y);
    }
    static __device__ __forceinline__ void bra_pair(const TeamPair& ab, const double (&Y)[kNH], double (&acc)[kNE])
    {
        gen::QCG_CAT(team_bra_pair_, QCG_CLASS)<double>(ab, Y, acc);
    }
#endif
};

constexpr int kThreads = Cls::kNW * 32;
constexpr int kNCD = ncart(Cls::LC) * ncart(Cls::LD);
constexpr size_t kSmem = team_smem(Cls::kNG, Cls::kStage, Cls::kRegs);   // the stages and the Boys columns
constexpr size_t kGroupSmem =
    ((size_t)Cls::kGroups * Cls::kStage * 32 + kBoysRows * kBoysColumns) * sizeof(double);
std::atomic<unsigned long long> g_smem_ready{0};
}   // namespace

TeamShape QCG_CAT(team_shape_, QCG_CLASS)(int nsm)
{
    auto k = eri_batch_team_kernel<Cls, double>;
    ensure_smem(k, kSmem, g_smem_ready);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, kSmem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    TeamShape sh;
    sh.grid = nsm * per_sm;
    sh.threads = kThreads;
    sh.nsm = nsm;
    sh.slot_doubles = (long long)Cls::kStage * 32;
    // [e0|f0] and [e0|cd]: lane-minor blocks of the group's 32 quartets (the J/K form: [e0|f0] of its groups)
    sh.hrr_doubles = (long long)Cls::kNE * (Cls::kNF + kNCD) * 32;
    sh.jk_doubles = (long long)Cls::kNE * Cls::kNF * 32;
    sh.group_grid = nsm * Cls::kJKBlocks;
    sh.group_doubles = sh.jk_doubles * Cls::kGroups;
    return sh;
}

namespace {
template <class OT>
void launch_batch(const BasisDev& bs, const int4* q, const int* order, long long nq, OT* out, const double* boys,
                  const TeamScratchDev& scr, const TeamShape& sh, cudaStream_t st)
{
    if (nq <= 0) return;
    auto k = eri_batch_team_kernel<Cls, OT>;
    static std::atomic<unsigned long long> ready{0};
    ensure_smem(k, kSmem, ready);
    // one wave of CTAs, each walking groups of the plan; the scratch has room for sh.grid CTAs
    k<<<(unsigned)sh.grid, kThreads, kSmem, st>>>(bs, q, order, (int)nq, out, boys, scr);
}
#if QCG_SS_KET
template <class OT, int SPLIT>
void launch_ss_split(const BasisDev& bs, const int4* q, const int* order, long long nq, OT* out, const double* boys,
                     int nsm, cudaStream_t st)
{
    auto k = eri_ss_kernel<Cls, OT, SPLIT>;
    constexpr int warps = kSSThreads / 32, per = warps * (32 / SPLIT);
    constexpr size_t smem =
        (kBoysRows * kBoysColumns + warps * kSSKetSlots * kSSKetDoubles * (32 / SPLIT)) * sizeof(double);
    static std::atomic<unsigned long long> ready{0};
    ensure_smem(k, smem, ready);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kSSThreads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const long long blocks = std::min<long long>((nq + per - 1) / per, (long long)nsm * per_sm);
    k<<<(unsigned)blocks, kSSThreads, smem, st>>>(bs, q, order, nq, out, boys);
}
// Lanes per quartet: one where one lane per quartet keeps every SM's sixteen warps busy, else as many of the up to nine
// bra primitive pairs as there are lanes (a quartet of 81 primitive quartets is a serial chain of 81 otherwise).
template <class OT>
void launch_ss(const BasisDev& bs, const int4* q, const int* order, long long nq, OT* out, const double* boys,
               int nsm, cudaStream_t st)
{
    if (nq <= 0) return;
    const long long lanes = (long long)nsm * 16 * 32;
    if (nq * 8 <= lanes) launch_ss_split<OT, 8>(bs, q, order, nq, out, boys, nsm, st);
    else if (nq * 3 <= lanes) launch_ss_split<OT, 4>(bs, q, order, nq, out, boys, nsm, st);
    else if (nq <= lanes) launch_ss_split<OT, 2>(bs, q, order, nq, out, boys, nsm, st);
    else launch_ss_split<OT, 1>(bs, q, order, nq, out, boys, nsm, st);
}
#endif
}   // namespace

void QCG_CAT(launch_eri_team_, QCG_CLASS)(const BasisDev& bs, const int4* q, const int* order, long long nq,
                                          double* out, const double* boys, const TeamScratchDev& scr,
                                          const TeamShape& sh, cudaStream_t st)
{
#if QCG_SS_KET
    launch_ss(bs, q, order, nq, out, boys, sh.nsm, st);
#else
    launch_batch(bs, q, order, nq, out, boys, scr, sh, st);
#endif
}
void QCG_CAT(launch_eri_team32_, QCG_CLASS)(const BasisDev& bs, const int4* q, const int* order, long long nq,
                                            float* out, const double* boys, const TeamScratchDev& scr,
                                            const TeamShape& sh, cudaStream_t st)
{
#if QCG_SS_KET
    launch_ss(bs, q, order, nq, out, boys, sh.nsm, st);
#else
    launch_batch(bs, q, order, nq, out, boys, scr, sh, st);
#endif
}

// the team form of the direct J/K build of this class (jk_team_kernel); the scratch has room for sh.grid CTAs
void QCG_CAT(launch_jk_team_, QCG_CLASS)(const JKWorkDev& w, const PairListDev& bra, const PairListDev& ket,
                                         const PrimPairsDev& P, const int* f0, const double* D, double* J,
                                         double* K, int n, const double* boys, const TeamScratchDev& scr,
                                         const TeamShape& sh, cudaStream_t st)
{
    const long long span = scr.list.n ? scr.list.total : w.gend - w.gbeg;
    if (span <= 0) return;
    const long long ngroups = (span + 31) / 32;
    if (scr.kmax == 1)
    {
        // one primitive quartet per quartet throughout: jk_group_kernel, one wave of CTAs.  A round has as many
        // groups as the class's group count gives every CTA, so that a small class still spreads over the SMs.
        auto k = w.det_lo ? jk_group_kernel<Cls, true> : jk_group_kernel<Cls, false>;
        static std::atomic<unsigned long long> ready{0}, ready_det{0};
        ensure_smem(k, kGroupSmem, w.det_lo ? ready_det : ready);
        const int per = (int)std::min<long long>(Cls::kGroups, std::max<long long>(1, ngroups / sh.group_grid));
        const long long blocks = std::min<long long>((ngroups + per - 1) / per, sh.group_grid);
        k<<<(unsigned)blocks, Cls::kJKWarps * 32, kGroupSmem, st>>>(w, bra, ket, P, f0, D, J, K, n, boys, scr.hrr, per);
        return;
    }
    auto k = w.det_lo ? jk_team_kernel<Cls, true> : jk_team_kernel<Cls, false>;
    static std::atomic<unsigned long long> ready{0}, ready_det{0};
    ensure_smem(k, kSmem, w.det_lo ? ready_det : ready);
    const long long blocks = ngroups < sh.grid ? ngroups : sh.grid;
    k<<<(unsigned)blocks, kThreads, kSmem, st>>>(w, bra, ket, P, f0, D, J, K, n, boys, scr);
}

}   // namespace qcg
