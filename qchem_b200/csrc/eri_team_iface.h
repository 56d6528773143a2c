// eri_team_iface.h -- launch interface of the team form of the FP64 ERI batches (eri_team.cu).
#pragma once
#include <cuda_runtime.h>

#include "batch_plan.h"
#include "qcg_internal.h"

namespace qcg {

// The contracted J/K build's own order of a class's screened quartets (jk_team_list, runtime.cu): entry e is a run of
// bra primitive pairs [y, y + z) of bra pair x against the kets kets[w ..] of one primitive-pair count, items
// offs[e] .. offs[e + 1); n = 0: the class's work list as it is.
struct JKTeamListDev
{
    int n;
    const long long* offs;
    const int4* entry;
    const int* kets;
    long long total;
};

// Device memory a team launch works in, beside its inputs and outputs (the handle owns it):
//   rcache -- per CTA, kmax stage slots: the primitive quartets' R tables and Hermite tables, written once
//             per group of quartets and streamed back into shared memory once per pass;
//   hrr    -- per CTA, the [e0|f0] and [e0|cd] blocks of the group's 32 quartets, lane-minor;
//   err    -- bit 0: a wait for a bulk copy gave up (the results of the launch are not valid);
//             bit 1: a group needed more stage slots than kmax.
struct TeamScratchDev
{
    double* rcache;
    int kmax;
    double* hrr;
    int* err;
    const BatchPlanDev* plan;   // ERI batches: the groups; null (and no order) for an uncontracted class
    JKTeamListDev list;         // contracted J/K builds: the order of the quartets
};

// The launch shape of class k on nsm SMs and the scratch it needs per CTA, in doubles.
struct TeamShape
{
    int grid, threads, nsm;
    long long slot_doubles;    // one stage slot of the R cache
    long long hrr_doubles;     // recurrence blocks
    // the J/K build: CTAs and [e0|f0] doubles per CTA of the uncontracted form, [e0|f0] doubles of the contracted one
    int group_grid;
    long long group_doubles, jk_doubles;
};

using EriTeamLauncher = void (*)(const BasisDev&, const int4*, const int*, long long, double*, const double*,
                                 const TeamScratchDev&, const TeamShape&, cudaStream_t);
// the FP32 batches: the same evaluation with float output
using EriTeam32Launcher = void (*)(const BasisDev&, const int4*, const int*, long long, float*, const double*,
                                   const TeamScratchDev&, const TeamShape&, cudaStream_t);
using EriTeamShapeFn = TeamShape (*)(int nsm);

using JKTeamLauncher = void (*)(const JKWorkDev&, const PairListDev&, const PairListDev&, const PrimPairsDev&,
                                const int*, const double*, double*, double*, int, const double*,
                                const TeamScratchDev&, const TeamShape&, cudaStream_t);

extern const EriTeamLauncher kEriTeamLaunchers[kNumQuartetClasses];
extern const EriTeam32Launcher kEriTeam32Launchers[kNumQuartetClasses];
extern const JKTeamLauncher kJKTeamLaunchers[kNumQuartetClasses];
extern const EriTeamShapeFn kEriTeamShapes[kNumQuartetClasses];

}   // namespace qcg
