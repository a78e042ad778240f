/*
 * eg_sweep.cuh -- parameters and control block of the sweep solver
 * (eg_sweep.cu).
 */
#ifndef EG_SWEEP_CUH
#define EG_SWEEP_CUH

#include "eg_device.cuh"

namespace eg {

/* Phases of a sweep solve, as SweepCtrl::phase holds them between rounds. */
enum { SWEEP_PRIMAL = 0, SWEEP_DUAL = 1, SWEEP_KILL = 2, SWEEP_DONE = 3, SWEEP_HANDOVER = 4 };

/* The schedule, held by every thread and advanced by each in the same way
 * after every round. */
struct SweepState {
    int phase;
    int left;                            /* sweeps, or rounds of a kill phase, left in this one */
    int primal_len, dual_len;            /* sweeps of the next phases          */
    int stop;                            /* 0 running; else an eg_status       */
    long long rounds;                    /* primal rounds completed            */
    long long sweeps;                    /* primal sweeps run                  */
};

struct SweepCtrl {
    SweepState s;                        /* as the solve ended                 */
    unsigned long long word[4][16];      /* round barriers: arrivals << 48 | flags | raises */
    int abort;                           /* a CTA gave up waiting              */
    int out_bits;                        /* width of the credits in `out`      */
    unsigned long long wait_site;
    unsigned long long t_start;
    unsigned long long mg, wmax;
    unsigned long long lifts, edges, changes, num_top;
};

struct SweepParams {
    const long long *rp;                 /* the input CSR, original order      */
    const int *succ, *w;
    const unsigned char *owner;          /* or null: vertex >= n0 is player 1  */
    int n, n0;
    void *F, *D, *K;                     /* grid kernel: credits, potentials, their copy (plan.values of 8 B each) */
    int2 *E;                             /* where a CTA's values or edges do not fit its shared memory: */
    int *vid, *soff;                     /* sliced edges, vertices and slice offsets; else null */
    void *out;                           /* credits, int32 or int64            */
    SweepCtrl *ctrl;
    long long max_rounds;                /* < 0: no cap                        */
    unsigned long long timeout_ns, wait_limit_ns;
    const int *cancel;
    int bits;                            /* 32, 64: width asked for            */
    int narrow;                          /* 64: may come out in 32 bits        */
    int smem_bytes;                      /* dynamic shared memory              */
    long long hand_sweeps;               /* 0, or hand over after this many primal sweeps when few credits rise */
    long long hand_raised;               /* "few": raises per round            */
};

/* Which kernel a game takes and what global scratch it needs. */
struct SweepPlan {
    int one_cta, grid, block, smem_bytes;
    size_t values;                       /* entries of F, D and K              */
    size_t edges, vids, offs;            /* entries of E, vid and soff         */
};
eg_status sweep_plan(int n, long long m, int max_ctas, SweepPlan *plan);
/* Launches the one-CTA kernel (game in shared memory) or the persistent
 * grid kernel on `st`. */
eg_status launch_sweep(SweepParams p, const SweepPlan &plan, cudaStream_t st);

}  // namespace eg

#endif
