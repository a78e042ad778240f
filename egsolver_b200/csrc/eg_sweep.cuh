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

struct SweepCtrl {
    /* grid_barrier's fields */
    unsigned bar_count, bar_gen;
    int stop, abort;
    long long rounds;                    /* primal rounds completed            */
    unsigned long long wait_site;
    unsigned long long t_start;
    /* the schedule, advanced by each round's last arriver */
    int phase;
    int left;                            /* primal sweeps left in this phase   */
    int primal_len, dual_len;            /* sweeps of the next phases          */
    long long sweeps, dual_sweeps, kill_sweeps; /* run so far                  */
    int attempts;                        /* certificates tried                 */
    int out_bits;                        /* width of the credits in `out`      */
    unsigned long long raised[2];        /* raises of a round, by parity       */
    /* of the game and of the solve */
    unsigned long long mg, wmax;
    unsigned long long lifts, edges, changes, certified, num_top;
};

struct SweepParams {
    const long long *rp;                 /* the input CSR, original order      */
    const int *succ, *w;
    const unsigned char *owner;          /* or null: vertex >= n0 is player 1  */
    int n, n0;
    long long m;
    long long *F, *D, *K;                /* grid kernel: credits, potentials   */
    void *out;                           /* credits, int32 or int64            */
    SweepCtrl *ctrl;
    long long max_rounds;                /* < 0: no cap                        */
    unsigned long long timeout_ns, wait_limit_ns;
    const int *cancel;
    int lanes;                           /* lanes per vertex: 1 .. 32          */
    int sweeps;                          /* primal sweeps between two barriers */
    int nshift;                          /* potentials count weights 2^nshift-fold */
    int bits;                            /* 32, 64: width asked for            */
    int narrow;                          /* 64: may come out in 32 bits        */
    int smem_bytes;                      /* dynamic shared memory              */
    long long hand_sweeps;               /* 0, or hand over after this many primal sweeps when few credits rise */
    long long hand_raised;               /* "few": raises per round            */
};

/* Bytes of dynamic shared memory with which the one-CTA kernel holds a game. */
long long sweep_cta_bytes(long long n, long long m);
/* Launches the one-CTA kernel (game in shared memory) or the persistent
 * grid kernel on `st`; *grid gets the CTAs. */
eg_status launch_sweep(SweepParams p, cudaStream_t st, int max_ctas, int *grid, int *block);

}  // namespace eg

#endif
