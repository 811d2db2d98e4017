// fas_adjoint_types.cuh -- what the host code shares with the replay kernels.
#pragma once

namespace fasdev {

// The ampar(k) entries the parameter adjoint covers (1-based k = 1, 2, 3, 5).
constexpr int ADJ_NP = 4;
__host__ __device__ constexpr int adj_ampar_index(int j) { return j < 3 ? j : 4; }

// The history and objective of a replay.  de: de(6, ngps, ninc), dr:
// dr(3, ngps, ninc), dt: dt(ninc), w / y: per GP.
struct ReplayDev {
    const double *de, *dr, *dt, *w, *y;
    double q[3];
    int ninc, chk;
    int zs;          // stride (in rows of ngps) of one state record: 9 + the widest ns
};

// Rows of one increment's record (k_replay_adj's layout) from `rec`, or null.
struct ReplayRows {
    double *commit, *next;       // records of the increment committed and of the one prepared
    double *chk;                 // checkpoint rows to write, or null
    const double *load;          // checkpoint rows to start from, or null
    int flag;                    // row of the branch in a record
};

}  // namespace fasdev
