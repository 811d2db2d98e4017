// fas_cp_types.h -- what the host code shares with the group pass
// (fas_cp_group.cuh).
#pragma once

namespace fasdev {

constexpr int CP_THREADS = 128;

// Scratch of a pass and its lists.  w holds CPW rows of [ngps]: compliance 21,
// rotated stress 6, stress guess 6, orientation a 9, gamcap; once a point's
// iterations have read them, the factors of its djac (36, row-major) and the
// spin of its slips (3) in their place.
constexpr int CPW = 43, CPW_T = 21, CPW_S = 27, CPW_A = 33, CPW_CAP = 42, CPW_SPIN = 36;
struct CpWork {
    double *w;
    double *chi;                 // points: tangents [36][ngps]
    int *count, *head;           // [3] points in a list / taken from it, by the bound on slip systems
    int *list[3];                // items that take CPSTRS
    double *rec;                 // records (null for points): stress from off_s, weight, tangent
    int reclen, off_s;
    const int *gp_of;            // Gauss point of an item (null: the item itself)
    const int *gp_iel;
    double *stress;              // replays: new stress [6][ngps] in place of G.ds; no tangent, and
                                 // cp_iters -1 for a point that fails
};

}  // namespace fasdev
