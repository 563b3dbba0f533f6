// launch_rules.h -- host rules that choose how a step's kernels are launched (plain C++).
#pragma once

namespace dpd {

// Parts that the flattened pair schedule cuts the entries of 32 particles into, each a warp's
// work, when it runs as one launch.  Several while the GPU has room for them (us a step or of the
// pass with 1 / 2 / 4 / 8 / 16 / 32 parts, "-" not measured): 2000 particles at density 10, skin 0.3
// - / 33 / 24 / 19 / 17 / 16; 4000 at 3 - / 19 / 17 / 16 / 15 / 17, at 25 - / 64 / 41 / 30 / 24 / 25;
// 8000 at 3 - / 19 / 17 / 16 / 18 / 21, at 25 - / 64 / 43 / 32 / 32 / 31; 16000 at 3 - / 20 / 18 / 19 /
// 21 / 27; the pass at 24000 22 / 16.3 / 14.3 / 14.4, at 81000 25.4 / 25.1 / 26.4, at 192000 44.2 /
// 44.3 / 50.  An engine that shares the GPU with others (a server's cohorts) takes one, since theirs
// fill the rest: of 22 pairs of runs taken in turn, a saturated stream of 64 jobs was served faster
// with one part in 14, by 2.5% on average (2.1e9 to 2.9e9 particle-steps/s either way, as the host's
// load allows).
inline int flat_parts(int warps, bool alone)
{
    if (!alone) return 1;
    if (warps <= 148) return 16;
    if (warps <= 148 * 2) return 8;
    return warps <= 148 * 6 ? 4 : (warps <= 148 * 20 ? 2 : 1);
}

// A cutoff squared as the kernels compare it: in float, whatever it is the cutoff of, so that equal
// cutoffs have equal squares (squared in double and then rounded, 75 of the cutoffs 0.50, 0.51 ..
// 3.99 come out one ulp smaller).
inline float cutoff2(double c)
{
    const float f = (float)c;
    return f * f;
}

// Whether the list holds entries outside the largest pair cutoff, which the flattened pair schedule
// then filters out first.  Where it holds none, the filter and its queue are work for nothing: a
// melt of rc 0.8 and skin 0 took 187.6 us a step with them and takes 171.3 (648000 particles; 83.2
// and 80.9 at 192000, 39.1 either way at 24000).
inline bool lists_beyond(double list_cut, double largest_rc)
{
    return cutoff2(list_cut) > cutoff2(largest_rc);
}

// Whether the filter is worth its pass, from the mean entries of a particle's half list.  It runs with
// 24 or 32 warps per SM where the pass without it has 32 or 40, and most of a dilute system's
// particles have an entry or none.  us a step with it and without, 1000000 particles, skin 0.3: 0.5
// entries 89.6 / 77.7, 1.4 87.7 / 85.6, 2.3 94.2 / 94.2, 4.6 114.9 / 114.4; skin 1.0: 1.7 78.4 / 75.8,
// 3.4 86.1 / 92.7; 3000000, skin 0.3: 0.5 246 / 228, 3.2 290 / 281, 4.6 318 / 325; small grids take
// the same with either.
inline bool filter_pays(double half_list) { return half_list >= 2.5; }

// The pair schedule that a step runs.  7, 8 and 9 are one schedule, the flattened one with log and
// non-log steps split, and an engine that cannot run the cell tiles (11) takes it too; small grids
// run it as one launch (4), or as a thread per list entry (10) where `entry` holds.
inline int pair_schedule(int asked, bool tile, bool small, bool entry)
{
    if (tile) return 11;
    const bool split = (asked >= 7 && asked <= 9) || asked == 11;
    if (!split) return asked;
    return small ? (entry ? 10 : 4) : 8;
}

// Whether the FP64 engine takes its forces with a warp per atom (steps of five kernels) rather than a
// warp per cell (steps of two).  In units of 0.2 ns a step, fitted to runs of 1000 to 300000 atoms at
// densities of 0.02 to 2: an occupied cell takes 10 and an empty one 1, since 4144 warps run at a time
// and each is a chain of loads; an atom takes 4 and its neighbours 1 for each atom of a cell; the
// longer step 62000 more.  us a step with a warp per atom and per cell, 100000 atoms: density 0.05
// 83 / 488, 0.5 95 / 207, 1.0 106 / 139, 1.5 120 / 117, 2.0 123 / 100; 10000 atoms: 0.05 25 / 55, 0.5
// 27 / 27, 1.0 29 / 22; 1000 atoms at 0.05 19 / 12.
inline bool atom_pass(double n, double ncell, double occupied)
{
    return 10.0 * occupied + ncell > 62000.0 + 4.0 * n + n * (n / ncell);
}

// The same for the force pass of a logged step alone, which holds ten sums a pair and runs with 16 warps
// per SM where it takes a cell.  us a step with every step logged, with a warp per atom and per cell in
// it: 10000 atoms at density 0.5 70 / 90, 20000 at 1.0 91 / 102, 100000 at 1.5 216 / 228 and at 2.0 222 /
// 201 (atoms at random fill 0.39, 0.63, 0.78 and 0.86 of the cells).
inline bool atom_pass_logged(double n, double occupied) { return n < 2.0 * occupied; }

}  // namespace dpd
