// to_rov_years.h - the order of launches of the ROV's backward pass: for each
// year, last to first, which years are prepared and have their neighbours
// selected before its fit, and whether that fit may start ahead of its
// predecessor's end.  Host only, no CUDA (compiled on the CPU by
// tests/test_rov_years.py).
#pragma once

struct to_rov_years {
    int slots, sel_slots;          // years prepared / selected at a time
    int t;                         // the year
    int low, sel;                  // first year prepared, first with neighbours
    int prepare, select;           // years to prepare / to select for now, from low / sel

    to_rov_years(int Y, int slots_, int sel_slots_)
        : slots(slots_), sel_slots(sel_slots_), t(Y - 1), low(Y - 1), sel(Y - 1), prepare(0),
          select(0) {}

    bool next() {
        if (--t <= 0) return false;
        prepare = select = 0;
        if (t < low) {
            low = t - slots + 1 > 1 ? t - slots + 1 : 1;
            prepare = t - low + 1;
        }
        if (t < sel) {
            sel = t - sel_slots + 1 > low ? t - sel_slots + 1 : low;
            select = t - sel + 1;
        }
        return true;
    }

    // The fit copies its lists of neighbours ahead of its wait for the kernel
    // before it.  Right after a selection that kernel is the one that writes
    // them, so the fit is launched plainly; the years after it follow a kernel
    // that was itself started after the selection's end.
    bool fit_ahead() const { return select == 0; }
};
