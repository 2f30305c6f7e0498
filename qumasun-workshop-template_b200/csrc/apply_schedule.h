// Order of the asynchronous copies in nl_apply_ring_kernel (nonlocal.cu), apart
// from the device code so that it can be checked on the host.
//
// A CTA walks the bundle's columns in groups, SLICE_GROUPS groups to a slice of
// coefficients.  Before the loop it commits PROLOGUE groups of copies, the first of
// them with coefficient slice 0; pass n of the loop waits until all but PENDING of
// the committed groups have landed, then issues and commits group n + PROLOGUE,
// with slice k + 1 when n is the first group of slice k.
//   Pass n has committed PROLOGUE + n groups and waits for all but PROLOGUE - 1 of
//   them, so groups 0 .. n have landed: group n's own columns, and at n = 0 slice 0.
//   Slice k + 1 travels with group k SLICE_GROUPS + PROLOGUE and is first read in
//   pass (k + 1) SLICE_GROUPS, which has waited for it if PROLOGUE <= SLICE_GROUPS.
//   Other threads' copies of a slice are made visible by the barrier behind the wait.
// A wait sees only groups that were committed: with no group before the loop
// (PROLOGUE 0, a form without a ring) slice 0 would be read unwaited for.
#pragma once

namespace qsb {

// STAGES: groups in the ring of columns (0 or 1: no ring, columns are read directly)
template <int STAGES, int SLICE_GROUPS>
struct ApplySchedule {
    static constexpr int PROLOGUE = STAGES > 1 ? STAGES - 1 : 1;
    static constexpr int PENDING = PROLOGUE - 1;
    static_assert(PROLOGUE >= 1, "slice 0 must be in a committed group before the first wait");
    static_assert(PROLOGUE <= SLICE_GROUPS, "a slice must have landed before its first group");
};

}  // namespace qsb
