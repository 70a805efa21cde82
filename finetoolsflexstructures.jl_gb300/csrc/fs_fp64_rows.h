// The FS_FP64 elements' row buffer (fs_elem_fp64.cu): a byte of mark per element,
// then the rows of a chunk of elements, in groups.  Host code without CUDA, so that
// it can be tested with made-up capacities.
#pragma once
#include <stddef.h>

#include <algorithm>

namespace fs {

static const size_t FX_LEAST_GROUPS = 608;  // the smallest chunk: four blocks of the Gram kernel an SM

// groups of `group` slots that a buffer of `cap` slots holds after its marks
inline size_t fx_groups_held(size_t cap, size_t marks, size_t group) { return cap > marks ? (cap - marks) / group : 0; }

// A buffer of `cap` slots (0: none) made ready for `marks` and chunks of `want`
// groups.  alloc(slots) replaces the buffer and returns `ok`, `oom` (there is no
// buffer then) or another code, which ends the search.  Where the memory for a
// whole chunk is not there, half of it is tried, and so on down to the smallest
// chunk; `asked` is the largest size that was tried for, so that a buffer that came
// out smaller is not asked for anew by each assembly, as long as it holds this
// mesh's marks and a smallest chunk.  `asked` is set back with every new mesh.
template <class Alloc>
int fx_reserve(size_t cap, size_t &asked, size_t marks, size_t want, size_t group, int ok, int oom, Alloc alloc)
{
    const size_t least = std::min(want, FX_LEAST_GROUPS), held = fx_groups_held(cap, marks, group);
    if (held >= want || (held >= least && held > 0 && asked >= marks + want * group)) return ok;
    asked = marks + want * group;
    for (;; want = std::max(want / 2, least)) {
        const int st = alloc(marks + want * group);
        if (st != oom) return st;
        if (want == least) return ok;
    }
}

// Whether the marks of the elements to do in double are those of the last element
// kernels.  The device's flag that there are any stays until it is read, so one
// that is left by a call which failed in between must not have a later call's
// matrices (other elements, another precision) done over.
struct FxMarks {
    bool fresh = false;
    void launch() { fresh = false; }  // element kernels are about to run
    void made() { fresh = true; }     // they write marks
    bool redo(bool flagged)           // the flag was read: are there elements to do over?
    {
        const bool r = fresh && flagged;
        fresh = false;
        return r;
    }
};

}  // namespace fs
