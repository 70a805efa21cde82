// Test-only host build of the FS_FP64 row buffer's sizes (csrc/fs_fp64_rows.h)
// with a made-up memory.  Not part of the product.
#include <stdint.h>

#include "fs_fp64_rows.h"

extern "C" {

// the buffer as a context keeps it
struct Rows {
    uint64_t cap, asked, tries;
};

// one assembly of a mesh: `marks` and `want` groups of `group` slots, in a memory
// that has no buffer above `memory` slots; the groups a chunk has
uint64_t rows_reserve(Rows *r, uint64_t marks, uint64_t want, uint64_t group, uint64_t memory)
{
    size_t asked = r->asked;
    const int st = fs::fx_reserve(r->cap, asked, marks, want, group, 0, 1, [&](size_t slots) {
        r->tries++;
        r->cap = slots <= memory ? slots : 0;
        return slots <= memory ? 0 : 1;
    });
    r->asked = asked;
    if (st) return UINT64_MAX;
    return std::min<uint64_t>(want, fs::fx_groups_held(r->cap, marks, group));
}

// a sequence of events: l(aunch), m(ade), R(ead with the flag set), r(ead without);
// the number of elements' redos
int marks_events(const char *events)
{
    fs::FxMarks marks;
    int redos = 0;
    for (; *events; events++) {
        if (*events == 'l') marks.launch();
        if (*events == 'm') marks.made();
        if (*events == 'R') redos += marks.redo(true);
        if (*events == 'r') redos += marks.redo(false);
    }
    return redos;
}

}
