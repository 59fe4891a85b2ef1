// When a context's workspace may be larger than a call needs (host code only).
#pragma once
#include <algorithm>
#include <cstddef>

namespace kq {

// Workspace that calls keep for speed alone.  512 MiB is 0.3 % of a B200's memory and holds all that the solver and the
// residual check ask for up to 32^4 with 12 shifts (378 MB more for the windowed solver, 302 MB of temporaries).
// Beyond it a solve's workspace comes from the context's pool, whose memory CUDA hands to any allocation of the
// process that would fail without it, and a residual check in a context that has solved nothing takes fewer shifts at a
// time (48^4, 12 shifts: 9.0 against 8.3 ms).
constexpr size_t kWorkKeep = size_t(512) << 20;

// Growth that is taken without a look at the free memory, which costs the host 70 us: 64 MiB, unless an allocation has
// failed before.
constexpr size_t kWorkSmall = size_t(64) << 20;

struct WorkPolicy {
    size_t limit = 0;  // the caller's (kq_set_workspace_limit); 0: none
    size_t failed = 0, failed_room = 0;  // size that last could not be allocated, and the room there was then

    // whether may_grow wants to know the free memory
    bool asks(size_t want, size_t have) const { return failed || (want > have && want - have > kWorkSmall); }

    // whether a workspace of `want` bytes may replace one of `have` bytes, `free` bytes of device memory being left,
    // for a call that also runs in a smaller one; it may take 1 / share of the free memory
    bool may_grow(size_t want, size_t have, size_t free, int share) const
    {
        if (limit && want > limit) return false;
        if (want > have && want - have > free / share) return false;
        return !(failed && want >= failed && have + free <= failed_room);
    }

    // room: the free memory without the workspace
    void note_failure(size_t want, size_t room)
    {
        failed = want;
        failed_room = room;
    }

    // whether a call that could run in `need` bytes may leave a workspace of `want` behind, `have` bytes being there; a
    // limit of the caller's takes the place of the rule
    bool keeps(size_t want, size_t have, size_t need) const { return limit || want <= std::max(have, need) + kWorkKeep; }

    // the most a call takes for speed alone, with a workspace of `have` bytes there already
    size_t budget(size_t have) const { return std::max(have, limit ? limit : kWorkKeep); }
};

}  // namespace kq
