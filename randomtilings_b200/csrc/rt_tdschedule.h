// rt_tdschedule.h -- the triangle-dimer phase program of a sequence of moves.
//
// The reference refreshes every array after every move
// (TriangleDimerTiler.cpp:243-347): the triangles and the three butterfly
// arrays from the lozenges, or the lozenges from what was flipped.  Most of
// these refreshes are overwritten by the next move's before anything reads
// them, since each rewrites its whole array inside the lattice from arrays
// that the same move has just changed.  TdSchedule notes which arrays await a
// refresh, and from what, and emits a refresh only when a later move reads the
// array; flush() emits the rest, so that every array ends as the reference
// leaves it.
//
// Over the fast mode's 30-move sweep that is 130 phases instead of 186, and of
// the 78 refreshes of a butterfly array 3 remain; over random moves 4.8 phases
// a move instead of 5.7.
#pragma once

#include <stdint.h>

#include "rt_tdops.h"

namespace rtb {

class TdSchedule {
public:
    // Phases one move, and flush(), emit at most.
    static constexpr int kMaxPhases = 8;

    // Lozenge flips of orientation t, class c.
    template <class Emit>
    void lozenges(uint32_t t, uint32_t c, Emit emit) {
        need_lozenges(emit);
        emit(TD_ROT_LOZ, t, c, true);
        emit(TD_LOZ_FLIPPED, t, c, false);
        emit(TD_LOZ_OTHER, t, 0u, false);
        up_ = FROM_LOZENGES;
        down_ = FROM_TRIANGLES;
        bfly_ = 7u;
    }
    // Triangle flips: down (1) or up (0) triangles, class c.
    template <class Emit>
    void triangles(uint32_t down, uint32_t c, Emit emit) {
        if (down)
            need_down(emit);
        else
            need_up(emit);
        emit(TD_ROT_TRI, down, c, true);
        emit(TD_TRI_FLIPPED, down, c, false);
        up_ = down ? FROM_TRIANGLES : CLEAN;
        down_ = down ? CLEAN : FROM_TRIANGLES;
        loz_ = FROM_TRIANGLES;
        bfly_ = 7u;
    }
    // Butterfly flips of orientation t, slice p1, parity p2.
    template <class Emit>
    void butterflies(uint32_t t, uint32_t p1, uint32_t p2, Emit emit) {
        need_butterflies(t, emit);
        emit(TD_ROT_BFLY, t, p1 | (p2 << 2), true);
        emit(TD_BFLY_SAME, t, p1 | (p2 << 2), false);
        emit(TD_BFLY_21, t, p1, false);
        emit(TD_BFLY_22, t, p1, false);
        emit(TD_BFLY_23, t, p1, false);
        loz_ = FROM_BUTTERFLIES + t;
        bfly_ = 7u & ~(1u << t);
        up_ = FROM_LOZENGES;
        down_ = FROM_TRIANGLES;
    }
    template <class Emit>
    void flush(Emit emit) {
        need_lozenges(emit);
        if (bfly_) {
            const bool up = up_ == FROM_LOZENGES;
            emit(TD_BFLY_FROM_LOZ, up ? 1u : 0u, bfly_, false);
            bfly_ = 0u;
            if (up) up_ = CLEAN;
        }
        need_up(emit);
        need_down(emit);
    }

private:
    enum : uint32_t { CLEAN = 0, FROM_LOZENGES = 1, FROM_TRIANGLES = 2 /* the other triangles */, FROM_BUTTERFLIES = 3 };
    // What awaits a refresh, and from what: the lozenges (from the triangles or
    // butterfly array t: FROM_BUTTERFLIES + t), the up and the down triangles, and
    // a mask of butterfly arrays (from the lozenges).  The sources are clean or
    // await theirs, and do not change before the refresh is emitted or dropped.
    uint32_t loz_ = CLEAN, up_ = CLEAN, down_ = CLEAN, bfly_ = 0u;

    template <class Emit>
    void need_lozenges(Emit emit) {
        if (loz_ == FROM_TRIANGLES) {
            need_up(emit);
            need_down(emit);
            emit(TD_LOZ_FROM_TRI, 0u, 0u, false);
        } else if (loz_ != CLEAN) {
            emit(TD_LOZ_FROM_BFLY, loz_ - FROM_BUTTERFLIES, 0u, false);
        }
        loz_ = CLEAN;
    }
    template <class Emit>
    void need_up(Emit emit) {
        if (up_ == FROM_LOZENGES) {
            need_lozenges(emit);
            emit(TD_UP_FROM_LOZ, 0u, 0u, false);
        } else if (up_ == FROM_TRIANGLES) {
            emit(TD_TRI_OTHER, 1u, 0u, false);
        }
        up_ = CLEAN;
    }
    template <class Emit>
    void need_down(Emit emit) {
        if (down_ == CLEAN) return;
        need_up(emit);
        emit(TD_TRI_OTHER, 0u, 0u, false);
        down_ = CLEAN;
    }
    template <class Emit>
    void need_butterflies(uint32_t t, Emit emit) {
        if (!(bfly_ >> t & 1u)) return;
        need_lozenges(emit);
        emit(TD_BFLY_FROM_LOZ, 0u, 1u << t, false);
        bfly_ &= ~(1u << t);
    }
};

// Move s of the fast mode's 30-move sweep over every flip class.
template <class Emit>
void td_fast_move(TdSchedule& td, uint32_t mv, Emit emit) {
    if (mv < 6)
        td.lozenges(mv / 2, mv % 2, emit);
    else if (mv < 12)
        td.triangles((mv - 6) / 3, (mv - 6) % 3, emit);
    else
        td.butterflies((mv - 12) / 6, ((mv - 12) / 2) % 3, (mv - 12) % 2, emit);
}

}  // namespace rtb
