// Which of a learned box's cells get their corrections in one launch.
//
// The corrections of all three directions take 192 bytes a cell and the FP32
// primitives that the network reads 32 more, beside 368 for the solver's own
// fields.  Where the device has no room for them (boxes of 795^3 to 930^3 cells on
// 288 GB), the corrections go where the corner EMFs lie, which nothing reads
// between two face updates: 24 bytes a cell, room for three eighths of the
// cells in one direction.  A sweep then goes in windows, runs of whole lines along
// it, each a launch of the network and one of the sweep.
#pragma once
#include <stdint.h>

#include "intdiv.cuh"  // IDFX_HD

namespace idfx {

// lines line0 .. line0 + lines - 1 along dir, of `per` positions each (the
// sweep's numbering, sweep_cell.cuh)
struct LearnedWindow {
  int dir;
  unsigned line0, lines, per;
};

// a window's cells in a row: neighbours along x next to each other
IDFX_HD unsigned window_index(const LearnedWindow& w, unsigned line, unsigned p) {
  const unsigned l = line - w.line0;
  return w.dir == 0 ? l * w.per + p : p * w.lines + l;
}
IDFX_HD void window_cell(const LearnedWindow& w, unsigned q, unsigned& line, unsigned& p) {
  if (w.dir == 0) {
    line = w.line0 + q / w.per;
    p = q % w.per;
  } else {
    line = w.line0 + q % w.lines;
    p = q / w.lines;
  }
}

// the window of `total` lines that starts at line0, of at most `room` cells
// (a box has 36 or more cells across a line, with its ghosts, so three eighths
// of its cells are room for thirteen lines at least)
IDFX_HD LearnedWindow window_from(int dir, unsigned line0, unsigned total, unsigned per, unsigned room) {
  const unsigned most = room / per, left = total - line0;
  return LearnedWindow{dir, line0, left < most ? left : most, per};
}

}  // namespace idfx
