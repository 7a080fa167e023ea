// Host check of the learned sweeps' windows (learned_window.cuh): over boxes of
// all shapes the windows of a direction hold every position of every line once,
// in places that fit the corner EMFs' memory, and the two maps between a place
// and its cell agree.  Prints the number of faults.
#include <cstdio>
#include <vector>

#include "../../idefix_gb300/csrc/learned_window.cuh"

using namespace idfx;

int main() {
  unsigned long long bad = 0, windows = 0;
  const int sizes[] = {2, 3, 5, 8, 17, 31, 64, 90};
  for (int n0 : sizes)
    for (int n1 : sizes)
      for (int n2 : sizes)
        for (int ext = 1; ext <= 3; ext++)
          for (int d = 0; d < 3; d++) {
            if ((long long)n0 * n1 * n2 > 60000) continue;
            const int n[3] = {n0, n1, n2}, a = d == 0 ? 1 : 0, b = d == 2 ? 1 : 2;
            const long long ncell = (n0 + 4LL) * (n1 + 4) * (n2 + 4);
            const unsigned room = (unsigned)(6 * ncell / 16), per = (unsigned)n[d] + 2;
            const unsigned lines = (unsigned)(n[a] + 2 * ext) * (unsigned)(n[b] + 2 * ext);
            std::vector<unsigned char> seen((size_t)lines * per, 0), place;
            for (unsigned l = 0; l < lines;) {
              const LearnedWindow w = window_from(d, l, lines, per, room);
              windows++;
              if (w.lines == 0 || w.line0 != l || w.line0 + w.lines > lines || (long long)w.lines * per > room) {
                bad++;
                break;
              }
              place.assign((size_t)w.lines * per, 0);
              for (unsigned line = w.line0; line < w.line0 + w.lines; line++)
                for (unsigned p = 0; p < per; p++) {
                  const unsigned q = window_index(w, line, p);
                  unsigned l2 = 0, p2 = 0;
                  if (q < w.lines * per) {
                    window_cell(w, q, l2, p2);
                    if (place[q]++) bad++;
                  } else {
                    bad++;
                  }
                  if (l2 != line || p2 != p) bad++;
                  if (seen[(size_t)line * per + p]++) bad++;
                }
              l += w.lines;
            }
            for (unsigned char s : seen) bad += s != 1;
          }
  std::printf("%llu faults in %llu windows\n", bad, windows);
  return bad != 0 || windows == 0;
}
