// Which graphs a loop of repeated periods is replayed from (the age rotation's periods of an increment
// loop, the accumulators' rotation of an ensemble).
//
// Kernels of one graph are chained, successive graphs are not (48^2 Q1: 1.4 us a graph launch), but
// recording and instantiating a launch costs about as much as two launches. So a phase of the loop
// first gets a graph of one period, which any run's length is made of, and once WORTH periods are
// replayed or due on the same vectors one of up to MOST as well, as many as the run has left. (A graph
// of whatever the first run had left made later, shorter runs and the ends of runs plain launches: 100
// increments of 128^2 Q1 Allen-Cahn 1.01 ms, 0.83 ms this way; and where the vectors change before every
// run it recorded 16 increments to replay them once. With 64 periods for WORTH the first run of 100
// increments on an adaptive mesh took 5 % longer.)
#pragma once

#include <algorithm>

namespace ppf {

struct GraphChoice {
  int capture;  // periods of the graph to capture first, 0: none
  int replay;   // periods of the graph to replay, as often as it fits
};

// periods: left in this run, at least one; one: whether a graph of one period is held, and how many
// periods were replayed from it; many: periods of the longer graph held, 0 without one
inline GraphChoice choose_graph(int periods, bool one, long long replayed, int many) {
  constexpr int MOST = 8, WORTH = 32;
  const int most = std::min(periods, MOST);
  const bool worth = (one ? replayed : 0) + periods >= WORTH;
  if (most > 1 && worth && many < most) return {most, most};
  if (many > 0 && many <= periods) return {0, many};
  return {one ? 0 : 1, 1};
}

}  // namespace ppf
