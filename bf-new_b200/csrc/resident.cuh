// Cluster-resident searches (resident.cu): host interface.
#pragma once

#include "engine_types.cuh"

#include <chrono>

namespace bfx {

// Block configurations that the current device can hold (counted from the
// smallest); called once per resident graph.
u32 resident_shapes();

// Sorts the prepared set's lanes largest first and keeps in `nets` those that
// a cluster holds; larger lanes of whole-graph batches (full[b]) go to `whole`
// (a team of blocks each); fit[b] gets the lanes of batch b in either.
void resident_select(bfx_workspace* ws, const std::vector<u32>& full, std::vector<ResidentNet>& nets,
                     std::vector<ResidentNet>& whole, std::vector<u32>& fit);

// Launches the prepared set's searches, whole-graph lanes and nets (those of
// batches on another engine return at once).  The work is ordered after what
// ws->stream holds, and ws->stream waits for it.  Returns the number of
// launches.
u32 launch_searches(bfx_workspace* ws, const LaunchParams& p, bool count);

// The same under host control (the nets only with `clusters`): launches of at
// most `chunk` rounds, after each of which the host looks whether a search has
// rounds left (counted in ws->last_host_checks) and, past the deadline, stops
// the run as a device failure.
u32 poll_searches(bfx_workspace* ws, const LaunchParams& p, bool count, bool clusters, u32 chunk,
                  std::chrono::steady_clock::time_point deadline);

// Releases the workspace's streams and events of these launches.
void resident_release(bfx_workspace* ws);

}  // namespace bfx
