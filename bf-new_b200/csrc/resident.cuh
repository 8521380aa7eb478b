// Cluster-resident searches (resident.cu): host interface.
#pragma once

#include "engine_types.cuh"

namespace bfx {

// Block configurations that the current device can hold (counted from the
// smallest); called once per resident graph.
u32 resident_shapes();

// Sorts the prepared set's lanes largest first, drops those that no cluster
// holds, and sets fit[b] to the lanes of batch b that stay.
void resident_select(bfx_workspace* ws, std::vector<ResidentNet>& nets, std::vector<u32>& fit);

// Launches the searches of the prepared set's nets (those of batches on
// another engine return at once).  The work is ordered after what ws->stream
// holds, and ws->stream waits for it.  Returns the number of launches.
u32 launch_resident(bfx_workspace* ws, const LaunchParams& p, bool count);

// Releases the workspace's streams and events of these launches.
void resident_release(bfx_workspace* ws);

}  // namespace bfx
