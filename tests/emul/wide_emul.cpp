// The chunks that mel_create builds for bodies above MEL_MAX_BODY_NODES nodes (test infrastructure).
// stats: [chunks, points, largest image in bytes, most points of a chunk]
#include <algorithm>
#include "mel_chunks.h"

extern "C" int emul_wide_chunks(const mel_model_desc* d, long long room, int mixed, long long* stats)
{
    mel_chunk_set CS;
    const int rc = mel_build_wide_chunks(d, (size_t)room, CS, mixed != 0);
    if (rc != MEL_OK) return rc;
    stats[0] = (long long)CS.chunks.size();
    stats[1] = stats[3] = 0;
    stats[2] = CS.img_max;
    for (const mel_chunk& c : CS.chunks) { stats[1] += c.ngp; stats[3] = std::max<long long>(stats[3], c.ngp); }
    return 0;
}
