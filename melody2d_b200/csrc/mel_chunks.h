// Host builder of the Gauss-point chunk images that the body kernel reads for bodies above
// MEL_MAX_BODY_NODES nodes (layout in mel_internal.h; the others have tiles, mel_tiles.h).
#pragma once
#include <cstdint>
#include <vector>
#include "mel_internal.h"

struct mel_chunk_set {
    std::vector<mel_chunk> chunks;
    std::vector<int> b_chunk0;     // [n_bodies+1] first chunk of each body
    std::vector<uint8_t> img;      // all images, each 16-byte aligned
    int img_max = 16;              // largest image (bytes)
    long long n_entries = 0;       // stored entries, padding included
    long long n_pad = 0;           // padding entries (rounding of each chunk to 8 entries)
    std::vector<int> b_pipe;       // [n_bodies] zeros: every body's images are those of the two-buffer loop
};

// Cuts the Gauss points of every deformable body of more than min_nodes nodes into chunks of at most
// `ecap` entries and at most MEL_CHUNK_GP_FP64 points.  mixed: dN pairs stored as FP32 instead of
// FP64, and pieces instead of pull slots (the number after it is not used).  Returns MEL_OK or an
// error code with the message set.
mel_status mel_build_chunks(const mel_model_desc* d, int ecap, mel_chunk_set& out, bool mixed = false, long long = 0,
                            int min_nodes = 0);
// The images of the bodies above MEL_MAX_BODY_NODES nodes, with the most entries a chunk (up to
// MEL_CHUNK_E_MAX) whose two buffers and mbarriers take at most `room` bytes of shared memory.
mel_status mel_build_wide_chunks(const mel_model_desc* d, size_t room, mel_chunk_set& out, bool mixed);
