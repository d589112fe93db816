// Decompression of one zstd frame (RFC 8878) block by block, with the blocks that are stored as they
// are copied by several threads.
#pragma once
#include <cstddef>
#include <cstdint>
#include <functional>

#include "zstd_api.h"

namespace asz::host {

// Runs f(0..n-1), on several threads if it likes.
using ParallelRun = std::function<void(uint64_t n, const std::function<void(uint64_t)> &f)>;

// Writes the content of the frame in[0, len) to dst[0, raw) and returns true, where `in` is exactly one
// frame with a content size of `raw`, no dictionary and no checksum. ready(n) is called now and then
// when dst[0, n) is final, the last time with n == raw. Returns false for every other input, and for
// frames that are not valid: what dst holds then means nothing, and ZSTD_decompress is the judge.
bool unframe(ZSTD_DCtx *z, const uint8_t *in, size_t len, uint8_t *dst, size_t raw, const ParallelRun &run,
             const std::function<bool(size_t)> &ready);

}  // namespace asz::host
