// pms_host_copy.h -- when K goes to a pageable host array through pinned pieces (pms_elements.cu).
#pragma once
#include <cstddef>

namespace pms {

constexpr size_t STAGE_PIECE = size_t(2) << 20;          // bytes of a piece
constexpr size_t STAGE_ONE_THREAD_MAX = size_t(16) << 20;  // most bytes that one host thread moves on

// Whether `bytes` go out in pinned pieces that `threads` host threads copy on, or in the driver's own copy.
// Pieces pay from one piece on with two threads or more.  With one thread (OMP_NUM_THREADS=1, a launcher's
// default for several processes; one CPU) they pay while the array is small: a step on Hex20 blocks, driver's copy and
// pieces, 8 MB of K 941 and 656 us, 16 MB 1,301 and 1,110, 22 MB 1,550 and 1,450, 33 MB 2,160 and 2,140, 72 MB
// 4,160 and 5,000, 239 MB 13.6 and 20 to 23 ms; two threads: 72 MB 4,020 and 2,830, 239 MB 12.4 and 11.0 ms.
inline bool pieces_pay(size_t bytes, int threads) {
    return bytes >= STAGE_PIECE && (threads > 1 || bytes <= STAGE_ONE_THREAD_MAX);
}

}  // namespace pms
