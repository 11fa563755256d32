// mail.h — pinned host memory for the words that a context's or a guide's calls wait for:
// written in the stream's order, read after one wait for the stream.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "devbuf.h"

namespace rgr {

struct Mail {
    unsigned long long next_pixel;
    uint32_t counts[8], stop, err;
    uint32_t link_err;  // the zero-copy path's error word, written by its kernel
    float loss;         // a guide's training step's, written by its kernel
};
// Pinning a page takes some 120 us and a context 15 to create, so the first 64 contexts and
// guides of the process share one allocation; a further one has its own.
constexpr int kSharedMails = 64;
inline std::mutex mail_mutex;
inline Mail* shared_mails = nullptr;
inline uint64_t shared_taken = 0;  // a bit each

inline Mail* take_mail() {
    std::lock_guard<std::mutex> lock(mail_mutex);
    Mail* m = nullptr;
    if (!shared_mails && !cuda_ok(cudaHostAlloc(&shared_mails, sizeof(Mail) * kSharedMails, cudaHostAllocPortable),
                                  "cudaHostAlloc")) {
        shared_mails = nullptr;
        return nullptr;
    }
    for (int k = 0; k < kSharedMails; ++k)
        if (!((shared_taken >> k) & 1u)) {
            shared_taken |= 1ull << k;
            return shared_mails + k;
        }
    return cuda_ok(cudaHostAlloc(&m, sizeof(Mail), cudaHostAllocPortable), "cudaHostAlloc") ? m : nullptr;
}
inline void give_mail(Mail* m) {  // nothing in flight writes to it
    if (!m) return;
    std::lock_guard<std::mutex> lock(mail_mutex);
    if (m >= shared_mails && m < shared_mails + kSharedMails)
        shared_taken &= ~(1ull << (m - shared_mails));
    else
        cudaFreeHost(m);
}

}  // namespace rgr
