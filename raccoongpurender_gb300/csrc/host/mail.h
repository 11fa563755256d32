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
// guides that live at a time share one allocation, which the process keeps; a further one has its
// own.  cudaDeviceReset frees the page with everything else of the process: the next slot is then
// of a new page, and slots of the old one are forgotten.
constexpr int kSharedMails = 64;
struct MailPage {
    std::mutex mutex;
    Mail* mails = nullptr;
    uint64_t taken = 0;  // a bit each
    uint64_t age = 0;    // pages before this one
};
inline MailPage mail_page;

inline bool is_pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeHost;
    cudaGetLastError();
    return false;
}

class MailSlot {
public:
    MailSlot() = default;
    MailSlot(const MailSlot&) = delete;
    MailSlot& operator=(const MailSlot&) = delete;
    ~MailSlot() { give(); }  // nothing in flight writes to it
    bool take() {
        MailPage& page = mail_page;
        std::lock_guard<std::mutex> lock(page.mutex);
        if (page.mails && !is_pinned(page.mails)) {
            page.mails = nullptr;
            page.taken = 0;
            ++page.age;
        }
        if (!page.mails &&
            !cuda_ok(cudaHostAlloc(&page.mails, sizeof(Mail) * kSharedMails, cudaHostAllocPortable), "cudaHostAlloc")) {
            page.mails = nullptr;
            return false;
        }
        age_ = page.age;
        for (index_ = 0; index_ < kSharedMails; ++index_)
            if (!((page.taken >> index_) & 1u)) {
                page.taken |= 1ull << index_;
                mail_ = page.mails + index_;
                return true;
            }
        if (!cuda_ok(cudaHostAlloc(&mail_, sizeof(Mail), cudaHostAllocPortable), "cudaHostAlloc")) mail_ = nullptr;
        return mail_ != nullptr;
    }
    Mail* operator->() const { return mail_; }

private:
    void give() {
        if (!mail_) return;
        MailPage& page = mail_page;
        std::lock_guard<std::mutex> lock(page.mutex);
        if (index_ == kSharedMails) {
            if (is_pinned(mail_)) cudaFreeHost(mail_);
        } else if (age_ == page.age) {
            page.taken &= ~(1ull << index_);
        }
        mail_ = nullptr;
    }
    Mail* mail_ = nullptr;
    int index_ = 0;  // in the page; kSharedMails: an allocation of its own
    uint64_t age_ = 0;
};

}  // namespace rgr
