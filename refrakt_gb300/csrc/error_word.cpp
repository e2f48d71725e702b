// The words come from pages that stay with the process, as many as are held at one time.
#include "error_word.h"

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace rfk {

namespace {

constexpr int kPageInts = 1024, kWordInts = 16;  // a word per 64 bytes
std::mutex g_mu;

std::vector<int*>& free_words() {
    static auto* words = new std::vector<int*>();  // (outlives every static object that may hold a word)
    return *words;
}

}  // namespace

bool ErrorWord::acquire() {
    if (p_) return true;
    std::lock_guard<std::mutex> lock(g_mu);
    auto& words = free_words();
    if (words.empty()) {
        int* page = nullptr;
        if (cudaHostAlloc((void**)&page, kPageInts * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        for (int k = 0; k < kPageInts; k += kWordInts) words.push_back(page + k);
    }
    p_ = words.back();
    words.pop_back();
    *p_ = 0;
    return true;
}

ErrorWord::~ErrorWord() {
    if (!p_) return;
    std::lock_guard<std::mutex> lock(g_mu);
    free_words().push_back(p_);
}

int ErrorWord::take() { return p_ ? __atomic_exchange_n(p_, 0, __ATOMIC_ACQ_REL) : 0; }

}  // namespace rfk
