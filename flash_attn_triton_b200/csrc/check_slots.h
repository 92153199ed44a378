// Words in host memory that value checks are answered in: who has which.  No CUDA in here.
#pragma once
#include <cstdint>
#include <mutex>

namespace fa {

// kWords words, a cache line each.  A call takes a word and gives it back before it returns; a ticket is a word that the
// caller hands in by a call of its own, some time later.  At most kTickets (less than kWords) are out, so a call gets a word
// in the end however many tickets the threads hold.  A word that a kernel on some stream may still write stays out of use
// until it has been written.
template <int kWords, int kTickets> class CheckSlots {
  static_assert(kTickets < kWords, "words for the calls that give them back themselves");

 public:
  static constexpr int kNone = -1;    // no word is free right now
  static constexpr int kNever = -2;   // nor will a call that is running give one back
  static volatile uint32_t* word_of(volatile uint32_t* base, int i) { return base + (int64_t)i * 16; }

  explicit CheckSlots(volatile uint32_t* base) : base_(base) {
    for (int i = 0; i < kWords; ++i) free_[nfree_++] = kWords - 1 - i;
  }
  // A word of zero, as a ticket (whose kernel runs on `device`) or for the call itself.
  int take(bool ticket, int device) {
    std::lock_guard<std::mutex> lock(mu_);
    if (ticket && tickets_ == kTickets) return kNone;
    if (nfree_ == 0 && lost_ > 0) find_again();
    if (nfree_ == 0) return tickets_ + lost_ == kWords ? kNever : kNone;
    const int i = free_[--nfree_];
    state_[i] = ticket ? kTicket : kCall;
    tickets_ += ticket;
    device_[i] = device;
    *word(i) = 0u;
    return i;
  }
  // A ticket becomes a word of the call that hands it in: false where it is not out, so that of two that hand in the
  // same one gets it.  *device: where its kernel is.
  bool hand_in(int i, int* device) {
    std::lock_guard<std::mutex> lock(mu_);
    if (i < 0 || i >= kWords || state_[i] != kTicket) return false;
    state_[i] = kCall;
    --tickets_;
    *device = device_[i];
    return true;
  }
  // Back from the call.  queued: a kernel was given the word.
  void give(int i, bool queued) {
    std::lock_guard<std::mutex> lock(mu_);
    tickets_ -= state_[i] == kTicket;
    if (queued && *word(i) == 0u) {
      state_[i] = kLost;
      ++lost_;
    } else {
      state_[i] = kFree;
      free_[nfree_++] = i;
    }
  }

 private:
  enum State : uint8_t { kFree, kCall, kTicket, kLost };
  volatile uint32_t* word(int i) { return word_of(base_, i); }
  void find_again() {
    for (int i = 0; i < kWords; ++i)
      if (state_[i] == kLost && *word(i) != 0u) {
        state_[i] = kFree;
        free_[nfree_++] = i;
        --lost_;
      }
  }
  std::mutex mu_;
  volatile uint32_t* base_;
  int free_[kWords], nfree_ = 0, tickets_ = 0, lost_ = 0;
  State state_[kWords] = {};
  int device_[kWords];
};

}  // namespace fa
