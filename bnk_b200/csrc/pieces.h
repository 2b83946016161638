// A large batch that is alone in flight goes over the link in pieces: while one is worked on, the next comes up and the
// one before goes down, so both copy engines are busy.  Pieces end on pages of the ring (a copy that starts elsewhere is
// up to a sixth slower: 190 MB up and down in 8 MB pieces 4.1 ms against 4.9), with small ones first and last, when one
// direction has nothing to do yet or any more.  Between two copies an engine rests ~15 us while the other direction is
// busy, so the pieces in the middle of a large ring are large: 190 MB sealed in pieces of at most 8 MB 5.0 ms, 16 MB 4.74,
// 24 MB 4.70, but 47 MB in at most 8 MB 1.35 ms, 24 MB 1.39.  Two streams for each direction share its engine's rate and
// finish later (5.7 ms).  Packets have to lie in the ring in order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

constexpr uint64_t kPieceLeast = 1ull << 20, kPieceMost = 8ull << 20, kPieceMostEver = 24ull << 20, kPage = 4096;
struct Piece {
    uint32_t first, count;       // packets
    uint64_t up, up_to;          // ring bytes that come up in front of them
    uint64_t down, down_to;      // ring bytes nobody works on any more behind them
};
class Pieces { // of n > 0 packets
  public:
    // `more`: a packet's kernel reads and writes at most len + more bytes from its offset on.  All of them have to be up: a
    // later copy must not run over what the kernel has written.
    Pieces(const uint32_t *off, const uint32_t *len, uint32_t n, uint32_t more, uint64_t ext)
        : off_(off), len_(len), n_(n), more_(more), ext_(ext), most_(std::min(std::max(kPieceMost, ext / 8), kPieceMostEver)) {}
    bool next(Piece &p) {
        if (at_ == n_) return false;
        p.first = at_;
        p.up = up_;
        p.down = down_;
        do { // a packet larger than a piece takes several
            const uint64_t left = ext_ - up_, size = std::min(std::min(most_, up_ + kPieceLeast), std::max(kPieceLeast, left / 2));
            up_ = left <= size + size / 2 ? ext_ : (up_ + size) & ~(kPage - 1);
            if (up_ == ext_) at_ = n_;
            while (at_ < n_ && (uint64_t)off_[at_] + more_ + len_[at_] <= up_) at_++;
        } while (at_ == p.first);
        down_ = at_ == n_ ? ext_ : std::max(down_, std::min(up_, (uint64_t)off_[at_]) & ~(kPage - 1));
        p.count = at_ - p.first;
        p.up_to = up_;
        p.down_to = down_;
        return true;
    }

  private:
    const uint32_t *off_, *len_;
    uint32_t n_, more_, at_ = 0;
    uint64_t ext_, most_, up_ = 0, down_ = 0;
};

struct PieceStreams {
    cudaStream_t up, down;
    cudaEvent_t ev_up, ev_down;
};
// The copies of one submit whose kernels run on stream s.  However the submit ends, s is done only when they are: the host
// ring is the caller's again when s has been waited for.
class PieceCopies {
  public:
    PieceCopies(const PieceStreams &ps, uint8_t *dev, uint8_t *host, cudaStream_t s) : ps_(ps), dev_(dev), host_(host), s_(s) {}
    ~PieceCopies() {
        if (!joined_) (void)join();
    }
    PieceCopies(const PieceCopies &) = delete;
    // Copies a piece up (is_up lets the kernels go on behind it) / copies down what the kernels are done with.
    cudaError_t up(const Piece &p) {
        const cudaError_t e = cudaMemcpyAsync(dev_ + p.up, host_ + p.up, p.up_to - p.up, cudaMemcpyHostToDevice, ps_.up);
        return e != cudaSuccess ? e : cudaEventRecord(ps_.ev_up, ps_.up);
    }
    cudaError_t is_up() { return cudaStreamWaitEvent(s_, ps_.ev_up, 0); }
    cudaError_t down(const Piece &p) {
        if (p.down_to == p.down) return cudaSuccess;
        cudaError_t e = cudaEventRecord(ps_.ev_down, s_);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(ps_.down, ps_.ev_down, 0);
        if (e == cudaSuccess) e = cudaMemcpyAsync(host_ + p.down, dev_ + p.down, p.down_to - p.down, cudaMemcpyDeviceToHost, ps_.down);
        return e;
    }
    cudaError_t join() {
        joined_ = true;
        cudaError_t e = cudaEventRecord(ps_.ev_up, ps_.up);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s_, ps_.ev_up, 0);
        if (e == cudaSuccess) e = cudaEventRecord(ps_.ev_down, ps_.down);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s_, ps_.ev_down, 0);
        if (e != cudaSuccess) { // then wait here
            cudaStreamSynchronize(ps_.up);
            cudaStreamSynchronize(ps_.down);
        }
        return e;
    }

  private:
    const PieceStreams ps_;
    uint8_t *const dev_, *const host_;
    const cudaStream_t s_;
    bool joined_ = false;
};
