// Side streams of one launch: forked from a main stream, joined to it again.
#pragma once

#include <cstddef>

namespace bfx {

// Api: Stream and Event types; record(event, stream) and wait(stream, event),
// which throw on an error; synchronize(stream), which does not.  (A parameter,
// so that its failures can be made on the host.)
//
// Leaving the scope before join() has finished -- a launch between the two
// failed -- waits on the host for every side stream that the main stream does
// not wait for: the caller may then rewrite or free what their kernels use.
template <typename Api>
class SideStreams {
 public:
  struct Side {
    typename Api::Stream stream;
    typename Api::Event done;
  };
  // The first `count` of `sides` start after what `main` holds.
  SideStreams(typename Api::Stream main, typename Api::Event fork, const Side* sides, std::size_t count)
      : main_(main), sides_(sides), count_(count) {
    if (count == 0) return;
    Api::record(fork, main);
    for (std::size_t i = 0; i < count; ++i) Api::wait(sides[i].stream, fork);
  }
  SideStreams(const SideStreams&) = delete;
  SideStreams& operator=(const SideStreams&) = delete;
  ~SideStreams() {
    for (std::size_t i = joined_; i < count_; ++i) Api::synchronize(sides_[i].stream);
  }
  // `main` continues after the sides' work.
  void join() {
    for (; joined_ < count_; ++joined_) {
      Api::record(sides_[joined_].done, sides_[joined_].stream);
      Api::wait(main_, sides_[joined_].done);
    }
  }

 private:
  typename Api::Stream main_;
  const Side* sides_;
  std::size_t count_;
  std::size_t joined_{0};
};

}  // namespace bfx
