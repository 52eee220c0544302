// A copy from the caller's memory on a stream of its own, beside work on the main
// stream that does not read it.  Api names the runtime's calls (api.cu: CUDA's; the
// CPU test: a fake whose calls fail on demand); each returns 0 on success.
#pragma once
#include <cstddef>

namespace rm {

template <class Api>
class SideCopy {
 public:
  using Error = typename Api::Error;
  using Stream = typename Api::Stream;
  using Event = typename Api::Event;

  SideCopy() = default;
  SideCopy(const SideCopy&) = delete;
  SideCopy& operator=(const SideCopy&) = delete;
  ~SideCopy() { close(); }

  // Makes the stream and the events, all three or none: after a failure the next
  // call starts again.
  Error open() {
    if (open_) return Error(0);
    Error e = Api::create_stream(&stream_);
    if (e != Error(0)) return e;
    e = Api::create_event(&begin_);
    if (e == Error(0)) {
      e = Api::create_event(&done_);
      if (e != Error(0)) Api::destroy_event(begin_);
    }
    if (e != Error(0)) {
      Api::destroy_stream(stream_);
      return e;
    }
    open_ = true;
    return e;
  }

  // The next copy comes after what `main` holds now.
  Error follow(Stream main) {
    const Error e = Api::record(begin_, main);
    return e != Error(0) ? e : Api::wait(stream_, begin_);
  }

  // Copies, and makes later work on `main` wait for it.  From here until settle()
  // or landed() the copy may be reading src and writing dst.
  Error copy(void* dst, const void* src, size_t bytes, Stream main) {
    in_flight_ = true;
    Error e = Api::copy(dst, src, bytes, stream_);
    if (e == Error(0)) e = Api::record(done_, stream_);
    return e != Error(0) ? e : Api::wait(main, done_);
  }

  bool in_flight() const { return in_flight_; }
  // The main stream has been waited for since copy(), and with it the copy.
  void landed() { in_flight_ = false; }
  // Before the caller gets its memory back on any other path.
  void settle() {
    if (in_flight_) Api::synchronize(stream_);
    in_flight_ = false;
  }

  void close() {
    if (!open_) return;
    settle();
    Api::destroy_event(begin_);
    Api::destroy_event(done_);
    Api::destroy_stream(stream_);
    open_ = false;
  }

 private:
  Stream stream_{};
  Event begin_{}, done_{};
  bool open_ = false, in_flight_ = false;
};

}  // namespace rm
