// mf_parse.cu -- batch files parsed on the device.
//
// A batch file is text: one update per line, "u v" with 1-based ids
// (core/cli_setup.h:66-82).  The reference reads a line with
// `iss >> src >> dst`: leading white space is skipped, an optional sign and
// decimal digits make a number (one that does not fit an int fails), and
// the line counts only if both numbers parse; anything after the second
// number is ignored.  Ids are then made 0-based, and lines with an id out of
// range or with equal ids are dropped.  Here the file goes to the device once,
// through two pinned chunks (the read of one overlaps the copy of the other); a
// scan over 16-byte words writes the line starts, and a scan over the lines
// parses them with those rules and writes the valid ones in file order, with the
// insert/delete flag of each against the current graph (mf_flag_updates), as
// the reference computes them for every batch before any runs.
#include <fcntl.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <cerrno>
#include <string>

#include "mf_internal.cuh"
#include "mf_scan.cuh"

namespace mf {
namespace {

// Line starts of the 16 bytes from 16 * w on: byte 0 of the file and every byte
// after a newline (also of an empty last line's place, which is past the end
// and not counted).
struct LineStarts {
  const char* text;   // padded to a multiple of 16 bytes
  int64_t size;
  __device__ __forceinline__ uint32_t mask(int64_t w) const {
    const uint4 x = reinterpret_cast<const uint4*>(text)[w];
    const uint32_t v[4] = {x.x, x.y, x.z, x.w};
    uint32_t newline = 0;
#pragma unroll
    for (int q = 0; q < 16; ++q) newline |= (uint32_t)(((v[q >> 2] >> ((q & 3) * 8)) & 0xffu) == '\n') << q;
    const bool before = w == 0 || text[16 * w - 1] == '\n';
    uint32_t m = (newline << 1 | (uint32_t)before) & 0xffffu;
    const int64_t rest = size - 16 * w;
    return rest < 16 ? m & ((1u << rest) - 1u) : m;
  }
  __device__ __forceinline__ int64_t operator()(int64_t w) const { return __popc(mask(w)); }
};

struct LineOut {
  LineStarts ls;
  int64_t words;
  int64_t* begin;
  int64_t* count;    // pinned host word
  __device__ __forceinline__ void operator()(int64_t w, int64_t at) const {
    if (w == words) {
      *count = at;
      return;
    }
    for (uint32_t m = ls.mask(w); m; m &= m - 1) begin[at++] = 16 * w + __ffs(m) - 1;
  }
};

__device__ __forceinline__ bool is_space(char ch) {
  return ch == ' ' || ch == '\t' || ch == '\r' || ch == '\v' || ch == '\f';
}

// One number as `istream >> int` reads it, from text[*k] on (white space
// first); false when there is none or it does not fit an int.
__device__ bool parse_int(const char* text, int64_t end, int64_t* k, int64_t* out) {
  int64_t i = *k;
  while (i < end && is_space(text[i])) ++i;
  bool neg = false;
  if (i < end && (text[i] == '+' || text[i] == '-')) {
    neg = text[i] == '-';
    ++i;
  }
  if (i >= end || text[i] < '0' || text[i] > '9') return false;
  int64_t v = 0;
  while (i < end && text[i] >= '0' && text[i] <= '9') {
    v = v * 10 + (text[i] - '0');
    if (v > 2147483648ll) return false;  // out of int range (checked again below)
    ++i;
  }
  if (neg) v = -v;
  if (v > 2147483647ll || v < -2147483648ll) return false;
  *out = v;
  *k = i;
  return true;
}

struct ParseLine {
  const char* text;
  int64_t size;
  const int64_t* begin;
  int64_t lines;
  int32_t n;
  __device__ __forceinline__ bool line(int64_t l, int32_t* u, int32_t* v) const {
    int64_t k = begin[l], a = 0, c = 0;
    const int64_t e = l + 1 < lines ? begin[l + 1] : size;  // up to the next line's start
    if (!parse_int(text, e, &k, &a) || !parse_int(text, e, &k, &c)) return false;
    *u = (int32_t)(a - 1);
    *v = (int32_t)(c - 1);
    return a >= 1 && a <= n && c >= 1 && c <= n && a != c;
  }
  __device__ __forceinline__ int64_t operator()(int64_t l) const {
    int32_t u, v;
    return line(l, &u, &v) ? 1 : 0;
  }
};

// The valid lines in file order, and their count in a pinned host word.
struct LinesOut {
  ParseLine pl;
  int32_t* u;
  int32_t* v;
  int64_t* count;
  __device__ __forceinline__ void operator()(int64_t l, int64_t at) const {
    if (l == pl.lines) {
      *count = at;
      return;
    }
    int32_t a, b;
    if (!pl.line(l, &a, &b)) return;
    u[at] = a;
    v[at] = b;
  }
};

// Chunks of the pinned block the file is read through.
constexpr int64_t kReadChunk = 256 << 10;

// The text and its line starts (nine bytes for each of the file) stay with the
// context for files up to this size; larger ones give them back.
constexpr int64_t kTextKept = 4 << 20;

struct TextScratch {
  mf_ctx* c;
  ~TextScratch() {
    if (c->txt.cap <= kTextKept && c->txt_begin.cap <= kTextKept) return;
    c->txt.release();
    c->txt_begin.release();
  }
};

struct Fd {
  int fd;
  ~Fd() {
    if (fd >= 0) ::close(fd);
  }
};

}  // namespace

// Parses the file into c->bu / c->bv (0-based, valid lines in file order) and
// returns the count.
int64_t parse_batch_file_device(mf_ctx* c, const char* path) {
  cudaStream_t s = c->stream;
  int64_t* h = c->h_counters;
  const Fd f{::open(path, O_RDONLY | O_CLOEXEC)};
  if (f.fd < 0) MF_FAIL(MF_EIO, std::string("could not open ") + path);
  struct stat sb;
  if (fstat(f.fd, &sb) != 0) MF_FAIL(MF_EIO, std::string("could not read ") + path);
  if (S_ISDIR(sb.st_mode)) MF_FAIL(MF_EIO, std::string("could not read ") + path);
  const int64_t size = S_ISREG(sb.st_mode) && sb.st_size > 0 ? (int64_t)sb.st_size : 0;
  if (size == 0) return 0;
  const int64_t words = (size + 15) / 16;
  const TextScratch text{c};
  c->txt.reserve(16 * words);
  c->txt_begin.reserve(size);
  if (!c->h_read) {
    note_alloc();
    MF_CUDA(cudaMallocHost(&c->h_read, 2 * kReadChunk));
  }
  // ev_a / ev_b: the copy out of chunk 0 / 1 is done
  cudaEvent_t copied[2] = {c->ev_a, c->ev_b};
  int64_t off = 0;
  for (int k = 0; off < size; ++k) {
    char* chunk = c->h_read + (k & 1) * kReadChunk;
    if (k >= 2) MF_CUDA(cudaEventSynchronize(copied[k & 1]));
    const int64_t want = std::min(kReadChunk, size - off);
    int64_t got = 0;
    while (got < want) {
      const ssize_t r = ::read(f.fd, chunk + got, (size_t)(want - got));
      if (r < 0 && errno == EINTR) continue;
      if (r <= 0) {
        MF_CUDA(cudaStreamSynchronize(s));
        MF_FAIL(MF_EIO, std::string("could not read ") + path);
      }
      got += r;
    }
    MF_CUDA(cudaMemcpyAsync(c->txt.p + off, chunk, (size_t)want, cudaMemcpyHostToDevice, s));
    MF_CUDA(cudaEventRecord(copied[k & 1], s));
    off += want;
  }
  const LineStarts ls{c->txt.p, size};
  scan_detail::scan_exclusive_to(ls, LineOut{ls, words, c->txt_begin.p, h}, words, c->ws, s);
  MF_CUDA(cudaStreamSynchronize(s));
  const int64_t lines = h[0];
  c->bu.reserve(std::max<int64_t>(lines, 1));
  c->bv.reserve(std::max<int64_t>(lines, 1));
  c->bins.reserve(std::max<int64_t>(lines, 1));
  const ParseLine pl{c->txt.p, size, c->txt_begin.p, lines, c->n};
  scan_detail::scan_exclusive_to(pl, LinesOut{pl, c->bu.p, c->bv.p, h}, lines, c->ws, s);
  MF_CUDA(cudaStreamSynchronize(s));
  return h[0];
}

}  // namespace mf
