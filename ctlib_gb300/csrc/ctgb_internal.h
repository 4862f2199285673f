// Internal declarations shared by the translation units of libctgb.so.
#ifndef CTGB_INTERNAL_H
#define CTGB_INTERNAL_H

#include <cstddef>
#include <string>

namespace ctgb {
// records `msg` as the calling thread's last error (ctgb_last_error) and
// returns `code`
int fail(int code, const std::string& msg);
// lets `kern` be launched with up to `most` bytes of dynamic shared memory, the most
// that any of its launches asks for
int allow_smem(const void* kern, size_t most, const char* what);
}  // namespace ctgb

#endif
