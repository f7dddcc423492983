// Writing a text that another memory holds.
#pragma once
#include <cerrno>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <memory>
#include <new>

#include "dc_internal.h"

namespace dc {

// Writes head (hn bytes) and the `total` bytes that fetch(to) brings here to
// path.  The file is opened once they are all here: a fetch that fails (its
// code is returned) leaves a file that was there as it was.
template <class Fetch>
int write_fetched(const char* path, const char* head, size_t hn, uint64_t total, Fetch fetch) {
    std::unique_ptr<char[]> text;
    if (total) {
        text.reset(new (std::nothrow) char[total]);
        if (!text) return set_error(DC_ERR_NOMEM, "'%s': no host memory for %llu bytes of text", path, (unsigned long long)total);
        if (int rc = fetch(text.get())) return rc;
    }
    FILE* f = fopen(path, "wb");
    if (!f) return set_error(DC_ERR_IO, "cannot write '%s': %s", path, strerror(errno));
    bool ok = fwrite(head, 1, hn, f) == hn && (!total || fwrite(text.get(), 1, total, f) == total);
    if (fclose(f) != 0) ok = false;
    return ok ? DC_OK : set_error(DC_ERR_IO, "short write to '%s'", path);
}

}  // namespace dc
