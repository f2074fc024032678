// Checks what a call does to the pages of its host memory (stim_gb300/csrc/sampler.h: HostRows, HostPages, write_in_place),
// on the CPU.  Usage: host_pages_check CASE  ->  prints "ok", or what is wrong, exit 1.
// Test infrastructure (tests/test_host_pages.py compiles it); the product never uses it.
#include <csetjmp>
#include <csignal>
#include <sys/mman.h>

#include <cstdio>
#include <cstring>
#include <string>

#include "sampler.h"

using namespace gfs_rt;

namespace {

const size_t kPage = (size_t)sysconf(_SC_PAGESIZE);

uint8_t *map(size_t bytes) {
    void *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    madvise(p, bytes, MADV_NOHUGEPAGE);
    return p == MAP_FAILED ? nullptr : (uint8_t *)p;
}

size_t resident(const uint8_t *p, size_t bytes) {
    std::string there(bytes / kPage, 0);
    mincore((void *)p, bytes, (unsigned char *)&there[0]);
    size_t n = 0;
    for (char c : there) {
        n += c & 1;
    }
    return n;
}

sigjmp_buf back;
void on_fault(int) {
    siglongjmp(back, 1);
}

// Whether f takes a memory fault on the host.
template <typename F>
int faults(F f) {
    struct sigaction a {};
    a.sa_handler = on_fault;
    sigaction(SIGSEGV, &a, nullptr);
    sigaction(SIGBUS, &a, nullptr);
    if (sigsetjmp(back, 1)) {
        return 1;
    }
    f();
    return 0;
}

int expect(const char *what, size_t got, size_t want) {
    if (got != want) {
        std::printf("%s: %zu, not %zu\n", what, got, want);
        return 1;
    }
    return 0;
}

}  // namespace

int main(int argc, char **argv) {
    const std::string c = argc > 1 ? argv[1] : "";
    const size_t size = 2048 * kPage;
    uint8_t *const p = map(size);
    int bad = p == nullptr;
    if (c == "rows_apart") {  // 100-byte rows eight pages apart: the pages between them are not asked for
        HostPages pages(true, {p, 256, 100, 8 * kPage});
        pages.before_copy({p, 256, 100, 8 * kPage});
        bad |= expect("pages of rows far apart, before their copy", resident(p, size), 0);
        bad |= expect("in place", write_in_place({{p, 16, 100, 8 * kPage}}, size), 0);
        bad |= expect("pages of rows far apart, in place", resident(p, size), 0);
    } else if (c == "last_row") {  // the gap after the last row is not the call's
        bad |= expect("in place", write_in_place({{p, 65, kPage / 2, 5 * kPage / 4}}, size), 1);
        bad |= expect("pages up to the last row's end", resident(p, size), 81);
    } else if (c == "dense") {  // contiguous rows: all their pages at once, and none after
        HostPages pages(true, {p, 1500, kPage, kPage});
        pages.before_copy({p, 1000, kPage, kPage});
        bad |= expect("pages of the first rows", resident(p, size), 1000);
        pages.before_copy({p + 1000 * kPage, 500, kPage, kPage});
        bad |= expect("pages of all rows", resident(p, size), 1500);
        bad |= expect("in place", write_in_place({{p + 1500 * kPage, 8, kPage, kPage}}, 8 * kPage), 1);
        bad |= expect("pages after rows in place", resident(p, size), 1508);
        bad |= expect("too large for in place", write_in_place({{p + 1508 * kPage, 9, kPage, kPage}}, 8 * kPage), 0);
        bad |= expect("pages after rows too large", resident(p, size), 1508);
    } else if (c == "read_only") {  // what the process may not write faults on the host
        std::memset(p, 1, 100 * kPage);
        mprotect(p + kPage, 99 * kPage, PROT_READ);
        bad |= expect("read-only pages may be read: a fault", faults([&] { touch_pages({p, 100, kPage, kPage}, false); }), 0);
        for (size_t n : {3 * kPage, 99 * kPage, 100 * kPage}) {
            bad |= expect("read-only pages in place: a fault", faults([&] { write_in_place({{p, n, 1, 1}}, size); }), 1);
        }
        bad |= expect("writable bytes beside them: a fault", faults([&] { write_in_place({{p, kPage, 1, 1}}, size); }), 0);
        bad |= expect("a writable byte", p[kPage - 1], 1);
        bad |= expect("read-only pages among writable ones: a fault",
                      faults([&] { write_in_place({{p + 99 * kPage, 100, kPage, kPage}}, size); }), 1);
    } else if (c == "gaps") {  // the bytes between rows belong to others: pages are touched at bytes of rows
        std::memset(p, 1, 64 * kPage);
        mprotect(p + kPage, kPage, PROT_READ);
        // The second row's first byte is the last of page 1.
        bad |= expect("a read-only page with one byte of a row: a fault",
                      faults([&] { write_in_place({{p + kPage - 8, 2, 8, kPage + 7}}, size); }), 1);
        bad |= expect("a read-only page after the last row: a fault",
                      faults([&] { write_in_place({{p + kPage / 2, 2, kPage / 4, kPage / 4}}, size); }), 0);
        bad |= expect("many rows across a read-only page: a fault",
                      faults([&] { write_in_place({{p, 30, 100, 3 * kPage / 4}}, size); }), 1);
    } else if (c == "inaccessible") {
        mprotect(p + 100 * kPage, kPage, PROT_NONE);
        bad |= expect("pages before one without access: a fault", faults([&] { touch_pages({p, 100, kPage, kPage}, false); }), 0);
        bad |= expect("pages up to one without access: a fault", faults([&] { touch_pages({p, 100 * kPage + 1, 1, 1}, false); }), 1);
        FILE *f = std::tmpfile();
        bad |= ftruncate(fileno(f), kPage + 5);
        void *m = mmap(nullptr, 100 * kPage, PROT_READ, MAP_SHARED, fileno(f), 0);
        bad |= expect("a file's pages up to its end: a fault", faults([&] { touch_pages({m, 2, kPage, kPage}, false); }), 0);
        bad |= expect("a file's pages past its end: a fault", faults([&] { touch_pages({m, 100, kPage, kPage}, false); }), 1);
    } else {
        std::printf("unknown case\n");
        return 2;
    }
    if (!bad) {
        std::printf("ok\n");
    }
    return bad;
}
