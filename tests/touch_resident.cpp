// First touch (axs_touch.h) of a destination whose pages exist: no thread is
// started and nothing is written. Of one whose pages exist in part: every
// missing page is there after wait(), the others keep their bytes.
#include <dlfcn.h>
#include <pthread.h>
#include <stdio.h>
#include <string.h>

#include <atomic>

#include "axs_touch.h"

static std::atomic<int> g_created{0};
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*fn)(void *), void *arg) {
    typedef int (*create_t)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static create_t real = (create_t)dlsym(RTLD_NEXT, "pthread_create");
    ++g_created;
    return real(t, a, fn, arg);
}

int main() {
    const size_t page = sysconf(_SC_PAGESIZE), bytes = (size_t)32 << 20, off = 24;   // not page-aligned
    char *whole = (char *)mmap(nullptr, bytes + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    madvise(whole, bytes + page, MADV_NOHUGEPAGE);
    char *p = whole + off;
    memset(whole, 0x5a, bytes / 2);   // the first half exists
    {
        axs::Touch touch({nullptr, p}, bytes, bytes / 8);
        for (size_t c = 0; c < 8; ++c) touch.wait(c);
        const int used = g_created;
        if (used < 1) return puts("missing pages not touched"), 1;
        std::vector<unsigned char> in((off + bytes + page - 1) / page);
        mincore(whole, off + bytes, in.data());
        for (size_t i = 0; i < in.size(); ++i)
            if (!(in[i] & 1)) return printf("page %zu missing\n", i), 1;
    }
    for (size_t i = 0; i < bytes / 2; ++i)
        if (whole[i] != 0x5a) return printf("existing byte %zu written\n", i), 1;
    memset(whole, 0x5a, bytes + page);
    g_created = 0;
    {
        axs::Touch touch({p, nullptr}, bytes, bytes / 8);
        for (size_t c = 0; c < 8; ++c) touch.wait(c);
    }
    if (g_created) return printf("%d threads for pages that exist\n", (int)g_created), 1;
    for (size_t i = 0; i < bytes + page; ++i)
        if (whole[i] != 0x5a) return printf("byte %zu written\n", i), 1;
    { axs::Touch none({nullptr, nullptr}, bytes, bytes); none.wait(0); }
    { axs::Touch unmapped({(void *)page}, bytes, bytes); unmapped.wait(0); }   // the copy's to report
    puts("ok");
    return 0;
}
