// First touch (axs_touch.h) when a thread cannot be created: nothing may write
// to the destination once wait() lets a copy begin. The second pthread_create
// fails; the first thread's store is held by a page fault (the destination is
// read-only, the handler waits before it makes it writable) while the "copy"
// (memset) runs, so a thread left running writes its zero after the copy.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <signal.h>
#include <stdio.h>
#include <string.h>
#include <sys/mman.h>
#include <time.h>

#include <atomic>

#include "axs_touch.h"

static const size_t kBytes = (size_t)16 << 20;
static char *g_buf;
static std::atomic<int> g_created{0}, g_faulted{0};

static void pause_ms(long ms) {
    timespec t{ms / 1000, (ms % 1000) * 1000000};
    nanosleep(&t, nullptr);
}

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*fn)(void *), void *arg) {
    typedef int (*create_t)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static create_t real = (create_t)dlsym(RTLD_NEXT, "pthread_create");
    if (g_created > 0) {
        for (int i = 0; i < 5000 && !g_faulted; ++i) pause_ms(1);   // the first thread is at its store
        return EAGAIN;
    }
    ++g_created;
    return real(t, a, fn, arg);
}

static void on_fault(int, siginfo_t *, void *) {
    g_faulted = 1;
    pause_ms(300);
    mprotect(g_buf, kBytes, PROT_READ | PROT_WRITE);
}

int main() {
    if (std::thread::hardware_concurrency() < 4) {   // one thread only: none to fail after it
        puts("skip");
        return 0;
    }
    struct sigaction sa;
    memset(&sa, 0, sizeof sa);
    sa.sa_sigaction = on_fault;
    sa.sa_flags = SA_SIGINFO;
    sigaction(SIGSEGV, &sa, nullptr);
    g_buf = (char *)mmap(nullptr, kBytes, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    {
        axs::Touch touch({g_buf}, kBytes, kBytes / 4);
        for (size_t c = 0; c < 4; ++c) touch.wait(c);
        mprotect(g_buf, kBytes, PROT_READ | PROT_WRITE);
        memset(g_buf, 0x5a, kBytes);
    }
    if (!g_faulted) return puts("no thread got to its store"), 2;
    for (size_t i = 0; i < kBytes; ++i)
        if (g_buf[i] != 0x5a) return printf("byte %zu overwritten after the copy\n", i), 1;
    puts("ok");
    return 0;
}
