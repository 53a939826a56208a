// What touch_pages (pm_pages.h) does to a buffer: its pages are there afterwards, its bytes
// are as they were, an address that cannot be written is left alone, and neither memory nor
// threads that cannot be had end the process.
#include "pm_pages.h"

#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include <dlfcn.h>
#include <pthread.h>

// the n-th thread from now on, or the memory it takes, cannot be had (-1: all can)
static int memory_after = -1, threads_after = -1;

void* operator new(size_t n)
{
    if (memory_after >= 0 && memory_after-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}

void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x)
{
    using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static Create create = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
    return threads_after >= 0 && threads_after-- == 0 ? EAGAIN : create(t, a, f, x);
}

#define CHECK(x) \
    do { \
        if (!(x)) { \
            std::printf("line %d: %s\n", __LINE__, #x); \
            std::exit(1); \
        } \
    } while (0)

static const size_t kPage = (size_t)sysconf(_SC_PAGESIZE);

static char* map(size_t bytes, int prot)
{
    void* p = mmap(nullptr, bytes, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    CHECK(p != MAP_FAILED);
    return static_cast<char*>(p);
}

static size_t present(char* p, size_t bytes)
{
    std::vector<unsigned char> v(bytes / kPage);
    CHECK(mincore(p, bytes, v.data()) == 0);
    size_t n = 0;
    for (unsigned char c : v) n += c & 1;
    return n;
}

static unsigned char at(size_t i) { return (unsigned char)(i * 131 + (i >> 12) * 7 + 1); }

// bytes of [off, off + len) of a mapping half of whose pages hold data
static void keeps(size_t bytes, size_t off, size_t len)
{
    char* p = map(bytes, PROT_READ | PROT_WRITE);
    for (size_t i = 0; i < bytes; ++i)
        if (i / kPage % 2) p[i] = (char)at(i);
    nyxpm::touch_pages(p + off, len);
    const size_t a = off / kPage * kPage, e = (off + len + kPage - 1) / kPage * kPage;
    CHECK(present(p + a, e - a) == (e - a) / kPage);
    for (size_t i = 0; i < bytes; ++i) CHECK((unsigned char)p[i] == (i / kPage % 2 ? at(i) : 0));
    munmap(p, bytes);
}

int main(int argc, char** argv)
{
    const size_t M = (size_t)1 << 20;
    const char* what = argc > 1 ? argv[1] : "";
    if (!std::strcmp(what, "keeps")) {
        for (size_t len : {(size_t)1, kPage - 1, kPage, kPage + 1, 3 * M + 17, 20 * M + 5, 150 * M + 9})
            for (size_t off : {(size_t)0, (size_t)8, kPage - 8}) keeps((len + 3 * kPage) / kPage * kPage, off, len);
    } else if (!std::strcmp(what, "there")) {   // every page in place: read only, by threads from 128 MB on
        for (size_t len : {(size_t)1, kPage + 1, 127 * M + 3, 128 * M, 200 * M + 11}) {
            const size_t bytes = (len + 2 * kPage) / kPage * kPage;
            char* p = map(bytes, PROT_READ | PROT_WRITE);
            for (size_t i = 0; i < bytes; ++i) p[i] = (char)at(i);
            CHECK(mprotect(p, bytes, PROT_READ) == 0);
            nyxpm::touch_pages(p + 5, len - 1, true);
            nyxpm::touch_pages(p, len, true);
            for (size_t i = 0; i < bytes; ++i) CHECK((unsigned char)p[i] == at(i));
            munmap(p, bytes);
        }
    } else if (!std::strcmp(what, "refused")) {
        for (int prot : {PROT_NONE, PROT_READ}) {
            char* p = map(40 * M, prot);
            nyxpm::touch_pages(p + 100, 40 * M - 200);
            munmap(p, 40 * M);
            nyxpm::touch_pages(p + 100, 40 * M - 200);   // nothing there any more
        }
        char* p = map(40 * M, PROT_READ | PROT_WRITE);
        CHECK(munmap(p + 20 * M, 10 * M) == 0);   // a hole
        nyxpm::touch_pages(p, 40 * M);
        CHECK(present(p, 20 * M) * kPage == 20 * M);
        nyxpm::touch_pages(nullptr, 1);
        nyxpm::touch_pages(p, 0);
    } else if (!std::strcmp(what, "memory") || !std::strcmp(what, "threads")) {
        for (int after = 0; after < 4; ++after) {
            char* p = map(200 * M, PROT_READ | PROT_WRITE);
            int& left = what[0] == 'm' ? memory_after : threads_after;
            left = after;
            nyxpm::touch_pages(p, 200 * M);
            CHECK((left == -1) == (after < 3));   // three threads beside the caller's
            left = -1;
            CHECK(present(p, 200 * M) * kPage == 200 * M);
            munmap(p, 200 * M);
        }
    } else {
        return 2;
    }
    std::printf("ok\n");
    return 0;
}
