// Preloaded by test_host_paths.py: a thread sleeps between finding nothing to
// do and going to sleep on the condition, so that a notice given without the
// condition's lock comes in between.
#include <dlfcn.h>
#include <pthread.h>
#include <unistd.h>

extern "C" int pthread_cond_wait(pthread_cond_t* c, pthread_mutex_t* m) {
    using Wait = int (*)(pthread_cond_t*, pthread_mutex_t*);
    static const Wait wait = (Wait)dlvsym(RTLD_NEXT, "pthread_cond_wait", "GLIBC_2.3.2");
    usleep(50000);
    return wait(c, m);
}
