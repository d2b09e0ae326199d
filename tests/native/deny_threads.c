/* For LD_PRELOAD: pthread_create fails, as where a process may have no more
 * threads, while deny_threads(1) is in force. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

static volatile int denied, count;

void deny_threads(int on) { denied = on; }
int threads_denied(void) { return count; }

int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  typedef int (*create)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  if (denied) {
    __sync_fetch_and_add(&count, 1);
    return EAGAIN;
  }
  return ((create)dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}
