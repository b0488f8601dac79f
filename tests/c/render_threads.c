/* Renders scenes on host threads of their own: n threads, each `calls`
   frames of one scene on one stream (noalloc[i]: by gbv_render_noalloc).
   Returns the number of calls that failed; *message: one of their errors. */
#include <pthread.h>
#include <stdio.h>
#include <string.h>
#include "gbvol.h"

typedef struct {
  const gbv_scene *scene;
  float *accum;
  void *stream;
  int width, height, noalloc, calls, failed;
  char message[256];
} job;

static void *work(void *arg) {
  job *j = (job *)arg;
  for (int k = 0; k < j->calls; k++) {
    const gbv_status st =
        j->noalloc ? gbv_render_noalloc(j->scene, j->accum, j->width, j->height, 0, 1, 0, j->stream)
                   : gbv_render(j->scene, j->accum, j->width, j->height, 0, 1, 0, j->stream);
    if (st != GBV_OK && j->failed++ == 0) snprintf(j->message, sizeof j->message, "%s", gbv_last_error());
  }
  return 0;
}

int render_threads(const gbv_scene *scenes, float *const *accums, void *const *streams, const int *noalloc, int n,
                   int width, int height, int calls, char message[256]) {
  enum { MAX = 32 };
  pthread_t threads[MAX];
  job jobs[MAX];
  int failed = 0;
  if (n > MAX) return -1;
  message[0] = 0;
  memset(jobs, 0, sizeof jobs);
  for (int i = 0; i < n; i++) {
    jobs[i].scene = scenes + i;
    jobs[i].accum = accums[i];
    jobs[i].stream = streams[i];
    jobs[i].width = width;
    jobs[i].height = height;
    jobs[i].noalloc = noalloc[i];
    jobs[i].calls = calls;
    if (pthread_create(threads + i, 0, work, jobs + i) != 0) return -1;
  }
  for (int i = 0; i < n; i++) {
    pthread_join(threads[i], 0);
    failed += jobs[i].failed;
    if (jobs[i].failed) memcpy(message, jobs[i].message, sizeof jobs[i].message);
  }
  return failed;
}
