"""A device that runs out of memory, as far as the library can tell: a preloaded stand-in for some of the
CUDA runtime's calls, which refuses allocations past a limit on the host, before they reach the driver.
It also keeps a log of the calls (M allocation, x refused one, F free, S and D stream and device
synchronisation, G cudaGetDevice, K kernel launch) and can report a launch as failed."""
import json
import os
import subprocess
import sys

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <pthread.h>
#include <stddef.h>
#include <string.h>
typedef struct { void* p; size_t n; } Block;
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static Block blocks[1 << 16];
static int nblocks, refused, fail_launch = -1;
static __thread int pending;  /* the runtime's last error is a thread's own, too */
static size_t used, peak, limit;
static char log_[1 << 22];
static size_t nlog;
static void note(char c) { if (nlog + 1 < sizeof log_) log_[nlog++] = c; }
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaMalloc(void** p, size_t n) {
  pthread_mutex_lock(&mu);
  int rc = 2;  /* cudaErrorMemoryAllocation */
  if ((limit && used + n > limit) || nblocks == 1 << 16) {
    ++refused;
    pending = 2;
    note('x');
  } else if ((rc = ((int (*)(void**, size_t))real("cudaMalloc"))(p, n)) == 0) {
    blocks[nblocks++] = (Block){*p, n};
    used += n;
    if (used > peak) peak = used;
    note('M');
  }
  pthread_mutex_unlock(&mu);
  return rc;
}
int cudaFree(void* p) {
  pthread_mutex_lock(&mu);
  for (int k = 0; k < nblocks; ++k)
    if (blocks[k].p == p) {
      used -= blocks[k].n;
      blocks[k] = blocks[--nblocks];
      break;
    }
  note('F');
  pthread_mutex_unlock(&mu);
  return ((int (*)(void*))real("cudaFree"))(p);
}
static int logged(char c) {
  pthread_mutex_lock(&mu);
  note(c);
  pthread_mutex_unlock(&mu);
  return 0;
}
int cudaStreamSynchronize(void* s) { logged('S'); return ((int (*)(void*))real("cudaStreamSynchronize"))(s); }
int cudaDeviceSynchronize(void) { logged('D'); return ((int (*)(void))real("cudaDeviceSynchronize"))(); }
int cudaGetDevice(int* d) { logged('G'); return ((int (*)(int*))real("cudaGetDevice"))(d); }
int cudaLaunchKernelExC(const void* cfg, const void* f, void** args) {
  logged('K');
  if (fail_launch == 0) { fail_launch = -1; return pending = 9; }  /* cudaErrorInvalidConfiguration */
  if (fail_launch > 0) --fail_launch;
  return ((int (*)(const void*, const void*, void**))real("cudaLaunchKernelExC"))(cfg, f, args);
}
int cudaPeekAtLastError(void) { return pending ? pending : ((int (*)(void))real("cudaPeekAtLastError"))(); }
int cudaGetLastError(void) {
  const int e = pending;
  pending = 0;
  return e ? e : ((int (*)(void))real("cudaGetLastError"))();
}
void short_memory_limit(long long bytes) { limit = (size_t)bytes; }
void short_memory_fail_launch(int k) { fail_launch = k; }
long long short_memory_used(void) { return (long long)used; }
long long short_memory_peak(void) { return (long long)peak; }
void short_memory_reset(void) { peak = used; refused = 0; nlog = 0; }
int short_memory_refused(void) { return refused; }
const char* short_memory_log(void) { log_[nlog] = 0; return log_; }
"""

PRELUDE = """
import ctypes, json, os, sys
sys.path[:0] = json.loads(os.environ["SHORT_MEMORY_PATH"])
import numpy as np
import hams_b200, meshgen
mem = ctypes.CDLL(os.environ["LD_PRELOAD"])
mem.short_memory_limit.argtypes = [ctypes.c_longlong]
mem.short_memory_used.restype = mem.short_memory_peak.restype = ctypes.c_longlong
mem.short_memory_log.restype = ctypes.c_char_p
log = lambda: mem.short_memory_log().decode()
rel = lambda a, b: float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))
answer = lambda **kw: print("ANSWER " + json.dumps(kw))
def deck(bodies):
    xyz, ncn, ncon, cnt = meshgen.combine(bodies)
    return hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((len(bodies), 3)))
"""


def build(folder):
    """The stand-in as a shared object in `folder`."""
    src, so = os.path.join(folder, "short_memory.c"), os.path.join(folder, "short_memory.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["/usr/bin/gcc", "-O1", "-fPIC", "-shared", "-o", so, src, "-ldl", "-lpthread"], check=True)
    return so


def run(so, script, timeout=300):
    """What `script` (after PRELUDE, in a process of its own with the stand-in) hands to answer()."""
    here = os.path.dirname(os.path.abspath(__file__))
    path = [here] + [os.path.join(os.path.dirname(here), d) for d in ("hams-mrel_b200", "oracle")]
    p = subprocess.run([sys.executable, "-c", PRELUDE + script], capture_output=True, text=True, timeout=timeout,
                       env=dict(os.environ, LD_PRELOAD=so, SHORT_MEMORY_PATH=json.dumps(path)))
    lines = [x for x in p.stdout.splitlines() if x.startswith("ANSWER ")]
    assert p.returncode == 0 and lines, p.stdout[-2000:] + p.stderr[-4000:]
    return json.loads(lines[-1][7:])
