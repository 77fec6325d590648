"""A data file that its file system has no room for: Stop reports GZ_IO, as write calls would, although
it copies into a mapping of the file, where a store to a page that cannot be allocated is a SIGBUS.

The pages are made present by csrc/file_pages.h, checked here on the CPU with a mapping that reaches past
the end of its file (pages that cannot be had, as on a full file system), and through Stop in a tmpfs
that is too small."""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from gazelle_plugin_gb300 import shuffle as S
from gazelle_plugin_gb300 import workloads as W
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <stdio.h>
#include <stdlib.h>
#include <sys/mman.h>
#include <memory>
#include "file_pages.h"
// d PATH FILE_BYTES MAP_BYTES WINDOW THREADS ALLOCATE: prints the windows that came up and the present pages
int main(int, char** v) {
  const int64_t file = atoll(v[2]), total = atoll(v[3]), W = atoll(v[4]);
  const bool heap = v[1][0] == 0;
  uint8_t* map;
  int fd = -1;
  std::unique_ptr<uint8_t[]> mem;
  if (heap) {
    mem.reset(new uint8_t[total]);
    map = mem.get();
  } else {
    fd = open(v[1] + (v[1][0] == '+'), O_RDWR | O_CREAT | O_TRUNC, 0600);
    if (fd < 0 || ftruncate(fd, file) != 0) return 2;
    map = static_cast<uint8_t*>(mmap(nullptr, total, PROT_READ | PROT_WRITE, MAP_SHARED, fd, 0));
    if (map == MAP_FAILED) return 2;
  }
  auto pages = std::make_shared<gz::PageToucher>(map, total, W, heap ? -1 : open("/dev/zero", O_RDONLY),
                                                 v[6][0] == '1' ? fd : -1);
  std::vector<std::thread> th;
  for (int i = 0; i < atoi(v[5]); i++) th.emplace_back([pages] { while (pages->Work()) {} });
  const int64_t nw = (total + W - 1) / W;
  int64_t ok = 0;
  for (int64_t w = 0; w < nw; w++) ok += pages->Wait(w);
  for (auto& t : th) t.join();
  const int64_t page = sysconf(_SC_PAGESIZE), n = (total + page - 1) / page;
  std::vector<unsigned char> in(n);
  int64_t present = 0;
  if (!heap && mincore(map, total, in.data()) == 0)
    for (unsigned char c : in) present += c & 1;
  if (v[1][0] == '+') {  // ranges that end on a boundary and 50 bytes after it, where the file ends there
    if (ftruncate(fd, page * 700) != 0) return 2;
    const int zero = open("/dev/zero", O_RDONLY);
    if (!gz::MakePresent(map, page * 3 + 100, page * 700, zero, -1)) return 3;
    if (gz::MakePresent(map, page * 3 + 100, page * 700 + 50, zero, -1)) return 4;
  }
  printf("%ld of %ld windows, %ld of %ld pages\n", (long)ok, (long)nw, (long)present, (long)n);
  return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("file_pages")
    (d / "d.cc").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "gazelle_plugin_gb300", "csrc"),
                    str(d / "d.cc"), "-o", str(d / "d")], check=True)
    return str(d / "d")


@pytest.mark.parametrize("allocate", ["0", "1"])
@pytest.mark.parametrize("threads", [0, 7])
@pytest.mark.parametrize("total", [1, (2 << 20) - 1, 2 << 20, (5 << 20) + 12345])
def test_pages_come_up_window_by_window(driver, tmp_path, total, threads, allocate):
    nw, page = -(-total // (2 << 20)), os.sysconf("SC_PAGESIZE")
    n = -(-total // page)
    r = subprocess.run([driver, str(tmp_path / "f"), str(total), str(total), str(2 << 20), str(threads), allocate], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, f"{nw} of {nw} windows, {n} of {n} pages\n")
    r = subprocess.run([driver, "", "0", str(total), str(2 << 20), str(threads), allocate], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith(f"{nw} of {nw} windows")


def test_every_page_of_a_range_off_the_page_boundaries(driver, tmp_path):
    total = os.sysconf("SC_PAGESIZE") * 800
    r = subprocess.run([driver, "+" + str(tmp_path / "f"), str(total), str(total), str(2 << 20), "0", "0"], capture_output=True, text=True)
    assert r.returncode == 0, r


@pytest.mark.parametrize("threads", [0, 7])
def test_pages_that_cannot_be_had_are_an_error_not_a_signal(driver, tmp_path, threads):
    total = 20 << 20
    r = subprocess.run([driver, str(tmp_path / "f"), str(total // 2), str(total), str(2 << 20), str(threads), "0"], capture_output=True, text=True)
    assert r.returncode == 0, r  # (a signal is negative)
    # with helpers ahead of it the caller may learn of it at any window
    assert int(r.stdout.split()[0]) in ([5] if threads == 0 else range(6))


@pytest.mark.parametrize("allocate", ["0", "1"])
@pytest.mark.parametrize("threads", [0, 7])
def test_pages_of_a_full_file_system(driver, tmp_path, threads, allocate):
    total = 20 << 20
    mnt, mount = _small_tmpfs(tmp_path)
    r = subprocess.run(mount + [driver, str(mnt / "f"), str(total), str(total), str(2 << 20), str(threads), allocate],
                       capture_output=True, text=True)
    assert r.returncode == 0, r
    assert int(r.stdout.split()[0]) in ([4] if threads == 0 else range(5))


def _small_tmpfs(tmp_path):
    """A directory and the command prefix that runs a program with 8 MB of tmpfs mounted there for it alone."""
    mnt = tmp_path / "small"
    mnt.mkdir()
    mount = ["unshare", "-m", "sh", "-c", 'mount -t tmpfs -o size=8m none "$0" && exec "$@"', str(mnt)]
    if subprocess.run(mount + ["true"], capture_output=True).returncode != 0:
        pytest.skip("no file system of its own may be mounted here")
    return mnt, mount


def _stop(path, device, tasks, n=56, **kw):
    """Map tasks of the wide table that write about 0.72 MB a batch (a child process: see below)."""
    rng = np.random.default_rng(5)
    batches = [W.c2_batch(rng, 4096) for _ in range(n)]
    w = S.ShuffleSplitterJniWrapper()

    def task(p):
        h = w.make(S.NativePartitioning("hash", 200, None, W.C2_KEYS, list(W.C2_SCHEMA)), dataFile=p,
                   keep_output_on_device=device, **kw)
        for b in batches:
            a, z = b.addrs_sizes()
            w.split(h, b.num_rows, a, z)
        try:
            w.stop(h)
            return open(p, "rb").read()
        except S.SplitterError as e:
            return e.status
        finally:
            w.close(h)

    # one alone, whose pages several threads make present, or as many at once as leave each only its own
    with ThreadPoolExecutor(tasks) as ex:
        assert list(ex.map(task, [f"{path}.{i}" for i in range(tasks)])) == [S.GZ_IO] * tasks
    # and the library goes on
    data = task(os.path.join(os.path.dirname(path), "..", "other"))
    assert data == O.run_oracle(W.C2_SCHEMA, batches, 200, W.C2_KEYS).data
    print("reported")


@pytest.mark.gpu
@pytest.mark.parametrize("device,tasks", [(0, 1), (1, 1), (0, 16)])
def test_gpu_stop_into_a_full_file_system_is_an_io_error(tmp_path, device, tasks):
    mnt, mount = _small_tmpfs(tmp_path)
    call = f"from tests.test_data_file_space import _stop; _stop({str(mnt / 'x.data')!r}, {device}, {tasks})"
    r = subprocess.run(mount + [sys.executable, "-c", call], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reported" in r.stdout, (r.returncode, r.stdout, r.stderr)


@pytest.mark.gpu
def test_gpu_large_file_gathered_by_the_cpu_into_a_full_file_system_is_an_io_error(tmp_path):
    """From 256 MB on the CPU copies into a mapping as well (passes may lie in local-dir files)."""
    mnt, mount = _small_tmpfs(tmp_path)
    call = (f"from tests.test_data_file_space import _stop; "
            f"_stop({str(mnt / 'x.data')!r}, 0, 1, n=400, host_budget=1 << 40, localDirs={str(tmp_path)!r})")
    r = subprocess.run(mount + [sys.executable, "-c", call], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reported" in r.stdout, (r.returncode, r.stdout, r.stderr)


SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <stdio.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>
/* no shared mapping of a file named *.data, as of a file system that has none */
void* mmap(void* a, size_t n, int prot, int flags, int fd, off_t off) {
  static void* (*next)(void*, size_t, int, int, int, off_t);
  if (!next) next = (void* (*)(void*, size_t, int, int, int, off_t))dlsym(RTLD_NEXT, "mmap");
  if (fd >= 0 && (flags & MAP_SHARED) && (prot & PROT_WRITE)) {
    char link[64], path[512];
    snprintf(link, sizeof(link), "/proc/self/fd/%d", fd);
    const ssize_t l = readlink(link, path, sizeof(path));
    if (l > 5 && memcmp(path + l - 5, ".data", 5) == 0) {
      fprintf(stderr, "no mapping\n");
      errno = ENODEV;
      return MAP_FAILED;
    }
  }
  return next(a, n, prot, flags, fd, off);
}
void* mmap64(void* a, size_t n, int prot, int flags, int fd, off_t off) { return mmap(a, n, prot, flags, fd, off); }
"""


def _stop_unmapped(path, n, device, kw):
    rng = np.random.default_rng(6)
    batches = [W.c2_batch(rng, 4096) for _ in range(n)]
    w = S.ShuffleSplitterJniWrapper()

    def task(p):
        h = w.make(S.NativePartitioning("hash", 200, None, W.C2_KEYS, list(W.C2_SCHEMA)), dataFile=p,
                   keep_output_on_device=device, **kw)
        for b in batches:
            a, z = b.addrs_sizes()
            w.split(h, b.num_rows, a, z)
        w.stop(h)
        data = open(p, "rb").read()
        w.close(h)
        return data

    got = task(path + ".data")
    if "codec" in kw:  # (the compressed bytes are the library's own: those of the mapped path)
        assert got == task(path + ".mapped")
    else:
        assert got == O.run_oracle(W.C2_SCHEMA, batches, 200, W.C2_KEYS).data
    print("equal")


@pytest.mark.gpu
@pytest.mark.parametrize("n,device,kw", [(9, 0, {}), (61, 1, {}), (61, 0, {"codec": "lz4"}),
                                         (370, 0, {"host_budget": 1 << 40, "localDirs": "."})])
def test_gpu_stop_into_a_file_that_cannot_be_mapped(tmp_path, n, device, kw):
    """Files of two windows and of several with a ragged last one, through a block of host memory and write
    calls; a large one that the CPU gathers."""
    (tmp_path / "s.c").write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(tmp_path / "s.c"), "-o", str(tmp_path / "s.so"), "-ldl"], check=True)
    call = f"from tests.test_data_file_space import _stop_unmapped as f; f({str(tmp_path / 'x')!r}, {n}, {device}, {kw!r})"
    r = subprocess.run([sys.executable, "-c", call], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(tmp_path / "s.so")))
    assert r.returncode == 0 and "equal" in r.stdout and "no mapping" in r.stderr, (r.returncode, r.stdout, r.stderr)
