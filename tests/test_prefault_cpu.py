"""The download buffers' prefault (csrc/afl_host.h): contents are kept, for
present, absent and partly present pages, at odd offsets and sizes, on memory that
cannot be written, and on null and tiny buffers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
#include "afl_host.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
int main() {
  afl::prefault(nullptr, 1 << 20);
  char small[64] = {7};
  afl::prefault(small, sizeof small);
  for (size_t mb : {1, 9, 70}) {
    const size_t n = (mb << 20) + 12345;
    for (int state = 0; state < 3; ++state) {  // pages absent, every fourth present, all
      char *p = static_cast<char *>(mmap(nullptr, n, PROT_READ | PROT_WRITE,
                                         MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
      for (size_t at = 0; state && at < n; at += state == 1 ? 4 * 4096 : 4096) p[at] = 5;
      afl::prefault(p + 3, n - 7);
      for (size_t at = 0; at < n; ++at) {
        const char want = state && at % (state == 1 ? 4 * 4096 : 4096) == 0 ? 5 : 0;
        if (p[at] != want) return printf("changed at %zu\n", at), 1;
      }
      munmap(p, n);
    }
    char *ro = static_cast<char *>(mmap(nullptr, n, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    afl::prefault(ro, n);
    munmap(ro, n);
  }
  puts("ok");
}
"""


def test_prefault_keeps_contents(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(CODE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I",
                           os.path.join(ROOT, "aether-core-engine_b200", "csrc"), str(src), "-o",
                           str(exe), "-lpthread"])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


NO_MEMORY = r"""
#include "afl_host.h"
#include <cstdio>
#include <cstdlib>
#include <new>
// The allocation number `fail_at` from here on throws.
static int fail_at = -1;
void *operator new(size_t n) {
  if (fail_at >= 0 && fail_at-- == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
int main() {
  for (int at = 0; at < 4; ++at) {
    const size_t n = size_t(70) << 20;
    char *p = static_cast<char *>(mmap(nullptr, n, PROT_READ | PROT_WRITE,
                                       MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    fail_at = at;
    afl::prefault(p, n);
    fail_at = -1;
    munmap(p, n);
  }
  puts("ok");
}
"""


def test_prefault_without_host_memory_for_its_threads(tmp_path):
    """No exception leaves it and no thread is left unjoined, whichever thread's state cannot
    be allocated: it is called from the C entries."""
    src, exe = tmp_path / "n.cpp", tmp_path / "n"
    src.write_text(NO_MEMORY)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I",
                           os.path.join(ROOT, "aether-core-engine_b200", "csrc"), str(src), "-o",
                           str(exe), "-lpthread"])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
