"""Work items of the expert-indexed decode kernels (engine_b200/csrc/hq_work_items.h, compiled for the host): the workspace of
the dispatch tables is a run of 32-bit words that may start at any of them, and where an item lies does not depend on how a
caller splits its assignments into tokens and slots.  Addresses are watched by the compiler's alignment sanitizer."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "hq_work_items.h"
WIDE
using namespace hq;
int main() {
  const int shapes[][3] = {{1, 8, 128}, {4, 8, 128}, {5, 8, 128}, {64, 8, 128}, {3, 64, 7}, {4096, 4, 512}};
  for (auto& s : shapes) {
    const DispatchLayout l = dispatch_layout(s[0], s[1], s[2]);
    for (int shift = 0; shift < 4; ++shift) {                    // a workspace behind an odd number of words
      int32_t* block = (int32_t*)aligned_alloc(16, (size_t)(l.total_words + 8) / 4 * 16 + 16);
      int32_t* ws = block + shift;
      for (int64_t i = 0; i < l.max_items; ++i) put_decode_item(ws, (int)l.rows_at, (int)i, 3 * (int)i, 5 * (int)i, 1 + (int)i % 8);
      for (int64_t i = 0; i < l.max_items; ++i) {
        const DecodeItem v = READ(ws, (int)l.rows_at, (int)i);
        if (v.expert != 3 * i || v.row0 != 5 * i || v.rows != 1 + i % 8) return 2;
      }
      free(block);
    }
    // the last item ends where the workspace does
    if (l.rows_at + l.max_items != l.total_words) return 3;
    if (l.tile_rows != (s[0] <= 4 ? 4 : 8)) return 4;
  }
  return 0;
}
"""


def run(tmp_path, wide, read):
    src, exe = str(tmp_path / "items.cpp"), str(tmp_path / "items")
    with open(src, "w") as f:
        f.write(PROGRAM.replace("WIDE", wide).replace("READ", read))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=alignment", "-fno-sanitize-recover=all", "-I",
                    os.path.join(ROOT, "engine_b200", "csrc"), src, "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True)


def test_items_are_read_at_any_word(tmp_path):
    res = run(tmp_path, "", "decode_item")
    assert res.returncode == 0, res.stderr


def test_a_wide_read_is_seen(tmp_path):
    # the reader this rule excludes: two words of an item in one 8-byte load
    wide = ("struct alignas(8) Pair { int32_t x, y; };\n"
            "hq::DecodeItem wide(const int32_t* ws, int rows_at, int i) {\n"
            "  const Pair v = *(const Pair*)(ws + 4 + 2 * i);\n"
            "  return hq::DecodeItem{v.x, v.y, ws[rows_at + i]};\n"
            "}\n")
    res = run(tmp_path, wide, "wide")
    assert res.returncode != 0 and "misaligned" in res.stderr


def test_the_kernels_read_items_so():
    with open(os.path.join(ROOT, "engine_b200", "csrc", "hq_gemv_shared.cuh")) as f:
        text = f.read()
    assert "decode_item(p.tiles, rows_at, " in text and re.search(r"p\.tiles *[\[+]|_cast<[^>]*>\(p\.tiles", text) is None


FIXED = r"""
#include <stdio.h>
#include <initializer_list>
#include "hq_work_items.h"
using namespace hq;
int main() {
  // every call the header promises the fixed arrays for, at the sizes where its tables are largest
  const int experts[] = {1, 7, 8, 128, 511, 512};
  for (int e : experts)
    for (int k = 1; k <= 64; ++k)
      for (int64_t t : {(int64_t)1, (int64_t)4, (int64_t)5, (int64_t)(62968 / k), (int64_t)(kCompatMaxAssign / k)}) {
        const int64_t ws = dispatch_layout(t, k, e).total_words;
        if (compat_words(t * k, e, ws) > kCompatWords || ws > dispatch_words_up_to(65536, 512)) {
          printf("%d experts, %lld x %d\n", e, (long long)t, k);
          return 1;
        }
      }
  return 0;
}
"""


def test_fixed_arrays_hold_what_the_headers_promise(tmp_path):
    src, exe = str(tmp_path / "fixed.cpp"), str(tmp_path / "fixed")
    with open(src, "w") as f:
        f.write(FIXED)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "engine_b200", "csrc"), src, "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    with open(os.path.join(ROOT, "include", "hanzoquant_compat.h")) as f:
        assert "calls of up to 65536 assignments and 512 experts" in " ".join(f.read().replace("*", " ").split())
    # the arrays are sized by these rules, not by numbers of their own
    for name, size in (("hq_compat.cu", "g_compat_scratch[kCompatWords]"), ("hq_dispatch.cu", "g_noalloc_scratch[kNoAllocWords]")):
        with open(os.path.join(ROOT, "engine_b200", "csrc", name)) as f:
            text = f.read()
        assert size in text and re.search(r"(Compat|NoAlloc)(Ws)?Words = [0-9(]", text) is None


def test_tables_of_any_number_of_experts_get_their_shared_memory(tmp_path):
    src, exe = str(tmp_path / "smem.cpp"), str(tmp_path / "smem")
    with open(src, "w") as f:
        f.write('#include <stdio.h>\n#include "hq_work_items.h"\n'
                "int main() {\n"
                "  for (int e = 1; e <= 4096; ++e)\n"
                '    printf("%lld %d\\n", (long long)hq::dispatch_smem(e), (int)hq::dispatch_asks_for_smem(hq::dispatch_smem(e)));\n'
                "}\n")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "engine_b200", "csrc"), src, "-o", exe], check=True)
    lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    declared = (2 * 256 + 2 * 32) * 4                # what the kernels declare: ids and keys of few assignments, warp totals
    for e in range(1, 4097):
        dynamic, asks = int(lines[2 * e - 2]), int(lines[2 * e - 1])
        assert dynamic >= 4 * 13 * e
        assert dynamic + declared <= (227 if asks else 48) * 1024, e
