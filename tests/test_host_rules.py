"""Sizes and rules the host decides for the kernels (csrc/pbf_internal.cuh),
evaluated on the CPU: small C++ programs against the library, over the sizes
where a rule can go wrong."""
from __future__ import annotations

import subprocess

from conftest import ROOT


def evaluate(pbf, tmp_path, code: str) -> list[str]:
    """Lines printed by a program whose main() is `code`."""
    import importlib

    build = importlib.import_module(pbf.__name__ + ".build")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text('#include <algorithm>\n#include <cstdint>\n#include <cstdio>\n'
                   '#include "pbf_host.hpp"\nusing namespace pbf;\n'
                   f'int main() {{\n{code}\n}}\n')
    pkg = pbf.LIB_PATH.parent
    subprocess.run([build.CXX, *build.CXX_FLAGS, "-I", str(pkg / "csrc"), str(src), "-o", str(exe),
                    f"-L{pkg}", "-lpbf_gb300", f"-Wl,-rpath,{pkg}"], check=True, cwd=ROOT)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True,
                          timeout=60).stdout.split("\n")[:-1]


def test_cleared_control_words_hold_every_layout(pbf, tmp_path):
    """A batch's control words are zeroed once, for its capacity: that has to
    cover those of every layout within it (fewer cells can mean smaller scan
    tiles, and more of them)."""
    lines = evaluate(pbf, tmp_path, r"""
  const uint32_t chunk = 2048;
  for (uint32_t c = 1; c < 1200; ++c)
    for (uint32_t cells : {c * chunk - 1, c * chunk, c * chunk + 1}) {
      const CellSortPlan cap = make_cell_sort_plan(100000, cells);
      const size_t zeroed = cell_sort_clear_words(cap);
      if (cap.off_ctl + zeroed > cap.off_small) std::printf("past the words: %u\n", cells);
      for (uint32_t k = 0; k <= c; k = k < 60 ? k + 1 : k * 2) {
        const CellSortPlan p = resize_cell_sort_plan(cap, 1000, std::min(cells, k * chunk));
        if (p.ctl_words > zeroed)
          std::printf("%u of %u cells: %zu words, %zu zeroed\n", p.ncells, cells, p.ctl_words,
                      zeroed);
      }
    }
""")
    assert lines == []


def test_grid_stride_ends_at_the_largest_counts(pbf, tmp_path):
    """The strided loops over cells visit every index once and end, also where
    the index after the last one is past 32 bits."""
    lines = evaluate(pbf, tmp_path, r"""
  const uint32_t stride = kStrideCtas * 256u;
  for (uint32_t end : {0u, 1u, 255u, stride - 1, stride, stride + 1, 3 * stride + 7,
                       0xffffffffu - stride, 0xffffffffu - 1, 0xffffffffu})
    for (uint32_t first : {0u, 1u, 255u, stride / 2, stride - 1}) {
      const uint64_t want = first < end ? ((uint64_t)end - first + stride - 1) / stride : 0;
      uint64_t trips = 0;
      uint64_t at = first;
      for (uint32_t i = first; i < end && trips <= want; i = stride_next(i, stride, end)) {
        if (i != at) std::printf("%u of %u\n", i, end);
        at += stride;
        ++trips;
      }
      if (trips != want) std::printf("%u to %u: %llu trips, not %llu\n", first, end,
                                     (unsigned long long)trips, (unsigned long long)want);
    }
""")
    assert lines == []


def test_items_within_the_largest_counts(pbf, tmp_path):
    """Whether a thread's eight cells lie below the end, also where the index
    after the eighth is past 32 bits."""
    lines = evaluate(pbf, tmp_path, r"""
  for (uint64_t end : {0ull, 1ull, 7ull, 8ull, 9ull, 2048ull, 0xfffffff7ull, 0xfffffff8ull,
                       0xfffffff9ull, 0xffffffffull})
    for (uint64_t at : {0ull, 8ull, 2040ull, 0xffffffe8ull, 0xfffffff0ull, 0xfffffff8ull})
      if (whole_items((uint32_t)at, 8, (uint32_t)end) != (at + 8 <= end))
        std::printf("%llu of %llu\n", (unsigned long long)at, (unsigned long long)end);
""")
    assert lines == []


def test_kernel_attributes_once_per_device(pbf, tmp_path):
    """A setting that belongs to a device is made on each of them, once, and
    again after a failure."""
    lines = evaluate(pbf, tmp_path, r"""
  OncePerDevice once;
  int calls = 0;
  const auto good = [&] { ++calls; return cudaSuccess; };
  const auto bad = [&] { ++calls; return cudaErrorInvalidValue; };
  for (int device : {0, 0, 1, 0, 1, 63, 63}) once.run(device, good);
  if (calls != 3) std::printf("%d calls on three devices\n", calls);
  calls = 0;
  if (once.run(2, bad) != cudaErrorInvalidValue) std::printf("failure lost\n");
  if (once.run(2, good) != cudaSuccess || once.run(2, bad) != cudaSuccess || calls != 2)
    std::printf("after a failure: %d calls\n", calls);
  calls = 0;
  for (int device : {64, 64, 1000}) once.run(device, good);  // beyond what it remembers
  if (calls != 3) std::printf("%d calls beyond the table\n", calls);
""")
    assert lines == []


def test_tuning_survives_the_round_trip(pbf, tmp_path):
    """What pbf_get_tuning reports selects, set again, the passes it was read
    from: for every field, also one thread per particle in the default shapes,
    which the tuner can pick for a small scene."""
    lines = evaluate(pbf, tmp_path, r"""
  int grouped = 0;
  for (uint32_t bits = 0; bits < 128; ++bits) {
    GatherTuning g, back;
    g.one_thread = bits & 1;
    g.fuse_first = bits >> 1 & 1;
    g.staged = bits >> 2 & 1;
    g.radix_sort = bits >> 3 & 1;
    g.masked_build = bits >> 4 & 1;
    if (bits >> 5 & 1) g.block[kKindDelta] = 0;
    if (bits >> 6 & 1) g.batch[kKindXsph] = 1;
    pbf_tuning t;
    to_pbf_tuning(g, nullptr, &t);
    if (to_gather_tuning(t, &back) != PBF_OK) std::printf("%u refused\n", bits);
    if (back.grouped() != g.grouped() || back.one_thread != g.one_thread ||
        back.fuse_first != g.fuse_first || back.staged != g.staged ||
        back.radix_sort != g.radix_sort || back.masked_build != g.masked_build ||
        !std::equal(g.block, g.block + kGatherKinds, back.block) ||
        !std::equal(g.batch, g.batch + kGatherKinds, back.batch))
      std::printf("%u comes back as another\n", bits);
    grouped += g.grouped();
    t.one_thread = 2;
    if (to_gather_tuning(t, &back) != PBF_ERR_INVALID) std::printf("%u: one_thread = 2\n", bits);
  }
  if (grouped != 2) std::printf("eight threads in %d of them\n", grouped);  // either sort
  const pbf_tuning zero{};  // a caller that leaves the field out: as the other fields say
  if (zero.one_thread != GatherTuning().one_thread) std::printf("not the default\n");
""")
    assert lines == []


def test_reference_lists_leave_the_memory(pbf, tmp_path):
    """Neighbour lists of the reference's equations take a bounded share of the
    device whatever its size and the scene's, do not depend on what else is
    allocated while that leaves twice the share, and are dropped where only lists
    too short to hold a set at rest would fit."""
    lines = evaluate(pbf, tmp_path, r"""
  const uint64_t gib = 1ull << 30;
  for (uint64_t total : {8 * gib, 80 * gib, 280 * gib})
    for (uint64_t n : {1ull, 1000ull, 1048576ull, 17000000ull, 34000000ull, 100000000ull,
                       300000000ull, 1073741823ull})
      for (uint32_t maxn : {1u, 8u, 9u, 16u, 24u, 31u, 32u, 40u, 64u, 100u, 128u, 1024u}) {
        const uint32_t all = ref_list_entries(maxn, n, ref_list_room(total, total));
        for (uint64_t eighths = 0; eighths <= 8; ++eighths) {
          const uint64_t left = total / 8 * eighths;
          const uint32_t e = ref_list_entries(maxn, n, ref_list_room(left, total));
          const uint64_t bytes = (uint64_t)paper_list_words(e) * sizeof(uint4) * n;
          const uint32_t most = std::min(128u, std::max(8u, maxn / 8 * 8));
          const char *wrong = nullptr;
          if (bytes > total / 16 || bytes > left / 2) wrong = "too much";
          else if (e % 8 || e > most || (e && e < std::min(most, 32u))) wrong = "entries";
          else if (eighths && e != all) wrong = "depends on the rest";
          else if (e != most && 4 * n * most <= std::min(left / 2, total / 16)) wrong = "too few";
          if (wrong) std::printf("%s: %u of %u, n %llu, %llu of %llu GiB\n", wrong, e, maxn,
                                 (unsigned long long)n, (unsigned long long)(left / gib),
                                 (unsigned long long)(total / gib));
        }
      }
  if (ref_list_entries(128, 4194304, ref_list_room(280 * gib, 280 * gib)) != 128)
    std::printf("4,194,304 particles without whole lists\n");
""")
    assert lines == []


def test_every_sprite_is_drawn(pbf, tmp_path):
    """The threads of the sprites' kernel hold every sprite's number, also where
    the threads number past 2^32."""
    lines = evaluate(pbf, tmp_path, r"""
  for (uint32_t count : {1u, 15u, 16u, 17u, 81920u, (1u << 29) - 1u, 1u << 29, (1u << 29) + 1u,
                         (1u << 30) - 1u}) {
    const uint32_t ctas = sprite_ctas(count);
    if ((uint64_t)ctas * kSpriteCta < (uint64_t)count * kSpriteThreads)
      std::printf("%u: too few CTAs\n", count);
    for (uint32_t block : {0u, ctas / 2u, ctas - 1u})
      for (uint32_t t = 0; t < kSpriteCta; ++t)
        if (sprite_of_thread(block, t) != ((uint64_t)block * kSpriteCta + t) / kSpriteThreads)
          std::printf("%u: thread %u of CTA %u draws %u\n", count, t, block,
                      sprite_of_thread(block, t));
  }
""")
    assert lines == []
