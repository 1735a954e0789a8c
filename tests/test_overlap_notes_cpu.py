"""Which launches come behind a call that overlaps the one before it (csrc/rt/ccb_overlap.h): two devices whose default
streams share a handle, two threads, captures beside eager launches, and places that are never launched to again."""
import os
import shutil
import subprocess

import pytest

SOURCE = r'''
#include <cstdio>
#include <thread>
#include <vector>
#include "ccb_overlap.h"
using ccb::LaunchPlace;
#define CHECK(x) if (!(x)) return std::printf("%d: %s\n", __LINE__, #x), 1
int main() {
  ccb::OverlapNotes notes;
  const LaunchPlace first{0, 7, 0}, second{1, 7, 0}, another{0, 8, 0};
  CHECK(!notes.any() && !notes.behind(first));
  notes.note(first);   // two devices, two streams: nobody else's launch settles it
  CHECK(notes.any() && !notes.behind(second) && !notes.behind(another) && notes.any());
  notes.note(second);
  notes.note(first);
  CHECK(notes.kept() == 2 && notes.behind(first) && !notes.behind(first));
  CHECK(notes.any() && notes.behind(second) && !notes.any());

  const LaunchPlace captured{0, 7, 21}, joined{0, 8, 21}, next_capture{0, 7, 22};
  notes.note(first);   // a launch into a capture does not settle what the stream had before it
  CHECK(!notes.behind(captured) && notes.behind(first));
  notes.note(captured);   // within one, other streams too, and no launch outside of it
  CHECK(!notes.behind(first) && !notes.behind(next_capture));
  CHECK(notes.behind(captured) && notes.behind(joined) && notes.behind(captured) && notes.any());

  ccb::OverlapNotes shared;   // threads, each with a stream of its own
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (unsigned long long id = 1; id <= 8; ++id)
    threads.emplace_back([&, id] {
      for (int k = 0; k < 20000; ++k) {
        if (shared.behind({0, id, 0})) ++wrong;
        shared.note({0, id, 0});
        if (!shared.any() || !shared.behind({0, id, 0})) ++wrong;
      }
    });
  for (auto& t : threads) t.join();
  CHECK(wrong == 0 && !shared.any());

  ccb::OverlapNotes many;   // streams that are gone: a bound, and no state that stays
  const size_t most = ccb::OverlapNotes::kMost;
  for (unsigned long long id = 0; id < 3 * most; ++id) many.note({0, id, 0});
  CHECK(many.kept() == most && many.behind({0, 2 * most, 0}) && many.behind({0, 3 * most - 1, 0}) && !many.behind({0, 5, 0}));
  CHECK(!many.behind({0, 3 * most, 0}) && many.kept() == most - 2);
  return 0;
}'''


def test_notes_of_calls_that_overlap(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + os.path.join(root, "csrc", "rt"), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    done = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
