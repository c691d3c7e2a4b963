"""Which activations a group of the network's passes takes (csrc/host/pass_room.hpp), on the host with an
allocator that refuses what it is told to: whatever is refused the handle's own room is there, a size
that was refused is not tried again, a capture never takes or moves the larger room, and what a call gets
is always allocated at that moment."""
import subprocess

from native import emulation as E

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "host/pass_room.hpp"
#define CHECK(x) do { if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1; } while (0)
int main() {
  for (int own = 1; own <= 3; ++own)
    for (int limit = 0; limit <= 20; ++limit)
      for (int per = 1; per <= 2; ++per) {
        fc::PassRoom room;
        room.own = own;
        int held = 0, tries = 0;  // what the larger room holds
        std::vector<int> refused;
        auto grow = [&](int passes) {
          ++tries;
          for (int r : refused) if (passes >= r) return held = 0, false;  // asked again
          held = passes <= limit ? passes : 0;
          if (!held) refused.push_back(passes);
          return held > 0;
        };
        const int mine = own >= per ? own / per * per : 1;
        for (int step = 0; step < 60; ++step) {
          const int pairs = (step * 7 + own) % 8 + 1, want = per * pairs, before = held, asked = tries;
          const bool capturing = step % 3 == 2;
          const auto c = room.choose(want, per, capturing, grow);
          CHECK(c.passes >= 1 && c.passes <= (want > mine ? want : mine) && (c.passes % per == 0 || c.passes == 1));
          CHECK(c.in_group ? held >= c.passes : c.passes <= own);
          CHECK(held == room.group);
          if (capturing) CHECK(!c.in_group && held == before && tries == asked);
          if (want <= mine) CHECK(!c.in_group && c.passes == want && tries == asked);
          if (!capturing && want > mine) {
            const int most = limit / per * per;  // the most that is to be had
            CHECK(c.passes == (most > mine ? (want < most ? want : most) : mine) || held >= c.passes);
            CHECK(c.passes >= mine);
          }
          for (int r : refused) CHECK(c.passes < r || !c.in_group);
        }
        const int asked = tries;
        for (int pairs = 1; pairs <= 8; ++pairs) room.choose(per * pairs, per, false, grow);
        const int settled = tries;
        for (int pairs = 8; pairs >= 1; --pairs) room.choose(per * pairs, per, false, grow);
        CHECK(settled - asked <= 8 && tries == settled);  // nothing is allocated twice
        CHECK(refused.size() <= 8);
      }
  // a smaller group does not give up a larger room, a larger one replaces it
  fc::PassRoom room;
  room.own = 2;
  int grown = 0;
  auto grow = [&](int p) { return grown = p, true; };
  CHECK(room.choose(8, 2, false, grow).passes == 8 && grown == 8);
  CHECK(room.choose(4, 2, false, grow).passes == 4 && room.group == 8 && grown == 8);
  CHECK(room.choose(16, 2, true, grow).passes == 2 && room.group == 8);
  CHECK(room.choose(16, 2, false, grow).passes == 16 && grown == 16);
  return 0;
}
"""


def test_every_refusal(tmp_path):
    src, exe = tmp_path / "room.cpp", tmp_path / "room"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", f"-I{E.HEADER.parent.parent}", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
