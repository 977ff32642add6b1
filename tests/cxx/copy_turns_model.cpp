// Drives copy_turns (cdocker_b200/csrc/copy_turns.cuh) over a model of the CTA: an mbarrier with an arrival
// count of one, copies that land when a wait succeeds, and a wait that gives up at a chosen turn. Prints the
// first violated rule and exits 1.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "copy_turns.cuh"

namespace {

void fail(const char* what) {
  std::printf("%s\n", what);
  std::exit(1);
}

struct Model {
  int give_up;            // turn (counted from 0) whose wait gives up; -1: none
  bool armed = false;     // the phase's arrival is used up and its copies are in flight
  unsigned phases = 0;    // completed
  int buffer = -1, pending = -1, waits = 0;
  bool flag = false;
  std::vector<int> worked;

  void load(int p) {
    if (flag) fail("copies issued after a wait gave up");
    if (armed) fail("the phase was armed twice");
    armed = true;
    pending = p;
  }
  void land() {
    armed = false;
    ++phases;
    buffer = pending;
  }
  void wait(unsigned parity) {
    if (parity != (phases & 1u)) fail("wait on another phase than the one in flight");
    if (!armed) fail("wait without copies in flight");
    if (waits++ == give_up) flag = true;
    else land();
  }
  void columns(int p) {
    if (!flag && buffer != p) fail("columns of another turn's copies");
  }
  bool failed() const { return flag; }
  void rows(int p) {
    if (armed) fail("rows while copies are in flight");
    worked.push_back(p);
  }
  void drain(unsigned parity) {
    if (!armed || parity != (phases & 1u)) fail("drain of another phase than the one in flight");
    land();
  }
};

}  // namespace

int main() {
  for (int end = 0; end <= 9; ++end)
    for (int step = 1; step <= 5; ++step)
      for (int first = 0; first < step; ++first) {
        const int turns = first < end ? (end - first + step - 1) / step : 0;
        for (int g = -1; g < turns; ++g) {
          Model m;
          m.give_up = g;
          const bool ok = cdk::copy_turns(first, step, end, m);
          if (ok != (g < 0)) fail("the result does not tell whether a wait gave up");
          if (m.armed) fail("left with copies in flight");
          const int want = g < 0 ? turns : g;
          if ((int)m.worked.size() != want) fail("turns done");
          for (int i = 0; i < want; ++i)
            if (m.worked[i] != first + i * step) fail("order of the turns");
        }
      }
  std::printf("ok\n");
  return 0;
}
