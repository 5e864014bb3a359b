// Explores every order in which the CTAs of a 2 x 2 grid can go through the
// resident solve's iterations, and counts the publications of a residual into a
// slot that some CTA has yet to read (drot::residual_slot).
//
// A CTA in iteration t: its words of t are added when it enters t (the earliest,
// so the others get as far ahead as they can); its items are done when the CTAs
// of its band and of its chunk have entered t, its mass when all have.  Its
// residual warp reads the residual that is out (two copies of X: the one of the
// iteration before; one copy: this iteration's, after everything else), when all
// CTAs have published it, and publishes this iteration's when the items are done.
// The CTA goes on to t + 1 when all of that is done.
//
// Prints a line per rule and schedule: <rule> <every> <copies> <states> <overwritten>
#include <array>
#include <cstdio>
#include <set>
#include <vector>

#include "drot_exchange.h"

namespace {

constexpr int kCtas = 4, kIters = 9;

struct Cta {
  int t = 0;
  bool items = false, mass = false, read = false, pub = false;
  bool operator<(const Cta& o) const {
    return std::array<int, 5>{t, items, mass, read, pub} <
           std::array<int, 5>{o.t, o.items, o.mass, o.read, o.pub};
  }
};
typedef std::array<Cta, kCtas> State;

struct Model {
  bool every, two_copies, by_parity;

  bool tested(int t) const { return t >= 0 && (every || t % 2 == 0); }
  int slot(int t) const { return by_parity ? t & 1 : drot::residual_slot(t, every); }
  bool published(const Cta& c, int t) const { return c.t > t || (c.t == t && c.pub); }
  // iteration whose residual is read during t (-1: none)
  int reads(int t) const {
    const int u = two_copies ? t - 1 : t;
    return tested(u) ? u : -1;
  }
  bool has_read(const Cta& c, int u) const {
    const int at = two_copies ? u + 1 : u;
    return c.t > at || (c.t == at && c.read);
  }

  // Every step that `s` allows; overwritten: publications over an unread slot.
  void next(const State& s, std::vector<State>& out, long& overwritten) const {
    for (int k = 0; k < kCtas; ++k) {
      const Cta& c = s[k];
      if (c.t >= kIters) continue;
      auto step = [&](auto change) {
        State n = s;
        change(n[k]);
        out.push_back(n);
      };
      bool band = true, all = true;
      for (int j = 0; j < kCtas; ++j) {
        const bool in = s[j].t >= c.t;
        all &= in;
        if (j / 2 == k / 2 || j % 2 == k % 2) band &= in;
      }
      if (!c.items && band) step([](Cta& n) { n.items = true; });
      if (!c.mass && all) step([](Cta& n) { n.mass = true; });
      // the residual warp, in its order
      const int u = reads(c.t);
      auto out_there = [&]() {
        for (int j = 0; j < kCtas; ++j)
          if (!published(s[j], u)) return false;
        return true;
      };
      const bool read_first = two_copies;
      if (!c.read && (read_first || c.pub) && (u < 0 || out_there()) &&
          (read_first || (c.items && c.mass)))
        step([](Cta& n) { n.read = true; });
      if (!c.pub && (c.read || !read_first) && (!tested(c.t) || c.items)) {
        if (tested(c.t))
          for (int v = 0; v < c.t; ++v)
            if (tested(v) && slot(v) == slot(c.t))
              for (int j = 0; j < kCtas; ++j)
                if (!has_read(s[j], v)) ++overwritten;
        step([](Cta& n) { n.pub = true; });
      }
      if (c.items && c.mass && c.read && c.pub)
        step([](Cta& n) {
          const int t = n.t + 1;
          n = Cta();
          n.t = t;
        });
    }
  }
};

}  // namespace

int main() {
  for (int rule = 0; rule < 2; ++rule)
    for (int every = 0; every < 2; ++every)
      for (int copies = 1; copies <= 2; ++copies) {
        Model m;
        m.every = every != 0;
        m.two_copies = copies == 2;
        m.by_parity = rule == 1;
        std::set<State> seen;
        std::vector<State> open(1), more;
        seen.insert(open[0]);
        long overwritten = 0;
        while (!open.empty()) {
          const State s = open.back();
          open.pop_back();
          more.clear();
          m.next(s, more, overwritten);
          for (const State& n : more)
            if (seen.insert(n).second) open.push_back(n);
        }
        std::printf("%s %d %d %zu %ld\n", rule ? "parity" : "slot", every, copies, seen.size(),
                    overwritten);
      }
  return 0;
}
