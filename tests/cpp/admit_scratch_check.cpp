// Host-side checks of the scratch part of the serving loop's admission
// (eigenrand_gb300/csrc/gr_admit.h), no GPU.
#include <cstdio>

#include "../../eigenrand_gb300/csrc/gr_admit.h"

using gr::AdmitReq;
using gr::Admission;

static int bad = 0;
#define CHECK(c)                                            \
  do {                                                      \
    if (!(c)) {                                             \
      std::printf("line %d: %s\n", __LINE__, #c);           \
      ++bad;                                                \
    }                                                       \
  } while (0)

int main() {
  {  // scratch counts, and comes back when the work is done
    Admission a(3, 100, 4, 1e9);
    CHECK(a.submit({1, 0, 30, 0.0, 40}) && a.submit({2, 1, 20, 0.1, 20}) && a.submit({3, 2, 10, 0.2}));
    auto r = a.admit(1.0);
    CHECK(r.size() == 2 && r[0].ticket == 1 && r[0].scratch == 40 && r[1].ticket == 3 && r[1].scratch == 0);
    CHECK(a.used() == 80);
    CHECK(a.admit(1.1).empty());  // 20 + 20 do not fit while others run
    a.finish(0);
    a.release(40);
    r = a.admit(1.2);
    CHECK(r.size() == 1 && r[0].ticket == 2 && r[0].scratch == 20 && a.used() == 80);
  }
  {  // results that are kept and nothing running: what is left, if the output fits
    Admission a(2, 100, 4, 1e9);
    CHECK(a.submit({1, 0, 60, 0.0, 40}));
    CHECK(a.admit(0.0).size() == 1 && a.used() == 100);
    a.finish(0);
    a.release(40);  // the result stays
    CHECK(a.submit({2, 1, 30, 0.1, 70}) && a.submit({3, 0, 50, 0.2, 10}));
    auto r = a.admit(0.3);
    CHECK(r.size() == 1 && r[0].ticket == 2 && r[0].scratch == 10 && a.used() == 100);
    a.finish(1);
    a.release(10);
    CHECK(a.admit(0.4).empty());  // 50 never fits beside 90
    a.release(60);
    r = a.admit(0.5);
    CHECK(r.size() == 1 && r[0].ticket == 3 && r[0].scratch == 10 && a.used() == 90);
  }
  {  // an output of the whole budget is accepted and runs without scratch
    Admission a(1, 100, 1, 1e9);
    CHECK(a.submit({1, 0, 100, 0.0, 0}) && !a.submit({2, 0, 101, 0.0, 0}));
    auto r = a.admit(0.0);
    CHECK(r.size() == 1 && r[0].scratch == 0);
  }
  {  // a request that waits for scratch too long holds back what is behind it
    Admission a(4, 100, 4, 0.25);
    CHECK(a.submit({1, 0, 50, 0.0}) && a.admit(0.0).size() == 1);
    CHECK(a.submit({2, 1, 40, 0.1, 60}) && a.submit({3, 2, 5, 0.1}));
    CHECK(a.admit(0.2).size() == 1);  // 3 goes ahead
    CHECK(a.submit({4, 3, 5, 0.3}));
    CHECK(a.admit(0.5).empty());
    a.finish(0);
    a.finish(2);
    auto r = a.admit(0.6);
    CHECK(r.size() == 1 && r[0].ticket == 2 && r[0].scratch == 5 && a.used() == 100);
  }
  if (!bad) std::printf("ok\n");
  return bad ? 1 : 0;
}
