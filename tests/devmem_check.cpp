// What asr_b200/csrc/devmem.h promises, on the made-up device of fake_cuda: one case per name on the command line.
#include <cstdio>
#include <cstring>
#include <string>

#include "../asr_b200/csrc/devmem.h"

using namespace asrb;

static const size_t MB = (size_t)1 << 20, GB = (size_t)1 << 30;
static int bad = 0;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); bad = 1; } } while (0)

// a call that plans with its largest array and takes arrays of the given sizes
static bool call(DevStore& st, std::initializer_list<size_t> sizes, const void* ctx = nullptr) {
  MemScope scope(&st, nullptr, ctx);
  size_t most = 0;
  for (size_t s : sizes) most = s > most ? s : most;
  st.plan({most});
  DevMem m[8];
  int k = 0;
  bool ok = true;
  for (size_t s : sizes) ok = ok && m[k++].get(s);
  while (k) m[--k].put();
  return ok;
}

// memory that a call took stays for the next one: no allocation, and no question to the device
static void reuse() {
  DevStore st;
  st.open(0, fake().total);
  CHECK(call(st, {4 * GB, 100 * MB, MB}));
  const int had = fake().mallocs, asked = fake().asked;
  for (int q = 0; q < 4; ++q) CHECK(call(st, {4 * GB, 100 * MB, MB}));
  CHECK(fake().mallocs == had && fake().asked == asked);
  CHECK(fake().used <= fake().total / 8 + DevStore::POOL_KEEP);
  CHECK(call(st, {20 * GB, 15 * GB, 10 * GB}));   // more than an eighth: the least recently used go
  CHECK(fake().used <= fake().total / 8 + DevStore::POOL_KEEP);
  st.close(nullptr, nullptr);
  CHECK(fake().used == 0 && fake().events == 0);
}
// more blocks than the store holds places for
static void many() {
  DevStore st;
  st.open(0, fake().total);
  for (int q = 0; q < 3 * DevStore::MOST; ++q) CHECK(call(st, {(33 + 70 * (size_t)q) * MB, 40 * MB}));
  CHECK(st.n <= DevStore::MOST && fake().used <= fake().total / 8 + DevStore::POOL_KEEP);
  st.close(nullptr, nullptr);
  CHECK(fake().used == 0 && fake().events == 0);
}
// nothing stays after a call that found less than a quarter of the device free: neither the blocks of earlier calls nor the
// pool, and also when the call's own arrays are small
static void scarce() {
  for (int small = 0; small < 2; ++small) {
    DevStore st;
    st.open(0, fake().total);
    CHECK(call(st, {4 * GB, 2 * GB, 200 * MB, MB}));
    CHECK(fake().used > 6 * GB);
    fake().others = fake().total - 30 * GB;
    CHECK(call(st, {small ? 3 * MB : 9 * GB}));
    if (small) call(st, {300 * MB});   // (a size that is not held)
    CHECK(fake().used == 0);
    fake().others = 0;
    st.close(nullptr, nullptr);
  }
}
// a program whose calls are served by what is held finds out within some calls that the device has become scarce
static void scarce_later() {
  DevStore st;
  st.open(0, fake().total);
  CHECK(call(st, {4 * GB, MB}));
  fake().others = fake().total - 10 * GB;
  for (int q = 0; q < DevStore::LOOK; ++q) CHECK(call(st, {4 * GB, MB}));
  CHECK(fake().used == 0);
  fake().others = 0;
  for (int q = 0; q < 2; ++q) CHECK(call(st, {4 * GB, MB}));
  CHECK(fake().used >= 4 * GB);   // and the other way
  st.close(nullptr, nullptr);
}

// several contexts of a device: together no more than one may hold; what one has left serves an allocation of another that
// would fail, and counts when another plans; it goes with its context alone
static void contexts() {
  DevStore& st = *dev_store(3);
  int a, b, c;
  for (int q = 0; q < 3; ++q) st.open(3, fake().total);
  CHECK(call(st, {12 * GB, MB}, &a) && call(st, {9 * GB, MB}, &b) && call(st, {11 * GB, MB}, &c));
  CHECK(fake().used <= fake().total / 8 + DevStore::POOL_KEEP);
  st.close(nullptr, &c);
  CHECK(call(st, {8 * GB}, &a) && call(st, {33 * MB, MB}, &b));
  fake().others = fake().total - 60 * GB;
  CHECK(st.plan({SIZE_MAX / 2}) == 60 * GB);
  CHECK(call(st, {59 * GB}, &b));
  fake().others = 0;
  st.trim();
  CHECK(call(st, {8 * GB}, &a) && call(st, {700 * MB}, &b));
  st.close(nullptr, &a);
  CHECK(fake().used == 700 * MB);
  st.close(nullptr, &b);
  CHECK(fake().used == 0 && fake().events == 0);
}

// an array that outlives the call gets what is held unused; where that is not enough, it fails and gives no pointer
static void lasting() {
  DevStore st;
  st.open(0, fake().total);
  CHECK(call(st, {4 * GB, MB}));
  fake().others = fake().total - 5 * GB;
  char *p = nullptr, *q = p + 1;
  CHECK(dev_alloc(&st, nullptr, &p, 3 * GB) && p && fake().used == 3 * GB);
  CHECK(!dev_alloc(&st, nullptr, &q, 3 * GB) && !q && fake().used == 3 * GB);
  fake().others = 0;
  cudaFree(p);
  st.close(nullptr, nullptr);
  CHECK(fake().used == 0);
}

// batches of two arrays a tile (a chain's vectors and its projections), planned as the chain driver does: what is planned
// fits, whatever is held
static void planned() {
  for (size_t held : {6 * GB, 9 * GB, 11 * GB, 19 * GB})
    for (size_t free : {0 * GB, 1 * GB, 3 * GB}) {
      DevStore st;
      st.open(0, fake().total);
      CHECK(call(st, {held}));
      fake().others = fake().total - held - free;
      const size_t proj = GB / 2, vec = 3 * GB / 4;   // a tile's
      MemScope scope(&st, nullptr, nullptr);
      size_t tiles = 8;
      const size_t freeb = st.plan({tiles * vec, tiles * proj});
      while (tiles > 1 && tiles * (proj + vec) > freeb / 2) tiles /= 2;
      DevMem a, b;
      CHECK(a.get(tiles * vec) && b.get(tiles * proj));
      b.put();
      a.put();
      fake().others = 0;
      st.close(nullptr, nullptr);
      CHECK(fake().used == 0);
    }
}

// several arrays that together need nearly all there is: a held block of up to twice an array's size is not taken for it
static void limit() {
  DevStore st;
  st.open(0, fake().total);
  CHECK(call(st, {20 * GB}));
  fake().others = fake().total - 46 * GB;
  {
    MemScope scope(&st, nullptr, nullptr);
    st.room(44 * GB, st.plan({SIZE_MAX / 2}));
    DevMem m[4];
    for (DevMem& x : m) CHECK(x.get(11 * GB));
    for (DevMem& x : m) x.put();
  }
  fake().others = 0;
  st.close(nullptr, nullptr);
  CHECK(fake().used == 0);
}

int main(int argc, char** argv) {
  for (int k = 1; k < argc; ++k) {
    const std::string s = argv[k];
    if (s == "reuse") reuse();
    else if (s == "many") many();
    else if (s == "scarce") scarce();
    else if (s == "scarce_later") scarce_later();
    else if (s == "contexts") contexts();
    else if (s == "lasting") lasting();
    else if (s == "planned") planned();
    else if (s == "limit") limit();
    else { std::printf("no case %s\n", argv[k]); bad = 1; }
  }
  return bad;
}
