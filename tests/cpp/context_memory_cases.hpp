// Frames of growing sizes, as a render asks for its scratch: fixed small blocks
// (counters, a table), blocks that grow with the pixels, and blocks that only
// some frames ask for.
using Plan = std::vector<ScratchNeed>;

static Plan frame(size_t npix, bool aov) {
  Plan p;
  for (int slot : {16, 18, 23, 24, 27, 28}) p.push_back({slot, 16 * npix});
  for (int slot : {17, 19, 20, 21, 22, 25, 26}) p.push_back({slot, 4 * npix});
  if (aov)
    for (int slot : {70, 71, 72}) p.push_back({slot, 16 * npix});
  return p;
}

static void render(Context& c, const Plan& plan) {
  ++c.call;
  scratchReserve(&c, plan);
  void* p;
  for (int slot : {33, 34, 37, 32}) check(scratchGet(&c, slot, 64 + 16, &p) == UBR_OK, "a counter");
  for (const ScratchNeed& n : plan) check(scratchGet(&c, n.slot, n.bytes, &p, n.slack) == UBR_OK, "a plane");
  consistent(c);
}

static void slabs() {
  const size_t mib = size_t(1) << 20;
  // a first frame in one allocation, then larger ones: the first one's memory
  // goes back, whatever small blocks were taken with it
  Context& c = fresh(0);
  render(c, frame(700000, true));
  check(c.slab.ptr != nullptr, "the first frame's scratch is one allocation");
  const size_t first = fake::held;
  check(first < blocks(c) + 8 * mib, "little beyond the blocks is held");
  render(c, frame(700000, true));
  check(fake::held == first, "the same frame again takes nothing");
  render(c, frame(1400000, true));
  check(fake::held < blocks(c) + 8 * mib, "the first allocation went back");
  render(c, frame(2400000, false));
  check(fake::held < blocks(c) + 8 * mib, "it goes back with blocks the new frame does not ask for");
  render(c, frame(20000000, false));  // more than one allocation of this kind holds
  check(fake::held < blocks(c) + 8 * mib, "and where the new frame takes its blocks one by one");
  render(c, frame(700000, true));
  check(fake::held < blocks(c) + 8 * mib, "a small frame after it");
  // blocks that are large enough already are not allocated for again
  Context& d = fresh(0);
  render(d, frame(600000, false));
  void* p;
  ++d.call;
  for (int slot : {70, 71, 72}) check(scratchGet(&d, slot, 64 * mib, &p) == UBR_OK, "a block on its own");
  const size_t before = fake::held;
  render(d, frame(1000000, true));
  check(fake::held < before + size_t(1.3 * 124 * 1000000) + 8 * mib - size_t(1.2 * 124 * 600000), "only what grows");
  // a block that outgrows the allocation leaves room that others take
  Context& g = fresh(0);
  render(g, frame(800000, true));
  check(scratchGet(&g, 16, 40 * mib, &p) == UBR_OK, "a block that grows on its own");
  consistent(g);
  const size_t grown = fake::held;
  check(scratchGet(&g, 30, 12 * mib, &p) == UBR_OK, "a new block");
  consistent(g);
  check(fake::held == grown, "in the room that was left");
  // an allocation that nothing was cut from
  Context& h = fresh(0);
  ++h.call;
  scratchReserve(&h, frame(800000, false));
  render(h, frame(900000, false));
  check(fake::held < blocks(h) + 8 * mib, "goes back at the next one");
  // no allocation for all: the blocks one by one
  Context& i = fresh(0);
  fake::limit = 100 * mib;
  render(i, frame(500000, false));
  // random sizes
  Context& e = fresh(0);
  unsigned x = 1;
  for (int k = 0; k < 300; ++k) {
    x = x * 1664525u + 1013904223u;
    render(e, frame(1000 + (x >> 8) % 3000000, (x >> 5) & 1));
    check(fake::held < blocks(e) + 8 * mib, "little beyond the blocks is held");
  }
}

static void workspaces() {
  const size_t kib = 1024, mib = 1024 * kib;
  void* p;
  size_t n;
  // under a cap that leaves room: all that is wanted, counted
  Context& c = fresh(1024 * mib);
  ++c.call;
  n = 300 * mib;
  check(workspaceGet(&c, kGatherSlot, 10 * kib, nullptr, 0, &p, &n) == UBR_OK && n == 300 * mib, "all it wants");
  check(p == c.scratch[kGatherSlot].ptr && c.arenaUsed == 300 * mib, "of its own, counted");
  scratchDone(&c, kGatherSlot);
  consistent(c);
  // ... and it does not stand in the way of what comes later, in this call or the next
  check(scratchGet(&c, 16, 640 * mib, &p) == UBR_OK, "a block of the same call");
  check(c.scratch[kGatherSlot].ptr == nullptr, "the workspace made room");
  ++c.call;
  n = 400 * mib;
  check(workspaceGet(&c, kAdjointSlot, 10 * kib, nullptr, 0, &p, &n) == UBR_OK && n == 400 * mib, "lent");
  check(p == c.scratch[16].ptr, "the block of the call before");
  n = 2000 * mib;
  check(workspaceGet(&c, kAdjointSlot, 10 * kib, nullptr, 0, &p, &n) == UBR_OK && n == 800 * mib, "lent whole");
  check(scratchGet(&c, 20, 700 * mib, &p) == UBR_OK, "scratch of an earlier call makes room");
  check(c.scratch[16].ptr == nullptr, "it went");
  check(scratchGet(&c, 21, 200 * mib, &p) == UBR_OUT_OF_MEMORY, "this call's own does not");
  check(c.scratch[20].ptr != nullptr, "and stays");
  consistent(c);
  // what a cap leaves, where that is more than what is lent
  Context& d = fresh(64 * mib);
  ++d.call;
  check(scratchGet(&d, 23, 16 * mib, &p) == UBR_OK, "a plane");
  void* const plane = p;
  n = 100 * mib;
  check(workspaceGet(&d, kGatherSlot, 10 * kib, plane, 16 * mib, &p, &n) == UBR_OK && n == 44 * mib, "what is left");
  check(d.arenaUsed == 64 * mib, "the cap in full");
  n = 100 * mib;
  const int before = fake::calls;
  check(workspaceGet(&d, kGatherSlot, 10 * kib, plane, 16 * mib, &p, &n) == UBR_OK && n == 44 * mib, "kept");
  check(fake::calls == before, "not taken again");
  check(scratchGet(&d, 24, 40 * mib, &p) == UBR_OUT_OF_MEMORY, "a workspace in use stays");
  scratchDone(&d, kGatherSlot);
  check(scratchGet(&d, 24, 44 * mib, &p) == UBR_OK && d.scratch[24].bytes == 44 * mib,
        "and goes when its work is queued; no slack where the cap has no room for it");
  n = 100 * mib;
  check(workspaceGet(&d, kGatherSlot, 10 * kib, plane, 16 * mib, &p, &n) == UBR_OK && p == plane && n == 16 * mib,
        "what is lent where the cap leaves less");
  // without a cap: its own, and what is lent where the device refuses
  Context& e = fresh(0);
  ++e.call;
  n = 100 * mib;
  check(workspaceGet(&e, kGatherSlot, 10 * kib, plane, 16 * mib, &p, &n) == UBR_OK && p != plane && n == 100 * mib,
        "its own");
  fake::limit = 120 * mib;
  n = 200 * mib;
  check(workspaceGet(&e, kGatherSlot, 10 * kib, plane, 16 * mib, &p, &n) == UBR_OK && p == plane && n == 16 * mib,
        "lent where the device has no more");
  consistent(e);
}

static void hardCap() {
  const size_t kib = 1024, mib = 1024 * kib;
  void* p;
  size_t n;
  // a cap that leaves less than the least workspace, and nothing to lend
  Context& c = fresh(1 * mib);
  ++c.call;
  check(scratchGet(&c, 16, 1 * mib - 4 * kib, &p) == UBR_OK, "nearly all of it");
  n = 10 * mib;
  check(workspaceGet(&c, kAdjointSlot, 5 * kib, nullptr, 0, &p, &n) == UBR_OUT_OF_MEMORY, "refused");
  check(fake::peak <= c.arenaCap, "and the cap holds");
  n = 10 * mib;
  check(workspaceGet(&c, kAdjointSlot, 4 * kib, nullptr, 0, &p, &n) == UBR_OK && n == 4 * kib, "what is left");
  check(fake::held == c.arenaCap && c.arenaUsed == c.arenaCap, "all counted");
  consistent(c);
  // random calls: blocks and workspaces, refused or not, stay within the cap
  unsigned x = 7;
  auto draw = [&](size_t most) {
    x = x * 1664525u + 1013904223u;
    return 1 + size_t(x >> 8) % most;
  };
  for (int round = 0; round < 20; ++round) {
    Context& d = fresh(draw(2 * mib));
    for (int k = 0; k < 100; ++k) {
      ++d.call;
      for (int b = int(draw(4)); b > 0; --b) {
        n = draw(300 * kib);
        scratchGet(&d, int(draw(12)), n, &p);
      }
      const size_t least = draw(20 * kib), lent = draw(2) == 1 ? draw(40 * kib) : 0;
      char frame[1];
      n = least + draw(600 * kib);
      const ubr_status st = workspaceGet(&d, kGatherSlot, least, lent ? frame : nullptr, lent, &p, &n);
      check(st != UBR_OK || n >= least, "at least what it asks for");
      check(st == UBR_OK || lent < least, "what is lent serves");
      if (draw(2) == 1) scratchDone(&d, kGatherSlot);
      check(fake::peak <= d.arenaCap, "the cap is hard");
      consistent(d);
    }
  }
}

static void cases() {
  slabs();
  workspaces();
  hardCap();
}
