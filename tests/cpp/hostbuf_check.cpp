// The server's reuse of host buffers (qcb_hostbuf.h): which buffer a request gets and when, and what is kept.
#include <stdio.h>

#include "qcb_hostbuf.h"

using namespace qcb;

static int bad = 0;
static void expect(bool ok, const char* what) {
    if (ok) return;
    printf("%s\n", what);
    bad++;
}

// a buffer above the limit is freed; those that wait stay
static void above_the_limit() {
    HostBufs<int> h(1000);
    const HostBuf a = h.take(300), b = h.take(400), big = h.take(1500);
    h.give(a);
    h.give(b);
    h.give(big);
    const HostBuf c = h.take(290), d = h.take(390);  // a new buffer would have the size asked for
    expect(c.cap == 300 && d.cap == 400, "a buffer above the limit drops the waiting ones");
    h.give(c);
    h.give(d);
}

// at the limit the oldest leave
static void at_the_limit() {
    HostBufs<int> h(1000);
    const HostBuf a = h.take(300), b = h.take(400), c = h.take(600);
    h.give(a);
    h.give(b);
    h.give(c);  // 1300: a leaves
    const HostBuf x = h.take(590), y = h.take(390);
    expect(x.cap == 600 && y.cap == 400, "the newer buffers stay");
    const HostBuf z = h.take(290);
    expect(z.cap == 290, "a new buffer where the old one left");
    h.give(x);
    h.give(y);
    h.give(z);
}

// the smallest that is large enough, but none of more than four times the size
static void choice() {
    HostBufs<int> h(1 << 20);
    const HostBuf a = h.take(100), b = h.take(200), c = h.take(4000);
    h.give(c);
    h.give(b);
    h.give(a);
    const HostBuf x = h.take(90), y = h.take(150), z = h.take(900);
    expect(x.cap == 100 && y.cap == 200, "the smallest that is large enough");
    expect(z.cap == 900, "not one of more than four times the size");
    h.give(x);
    h.give(y);
    h.give(z);
}

// a buffer whose copy has not ended is not handed out
static void copies() {
    HostBufs<int> h(1000);
    const HostBuf a = h.take(300), b = h.take(300);
    expect(h.give_after(a, 1) && h.give_after(b, 2), "noted");
    int released = 0;
    auto release = [&](int e) { released |= e; };
    h.reclaim([](int) { return false; }, release);
    const HostBuf x = h.take(290);
    expect(x.cap == 290 && released == 0, "a buffer handed out while a copy reads it");
    h.reclaim([](int e) { return e == 2; }, release);
    const HostBuf y = h.take(290);
    expect(y.p == b.p && released == 2, "the buffer whose copy has ended, and its event alone");
    h.reclaim([](int) { return true; }, release);
    const HostBuf z = h.take(290);
    expect(z.p == a.p && released == 3, "the other one after its copy");
    h.give(x);
    h.give(y);
    h.give(z);
    expect(h.give_after(h.take(50), 4), "noted");  // a copy not reclaimed: freed with the class
}

int main() {
    copies();
    above_the_limit();
    at_the_limit();
    choice();
    return bad != 0;
}
