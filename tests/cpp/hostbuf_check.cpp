// The server's reuse of host buffers (qcb_hostbuf.h): which buffer a request gets, and what is kept.
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
    HostBufs h(1000);
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
    HostBufs h(1000);
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
    HostBufs h(1 << 20);
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

int main() {
    above_the_limit();
    at_the_limit();
    choice();
    return bad != 0;
}
