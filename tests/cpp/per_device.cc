// PerDevice: found once per device, never from another one's value, errors not kept.
#include <cstdio>
#include "per_device.h"

int main() {
  aslb::PerDevice kept;
  int calls = 0, n = 0;
  auto find = [&](int value, int error) {
    return [&calls, value, error](int& out) {
      ++calls;
      out = value;
      return error;
    };
  };
  bool ok = kept.get(0, n, find(3, 7)) == 7 && calls == 1;        // an error
  ok = ok && kept.get(0, n, find(3, 0)) == 0 && n == 3 && calls == 2;
  ok = ok && kept.get(0, n, find(9, 0)) == 0 && n == 3 && calls == 2;
  ok = ok && kept.get(1, n, find(5, 0)) == 0 && n == 5 && calls == 3;  // another device
  ok = ok && kept.get(0, n, find(9, 0)) == 0 && n == 3 && calls == 3;
  ok = ok && kept.get(64, n, find(6, 0)) == 0 && n == 6 && calls == 4;  // beyond what is kept
  ok = ok && kept.get(64, n, find(8, 0)) == 0 && n == 8 && calls == 5;
  std::printf(ok ? "ok\n" : "wrong\n");
  return ok ? 0 : 1;
}
