// The form of the RoPE kernel by the sizes of a call.  Resident CTAs as on a B200 (148 SMs).
#include <cstdio>
#include <initializer_list>

#include "kpx_rope_form.h"

using namespace kpx;

static int bad = 0;
static void expect(RopeForm want, int elt_bytes, int head_size, int q_heads, int kv_heads, int64_t tokens, bool norm = true, bool aligned = true) {
  const int per = 16 / elt_bytes;
  const int64_t work = tokens * ((q_heads + kv_heads) * (head_size / 2 / per) + kv_heads * head_size / per);
  const RopeCall call{elt_bytes, head_size, tokens, norm, aligned, (work + 255) / 256, elt_bytes == 2 ? 740 : 888, elt_bytes == 2 ? 444 : 592};
  const RopeForm got = rope_form(call);
  if (got == want) return;
  ++bad;
  std::printf("%d bytes, heads %d/%d of %d, %lld tokens, norm %d, aligned %d: form %d, not %d\n", elt_bytes, q_heads, kv_heads, head_size,
              static_cast<long long>(tokens), norm, aligned, int(got), int(want));
}

int main() {
  const RopeForm flat = RopeForm::kFlat, early = RopeForm::kEarlyTables, one = RopeForm::kOneToken, two = RopeForm::kTwoTokens;
  // 16-bit heads of 128: early up to what the SMs hold of that form, flat up to what they hold of the other
  for (int n : {1, 64, 160, 256}) expect(early, 2, 128, 32, 8, n);
  for (int n : {288, 320, 399}) expect(flat, 2, 128, 32, 8, n);
  for (int n : {192, 256}) expect(flat, 2, 128, 64, 8, n);
  for (int n : {288, 320, 399}) expect(early, 2, 128, 64, 8, n);
  for (int n : {1, 399}) expect(early, 2, 128, 12, 2, n);
  for (int n : {400, 1399}) expect(one, 2, 128, 12, 2, n);
  for (int n : {1400, 131072}) expect(two, 2, 128, 12, 2, n, false);
  // heads of 64: two rounds more than the flat form are too many
  for (int n : {600, 800, 1600}) expect(flat, 2, 64, 32, 8, n);
  for (int n : {1, 400, 1200, 2048}) expect(early, 2, 64, 32, 8, n);
  // fp32: never the form of a CTA per token
  for (int n : {1, 64, 160, 288, 399, 800}) expect(early, 4, 128, 32, 8, n);
  for (int n : {192, 224, 256, 20000}) expect(flat, 4, 128, 32, 8, n);
  // heads of 256: early whatever the size
  for (int n : {1, 200, 399, 900, 8000}) expect(early, 2, 256, 28, 4, n);
  expect(early, 4, 256, 12, 2, 399);
  // no norm, or tables off 16-byte boundaries
  for (int n : {1, 256, 399}) expect(flat, 2, 128, 32, 8, n, false), expect(flat, 2, 128, 32, 8, n, true, false), expect(flat, 4, 128, 32, 8, n, false);
  return bad != 0;
}
