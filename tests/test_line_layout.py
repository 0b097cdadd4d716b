"""The shared-memory layout of a pass' lines (PassShape LS and line_off, restated): lines never overlap and,
for lines of fewer threads than a bank cycle has slots, the exchanges' and the staging copy's accesses of
one bank cycle fall on distinct slots."""
import pytest


def layout(L, slots, G):
    E = min(L, 16)
    T = L // E
    raw = L + L // E + (T - 1 if T < slots else 0)
    target = T if T < slots else (1 if G >= slots else slots // G)
    stride = raw + (target - raw) % slots
    return E, T, stride, lambda w: w * stride + (w // (slots // T) % T if T < slots else 0)


@pytest.mark.parametrize("slots", [8, 16])  # 16-byte and 8-byte values
@pytest.mark.parametrize("L", [2 ** k for k in range(1, 13)])
def test_lines_and_bank_slots(slots, L):
    T0 = L // min(L, 16)
    g0 = 1 if T0 >= 128 else 128 // T0
    for G in sorted({g0, max(1, g0 // 2), 2 * g0, 7}):
        E, T, stride, off = layout(L, slots, G)
        for w in range(G):
            assert off(w) + L + L // E <= (off(w + 1) if w + 1 < G else G * stride)
        if T >= slots or G < slots:
            continue
        q = slots // T  # lines of one bank cycle
        for w0 in range(0, G - q + 1, q):
            for r in range(E):
                hit = {(off(w0 + k) + (E * t + r) + (E * t + r) // E) % slots for k in range(q) for t in range(T)}
                assert len(hit) == slots
        for w0 in range(0, G - slots + 1, slots):
            assert len({off(w0 + k) % slots for k in range(slots)}) == slots
