"""The binding through which tensors reach the kernels' C entry points (csrc/binding/calls.cpp), on functions compiled here."""
import ctypes
import subprocess
import threading

import pytest
import torch

import llm_infer_rust_b200.kernels.build as build

_SOURCE = r"""
#include <cstdint>
#include <cstdio>
// pointers, ints, 64-bit ints and floats in every order that a signature may have them; from the seventh on integers lie on the stack
extern "C" int sum3(const float* a, float x, int n) { return static_cast<int>(a[0] + x) + n; }
extern "C" int eight(float a, int i, float b, float c, long long l, float d, float e, float f, float g, float h, char* out) {
  return std::snprintf(out, 200, "%g %g %g %g %g %g %g %g %d %lld", a, b, c, d, e, f, g, h, i, l);
}
extern "C" int many(int a, const void* b, float x, long long c, int d, int e, int f, int g, int h, float y, int i, int j, int k, int l,
                    int m, int n, int o, long long p, void* q, int r, float z, int s, char* out) {
  return std::snprintf(out, 400, "%d %d %g %lld %d %d %d %d %d %g %d %d %d %d %d %d %d %lld %d %d %g %d", a, b != nullptr, x, c, d, e, f,
                       g, h, y, i, j, k, l, m, n, o, p, q != nullptr, r, z, s);
}
extern "C" int negative(int a, long long b) { return a == -3 && b == -(1ll << 40) ? -2 : 1; }
"""


@pytest.fixture(scope="module")
def entries(tmp_path_factory):
    folder = tmp_path_factory.mktemp("entries")
    source, library = folder / "entries.cpp", folder / "entries.so"
    source.write_text(_SOURCE)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", str(source), "-o", str(library)], check=True)
    return build.EntryPoints(ctypes.CDLL(str(library)))


def test_every_kind_of_argument_arrives(entries):
    assert entries.sum3(torch.tensor([4.0, 9.0]), 2.5, 7) == 13
    out = ctypes.create_string_buffer(400)
    assert entries.eight(0.5, -7, 1.5, 2.5, 1 << 40, 3.5, 4.5, 5.5, 6.5, 7.5, out) > 0
    assert out.value == b"0.5 1.5 2.5 3.5 4.5 5.5 6.5 7.5 -7 1099511627776"
    args = [1, None, 0.25, -(1 << 33), 4, 5, 6, 7, 8, 1e-3, 9, 10, 11, 12, 13, -14, 15, 1 << 50, torch.zeros(1), True, -2.0, 17, out]
    assert entries.many(*args) > 0
    assert out.value == b"1 0 0.25 -8589934592 4 5 6 7 8 0.001 9 10 11 12 13 -14 15 1125899906842624 1 1 -2 17"
    assert entries.negative(-3, -(1 << 40)) == -2


def test_what_is_no_argument_is_refused(entries):
    for bad in ("text", b"bytes", ctypes.c_void_p(8), ctypes.c_float(1.0), [1], object()):
        with pytest.raises(TypeError):
            entries.sum3(torch.zeros(1), bad, 1)
    with pytest.raises(TypeError):
        entries.sum3(*range(49))
    with pytest.raises(TypeError):
        entries.sum3(*[1.0] * 9)
    with pytest.raises(TypeError):
        entries.sum3(torch.zeros(1), 1.0, n=1)
    with pytest.raises(OverflowError):
        entries.sum3(1 << 70, 1.0, 1)
    with pytest.raises(AttributeError):
        entries.no_such_function


def test_checks_and_outputs():
    calls = build.load_call_binding()
    a = torch.zeros(3, 4)
    assert not calls.all_cuda(a) and calls.all_cuda(None) and calls.all_cuda()
    assert calls.all_contiguous(a, None, a[1:]) and not calls.all_contiguous(a, a.t())
    with pytest.raises(TypeError):
        calls.all_cuda(None, 3)
    for shape in ((5, 7), torch.Size([0, 3]), (4,), ()):
        got = calls.empty(shape, torch.bfloat16, a.device)
        assert got.shape == torch.Size(shape) and got.dtype == torch.bfloat16 and got.device == a.device and got.is_contiguous()
    with pytest.raises(RuntimeError):
        calls.empty((-1, 2), torch.float32, a.device)
    x, w = torch.randn(3, 8), torch.randn(5, 8)
    assert torch.equal(calls.mm_t(x, w), torch.mm(x, w.t()))
    with pytest.raises(RuntimeError):
        calls.mm_t(x, torch.randn(5, 9))


def test_several_threads(entries):
    got = []

    def work(i):
        out = ctypes.create_string_buffer(400)
        for _ in range(200):
            entries.eight(float(i), i, 1.5, 2.5, i, 3.5, 4.5, 5.5, 6.5, 7.5, out)
            got.append(out.value == f"{i} 1.5 2.5 3.5 4.5 5.5 6.5 7.5 {i} {i}".encode())
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 800 and all(got)


_ADD = r"""
extern "C" int add(float* out, const float* a, const float* b, float scale, int n) {
  for (int i = 0; i < n; ++i) out[i] = a[i] + scale * b[i];
  return n > 100 || out[0] > 1e30f ? -2 : 0;
}
"""


@pytest.fixture(scope="module")
def adding(tmp_path_factory):
    folder = tmp_path_factory.mktemp("adding")
    (folder / "add.cpp").write_text(_ADD)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", str(folder / "add.cpp"), "-o", str(folder / "add.so")], check=True)
    return build.EntryPoints(ctypes.CDLL(str(folder / "add.so")))


def _layer(adding, calls, h, w, b, scale=2.0):
    """h <- h + scale b in place; the product with w^T, to which an inner buffer adds b again."""
    n = h.numel()
    assert adding.add(h, h, b, scale, n) == 0
    inner = torch.empty_like(h)
    assert adding.add(inner, h, b, 1.0, n) == 0
    return calls.mm_t(inner, w)


def test_a_layers_calls_are_made_again_with_anothers_weights(adding):
    calls = build.load_call_binding()
    ws, bs = [torch.randn(4, 4) for _ in range(5)], [torch.randn(3, 4) for _ in range(5)]
    want = start = torch.randn(3, 4)
    for w, b in zip(ws, bs):
        want = _layer(adding, calls, want.clone(), w, b)
    h = start.clone()
    calls.record()
    out = _layer(adding, calls, h, ws[0], bs[0])
    kept = calls.finish((h, out, ws[0], bs[0]))
    spare = h
    for w, b in zip(ws[1:], bs[1:]):
        assert calls.replay(kept, (out, spare, w, b)) == 0
        out, spare = spare, out
    assert torch.equal(out, want)


def test_values_that_are_not_like_their_slots_are_left_to_the_caller(adding):
    calls = build.load_call_binding()
    h, w, b = torch.randn(3, 4), torch.randn(4, 4), torch.randn(3, 4)
    calls.record()
    with pytest.raises(RuntimeError):
        calls.record()                                          # one at a time
    out = _layer(adding, calls, h, w, b)
    kept = calls.finish((h, out, w, b))
    odd = torch.randn(17)[1:].reshape(4, 4)                     # not on the boundary that w was on
    before = h.clone()
    for bad in ((h, out, w), (h, out, w.double(), b), (h, out, torch.randn(4, 5), b), (h, out, w.t(), b), (h, out, odd, b),
                (h, out, ctypes.create_string_buffer(64), b)):
        assert calls.replay(kept, bad) is None and torch.equal(h, before)
    with pytest.raises(TypeError):
        calls.replay(kept, (h, out, w, 3))
    with pytest.raises(RuntimeError):
        calls.finish((h,))                                      # nothing is recorded
    calls.record()
    calls.discard()
    calls.record()
    big = torch.zeros(128)
    assert adding.add(big, big, big, 1.0, 100) == 0
    kept = calls.finish((big,))
    assert calls.replay(kept, (torch.zeros(128),)) == 0
    assert calls.replay(kept, (torch.full((128,), 1e30),)) == -2     # an entry point's code comes back
    calls.record()
    assert adding.add(big, big, big, 1.0, 101) == -2            # as an answer that is no code: asked once, not made again
    other = torch.ones(128)
    assert calls.replay(calls.finish((big,)), (other,)) == 0 and torch.equal(other, torch.ones(128))
    calls.record()
    adding.add(big, big, big, 1.0, 100)
    kept = calls.finish((big, big))                             # which of the two an argument leads to is not known
    assert calls.replay(kept, (torch.zeros(128), torch.zeros(128))) is None


class _Block(ctypes.Structure):
    _fields_ = [("address", ctypes.c_void_p)]


@pytest.mark.parametrize("way", ["start", "inside", "address", "address inside", "block", "array", "product of a part", "product behind it"])
def test_a_slots_memory_reached_by_other_ways(adding, way):
    """Whatever leads into a slot's memory other than by its start is not exchanged, so such a layer is left to Python."""
    calls = build.load_call_binding()
    h, b, w = torch.zeros(4, 4), torch.arange(16.0).view(4, 4), torch.randn(4, 4)
    block = _Block(b.data_ptr())
    array = (ctypes.c_float * 16)()
    reach = {"start": b, "inside": b[1:], "address": b.data_ptr(), "address inside": b.data_ptr() + 16, "block": block, "array": array}
    calls.record()
    if way in reach:
        assert adding.add(h, h, reach[way], 0.0 if way == "block" else 1.0, 1) == 0
    else:
        calls.mm_t(b[:2] if way == "product of a part" else b[1:], w)
    kept = calls.finish((h, b, w))
    assert calls.replay(kept, (torch.zeros(4, 4), b.clone(), w)) == (0 if way == "start" else None)


def test_recordings_are_a_threads_own(adding):
    calls = build.load_call_binding()
    h, b = torch.zeros(3, 4), torch.ones(3, 4)
    calls.record()
    other = threading.Thread(target=lambda: adding.add(torch.zeros(3, 4), b, b, 1.0, 12))
    other.start()
    other.join()
    adding.add(h, h, b, 1.0, 12)
    kept = calls.finish((h, b))
    assert calls.replay(kept, (h, b)) == 0 and torch.equal(h, 2 * b)
