"""The C-ABI library loads without a GPU and exports every symbol the headers under include/ declare;
argument validation and launch planning run on the host."""
import ctypes
import os
import re

import pytest

from mamba2d_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def L():
    from mamba2d_b200 import build
    build.build()
    return _lib.lib()


def declared_symbols():
    inc = os.path.join(ROOT, "include")
    text = "".join(open(os.path.join(inc, f)).read() for f in sorted(os.listdir(inc)) if f.endswith(".h"))
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(m2d_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(L):
    syms = declared_symbols()
    assert set(_lib.EXPORTS) <= set(syms)
    raw = ctypes.CDLL(_lib.LIB_PATH)
    for s in syms:
        assert getattr(raw, s) is not None, s


def test_version_and_strerror(L):
    assert L.m2d_abi_version() == _lib.ABI_VERSION
    assert _lib.strerror(0) == "ok"
    for code in range(-10, 0):
        assert _lib.strerror(code) not in ("ok", "unknown status")
    assert _lib.strerror(-99) == "unknown status"


def _desc(**kw):
    d = _lib.ScanDesc()
    d.struct_bytes = ctypes.sizeof(_lib.ScanDesc)
    d.dtype = _lib.M2D_F32
    d.B, d.H, d.W, d.E, d.N = 2, 8, 8, 64, 16
    d.BT_pitch = d.BL_pitch = d.C_pitch = 16
    for k, v in kw.items():
        setattr(d, k, v)
    return d


def test_descriptor_validation_without_a_device(L):
    d = _desc()
    assert L.m2d_scan_fwd(ctypes.byref(d), None) == -1          # NULL pointers
    assert L.m2d_scan_fwd(ctypes.byref(_desc(H=1)), None) == -3  # H < 2, as the reference's ValueError
    assert L.m2d_scan_fwd(ctypes.byref(_desc(W=1)), None) == -3
    assert L.m2d_scan_bwd(ctypes.byref(_desc(N=32)), None) == -4
    assert L.m2d_scan_fwd(ctypes.byref(_desc(dtype=7)), None) == -2
    assert L.m2d_scan_fwd(ctypes.byref(_desc(C_pitch=8)), None) == -5
    assert L.m2d_scan_fwd(ctypes.byref(_desc(struct_bytes=8)), None) == -8
    assert L.m2d_scan_fwd(ctypes.byref(_desc(flags=8)), None) == -10   # unknown flag bit
    assert L.m2d_scan_bwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_A_LOG)), None) == -1     # known to both entries
    assert L.m2d_scan_fwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_GELU_OUT)), None) == -1   # forward-only bit: next check
    assert L.m2d_scan_bwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_GELU_OUT)), None) == -10  # ... the backward refuses it
    assert L.m2d_scan_bwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_REVERSE)), None) == -1   # known bit: next check
    assert L.m2d_scan_fwd(None, None) == -1


def test_workspace_queries(L):
    # one band (no more rows than a CTA has row-warps): the forward needs the status word only
    assert L.m2d_scan_fwd_workspace(ctypes.byref(_desc(H=4))) == 256
    # several bands: a per-CTA ring of W slots of 2 KiB
    d = _desc(B=128, H=56, W=56)
    ws = L.m2d_scan_fwd_workspace(ctypes.byref(d))
    assert ws > 256 and ws % 256 == 0 and ws <= 256 + 128 * 2 * 56 * 2048
    # backward: state record B*groups*H*W*2 KiB plus accumulators
    wb = L.m2d_scan_bwd_workspace(ctypes.byref(d))
    assert wb >= 128 * 2 * 56 * 56 * 2048
    assert L.m2d_scan_fwd_workspace(ctypes.byref(_desc(H=1))) == 0    # invalid descriptor


@pytest.mark.parametrize("B,H,W,E", [(2, 200, 336, 64), (6, 45, 31, 192), (1, 1024, 1024, 64), (4, 14, 14, 384), (1, 9, 2, 40), (400, 9, 2, 16)])
@pytest.mark.parametrize("dtype", [_lib.M2D_F32, _lib.M2D_BF16])
def test_scratch_of_few_images_is_bounded(L, B, H, W, E, dtype):
    """Bytes per element as include/m2d_scan.h states them: rows in bands of eight, channels in groups of 16 or 32."""
    d = ctypes.byref(_desc(B=B, H=H, W=W, E=E, dtype=dtype))
    rows, bands, chans = (H + 7) // 8 * 8, (H + 7) // 8, (E + 31) // 32 * 32
    boundary = B * bands * W * chans * 16 * 4                 # a row of 16 states per band
    record = B * rows * (W + 7) * chans * 16 * 4              # every state of every step, fp32
    sums = 0 if dtype == _lib.M2D_F32 else 4 * (3 * B * H * W * 16 + 2 * E * 16 + E)
    slack = 8 * 256
    assert L.m2d_scan_fwd_workspace(d) <= boundary + slack
    assert L.m2d_scan_bwd_workspace(d) <= record + 2 * boundary + sums + slack


@pytest.mark.parametrize("B,H,W,E,N", [(564, 3, 2984, 392, 16), (427, 8, 1611, 74, 16), (43, 3, 2615, 879, 5), (18, 6, 593, 892, 5), (72, 33, 327, 351, 16)])
def test_rings_stay_small_where_some_plan_has_small_ones(L, B, H, W, E, N):
    """A launch of many short bands is not bought with gigabytes of boundary rows; the backward's are beside the record."""
    d = _desc(B=B, H=H, W=W, E=E, N=N, BT_pitch=N, BL_pitch=N, C_pitch=N)
    rings = 96 << 20
    assert L.m2d_scan_fwd_workspace(ctypes.byref(d)) <= 256 + rings
    assert L.m2d_scan_bwd_workspace(ctypes.byref(d)) <= 256 + rings + B * H * W * ((E + 15) // 16) * 1024


@pytest.mark.parametrize("B,H,W,E,dtype,limit", [(316, 7, 9400, 71, _lib.M2D_F32, 12e9), (226, 7, 5000, 100, _lib.M2D_BF16, 8e9),
                                                 (40, 900, 900, 64, _lib.M2D_BF16, 91e9), (40, 700, 700, 64, _lib.M2D_F32, 51e9)])
def test_large_calls_take_the_plan_of_less_scratch(L, B, H, W, E, dtype, limit):
    """The wave kernels' lists of images need a record each; one of all images would take 106, 58, 172 and 100 GB."""
    d = ctypes.byref(_desc(B=B, H=H, W=W, E=E, dtype=dtype))
    assert L.m2d_scan_bwd_workspace(d) <= limit and L.m2d_scan_bwd_chain(d) == 1


@pytest.mark.parametrize("B,H,W,E,chained,wide", [
    (128, 28, 28, 128, False, False), (40, 56, 56, 64, True, True), (8, 69, 49, 320, True, True), (8, 82, 84, 384, True, True),
    (12, 20, 20, 128, False, True), (4, 70, 64, 320, True, True), (10, 62, 63, 128, True, True)])
def test_type_of_the_state_record(L, B, H, W, E, chained, wide):
    """bf16 I/O: a large batch keeps its states in bf16 (32 bytes per element), few images and the calls with several CTAs per image in
    fp32 (64), as fp32 I/O always does.  Beside it at most a boundary row per band of eight for each sweep."""
    record = B * H * W * ((E + 15) // 16) * 16 * 16 * 4
    rows = 2 * B * ((H + 7) // 8) * W * ((E + 15) // 16) * 16 * 16 * 4 + 2 * 256
    for dtype, sums, size in ((_lib.M2D_F32, 0, record), (_lib.M2D_BF16, 4 * (3 * B * H * W * 16 + 2 * E * 16 + E) + 256, record if wide else record // 2)):
        d = _desc(B=B, H=H, W=W, E=E, dtype=dtype)
        assert (L.m2d_scan_bwd_chain(ctypes.byref(d)) > 1) == chained
        assert size + sums - 256 <= L.m2d_scan_bwd_workspace(ctypes.byref(d)) <= size + sums + rows + 512


def test_plans_do_not_depend_on_the_environment(L, monkeypatch):
    """The workspace query and the launch plan separately; nothing a program can change in between may tell them apart."""
    d = ctypes.byref(_desc(B=128, H=56, W=56))
    before = L.m2d_scan_bwd_workspace(d), L.m2d_scan_fwd_workspace(d)
    for v in "1235":
        monkeypatch.setenv("M2D_BWD_WARPS", v)
        assert (L.m2d_scan_bwd_workspace(d), L.m2d_scan_fwd_workspace(d)) == before


def test_a_kept_plan_is_used_for_its_own_sizes_only(L, monkeypatch):
    """A thread keeps its last plan of each kind.  Descriptors that differ in one size, asked for in turn, from two threads and under
    other environments, get what a thread that has kept nothing gets."""
    import threading
    base = dict(B=24, H=57, W=50, E=64, N=16, dtype=_lib.M2D_BF16)
    others = [dict(base, **c) for c in ({}, {"B": 25}, {"H": 58}, {"W": 51}, {"E": 80}, {"N": 12}, {"dtype": _lib.M2D_F32})]

    def ask(c):
        d = ctypes.byref(_desc(**c))
        return (L.m2d_scan_fwd_workspace(d), L.m2d_scan_bwd_workspace(d), L.m2d_scan_fwd_chain(d), L.m2d_scan_bwd_chain(d),
                L.m2d_scan_fwd_cleared(d), L.m2d_scan_fwd_noalloc_need(d))

    def in_a_thread(f):
        out = []
        t = threading.Thread(target=lambda: out.append(f()))
        t.start()
        t.join()
        return out[0]
    want = [in_a_thread(lambda c=c: ask(c)) for c in others]
    assert len(set(want)) == len(others)
    for v in "1235":
        monkeypatch.setenv("M2D_BWD_WARPS", v)
        for i in range(len(others)):
            for k in (0, i, 0, i, i):
                assert ask(others[k]) == want[k]
    # two threads in step, each with sizes of its own
    gate, got = threading.Barrier(2), {}

    def turns(k):
        got[k] = []
        for _ in range(20):
            gate.wait(20)
            got[k].append(ask(others[k]))
    both = [threading.Thread(target=turns, args=(k,)) for k in (1, 2)]
    for t in both:
        t.start()
    for t in both:
        t.join()
    assert got == {k: [want[k]] * 20 for k in (1, 2)}


def test_status_word_and_chain_queries(L):
    d = _desc(B=128, H=56, W=56)
    assert L.m2d_scan_fwd_status_offset(ctypes.byref(d)) == 0
    assert L.m2d_scan_bwd_status_offset(ctypes.byref(d)) == 0
    assert L.m2d_scan_fwd_chain(ctypes.byref(d)) == 1 and L.m2d_scan_bwd_chain(ctypes.byref(d)) == 1   # enough images: one CTA each
    d = _desc(B=1, H=256, W=256)
    assert L.m2d_scan_fwd_chain(ctypes.byref(d)) > 1 and L.m2d_scan_bwd_chain(ctypes.byref(d)) > 1
    assert L.m2d_scan_fwd_status_offset(ctypes.byref(_desc(H=1))) == -1 and L.m2d_scan_fwd_chain(ctypes.byref(_desc(H=1))) == 0
    # more bands than resident CTAs: the chain stays shorter than one row of steps (W / 8 - 1)
    d = _desc(B=1, H=2400, W=24, E=32)
    assert L.m2d_scan_fwd_chain(ctypes.byref(d)) == 24 // 8 - 1
    d = _desc(B=1, H=2400, W=200, E=32)
    assert L.m2d_scan_fwd_chain(ctypes.byref(d)) == 200 // 8 - 1


def test_chain_bound_over_shrink_sequences(L):
    """A planned chain and every chain a launch may fall back to obey the same rule: never more CTAs
    than bands, and a chain shorter than that stays below one row of steps per band height."""
    for nbands in (1, 2, 7, 10, 128, 300):
        for steps in (2, 3, 12, 24, 56, 1024):
            for rb in (1, 2, 6, 8):
                if rb > steps:
                    continue
                want = 296
                for _ in range(40):
                    c = L.m2d_scan_chain_bound(want, nbands, steps, rb)
                    assert 1 <= c <= nbands
                    assert c == nbands or c == 1 or c <= steps // rb - 1
                    assert c <= max(want, 1)
                    if c == 1:
                        break
                    want = c - c // 4 - 1 if c > 2 else 1      # how a refused cooperative launch shrinks it
                else:
                    raise AssertionError("the shrink sequence did not reach 1")
    assert L.m2d_scan_chain_bound(4, 0, 8, 2) == 0


def test_test_hook_flag_needs_the_environment(L, monkeypatch):
    monkeypatch.delenv("M2D_TEST_HOOKS", raising=False)
    assert L.m2d_scan_fwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_TEST_WITHHOLD)), None) == -10
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    assert L.m2d_scan_fwd(ctypes.byref(_desc(flags=_lib.M2D_SCAN_TEST_WITHHOLD)), None) == -1   # accepted: next check


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_LIB", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _lib.lib()


def _pdesc(**kw):
    d = _lib.ProjDesc()
    d.struct_bytes = ctypes.sizeof(_lib.ProjDesc)
    d.dtype = _lib.M2D_F32
    d.P, d.E, d.R, d.N = 1000, 64, 4, 16
    d.proj_pitch = 56
    for k, v in kw.items():
        setattr(d, k, v)
    return d


def test_projection_descriptor_validation_without_a_device(L):
    assert L.m2d_dtproj_fwd(ctypes.byref(_pdesc()), None) == -1                  # NULL pointers
    assert L.m2d_dtproj_bwd(ctypes.byref(_pdesc(struct_bytes=8)), None) == -8
    assert L.m2d_dtproj_fwd(ctypes.byref(_pdesc(dtype=5)), None) == -2
    assert L.m2d_dtproj_fwd(ctypes.byref(_pdesc(P=0)), None) == -3
    assert L.m2d_dtproj_fwd(ctypes.byref(_pdesc(E=_lib.PROJ_MAX_E + 4)), None) == -9
    assert L.m2d_dtproj_bwd(ctypes.byref(_pdesc(R=_lib.PROJ_MAX_R + 1, proj_pitch=400)), None) == -9
    assert L.m2d_xproj_wgrad(ctypes.byref(_pdesc(proj_pitch=55)), None) == -5     # narrower than 2R+3N
    ws = L.m2d_proj_workspace(ctypes.byref(_pdesc()))
    assert ws > 0 and ws % 256 == 0
    assert L.m2d_proj_workspace(ctypes.byref(_pdesc(R=0))) == 0                   # invalid descriptor
