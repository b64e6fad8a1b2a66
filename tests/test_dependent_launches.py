"""Which launches may start under the end of the kernel before them (no GPU: stand-ins for the libraries that note how each was
launched). Several products and the decode attention read weights, positions and older cache pages before they wait, so outside of
a model's step, where the call before may have written those, nothing may start early; and nothing at the head of a step."""
import threading

import pytest

from dryft_challenge_htn_2026_b200.csrc import api, build


class _Call:
    """A C function: takes attributes as ctypes' do."""

    def __init__(self, fn):
        self.fn = fn

    def __call__(self, *args):
        return self.fn(*args)


class Library:
    """The two switches of common.cuh, and a launch that notes what they say."""

    def __init__(self):
        self.everybody, self.threads, self.launched = 0, threading.local(), []
        self.dk_set_pdl = _Call(lambda on: setattr(self, "everybody", on))
        self.dk_set_thread_pdl = _Call(lambda on: setattr(self.threads, "on", on))
        self.dk_error_string = _Call(lambda e: b"")

    def launch(self):
        on = getattr(self.threads, "on", -1)
        self.launched.append(bool(on if on >= 0 else self.everybody))
        return 0


@pytest.fixture
def libs(monkeypatch):
    found = {"a.cu": Library(), "b.cu": Library()}
    monkeypatch.setattr(api, "_cuda_seen", True)
    monkeypatch.setattr(api, "_stream_ptr", lambda: 0)
    monkeypatch.setattr(build, "load_lib", lambda source, defines=None: build._libs.setdefault(
        (source, tuple(sorted((defines or {}).items()))), found[source]))
    yield found
    for source in found:
        build._libs.pop((source, ()), None)
        getattr(api._thread, "told", {}).pop((source, ()), None)


def call(source, kernels=1):
    lib = api._lib(source)
    for _ in range(kernels):
        err = lib.launch()
    api._check(lib, err, source, kernels)


def test_single_calls_never_start_early(libs):
    for source in ("a.cu", "b.cu", "a.cu"):
        call(source)
    assert libs["a.cu"].launched == [False, False] and libs["b.cu"].launched == [False]


def test_a_step_starts_whole_and_goes_on_dependent(libs):
    call("a.cu")
    with api.dependent_launches():
        call("b.cu", 2)                      # one call, two kernels
        with api.dependent_launches():       # the model's forward within a decode step
            call("a.cu")
        call("b.cu")
    call("a.cu"), call("b.cu")
    assert libs["a.cu"].launched == [False, True, False]
    assert libs["b.cu"].launched == [False, False, True, False]
    with pytest.raises(ZeroDivisionError):
        with api.dependent_launches():
            call("a.cu"), call("a.cu")
            1 / 0
    call("a.cu")
    assert libs["a.cu"].launched[3:] == [False, True, False]


def test_a_second_stream_within_a_step_starts_whole_as_well(libs, monkeypatch):
    on = [0]
    monkeypatch.setattr(api, "_stream_ptr", lambda: on[0])
    for _ in range(2):
        with api.dependent_launches():
            for on[0] in (0, 0, 7, 7, 0, 7):
                call("a.cu")
    assert libs["a.cu"].launched == [False, True, False, True, True, True] * 2


def test_another_threads_calls_are_not_part_of_the_step(libs):
    with api.dependent_launches():
        call("a.cu"), call("a.cu")
        t = threading.Thread(target=lambda: [call("a.cu"), call("a.cu")])
        t.start(), t.join()
        call("a.cu")
    assert libs["a.cu"].launched == [False, True, False, False, True]


def test_a_callers_own_choice_holds_everywhere(libs):
    try:
        for on in (True, False):
            api.set_pdl(on)
            call("a.cu")
            with api.dependent_launches():
                call("a.cu"), call("a.cu")
        assert libs["a.cu"].launched == [True] * 3 + [False] * 3
    finally:
        api.set_pdl(None)
    call("a.cu")
    assert libs["a.cu"].launched[-1] is False


@pytest.mark.parametrize("on", [False, True, None])
def test_what_a_test_chose_does_not_reach_the_next(on):
    assert api._pdl is None
    api.set_pdl(on)
