"""``lib.call`` goes to the library, and the entry point in it, that are there at the time of the call.  No GPU."""
import pytest

from qutai_b200 import lib


class Library:
    def __init__(self, code):
        self.code = code

    def qmoe_device_status(self):
        return self.code

    def qmoe_last_error(self):
        return b"from the stand-in"


def test_a_library_swapped_between_two_calls_is_seen(monkeypatch):
    monkeypatch.setattr(lib, "_library", Library(0))
    lib.call("qmoe_device_status")
    monkeypatch.setattr(lib, "_library", Library(-1))
    with pytest.raises(ValueError, match="from the stand-in"):
        lib.call("qmoe_device_status")


def test_an_entry_point_swapped_between_two_calls_is_seen(monkeypatch):
    library = Library(0)
    monkeypatch.setattr(lib, "load", lambda: library)
    lib.call("qmoe_device_status")
    library.qmoe_device_status = lambda: 7
    with pytest.raises(RuntimeError, match="from the stand-in"):
        lib.call("qmoe_device_status")
