"""What build() leaves in the tree: the extension, and nothing beside it."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_keeps_its_objects_out_of_the_tree(monkeypatch):
    monkeypatch.syspath_prepend(ROOT)
    import __graft_entry__ as entry

    calls = []

    def run(args, **kw):
        calls.append(args)
        raise KeyboardInterrupt                          # nothing is compiled here

    monkeypatch.setattr(entry.subprocess, "run", run)
    try:
        entry.build()
    except KeyboardInterrupt:
        pass
    args = calls[0]
    assert args[:3] == [sys.executable, "setup.py", "build_ext"] and "--inplace" in args
    for option in ("--build-temp", "--build-lib"):
        assert not os.path.abspath(args[args.index(option) + 1]).startswith(ROOT + os.sep)
