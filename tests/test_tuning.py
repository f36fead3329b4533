"""The run-time kernel configuration table (rocsolver_b200_tuning_*): parsing, round trip,
rejection of malformed text, loading from a file.  Host-only: no kernel runs."""
import rocsolver_b200 as rs

SUCCESS, INVALID_POINTER, INVALID_VALUE = 0, 3, 11


def _restore(text):
    assert rs.set_tuning_table(text) == SUCCESS


def test_roundtrip_sorted_and_comments():
    old = rs.tuning_table()
    try:
        text = ("# comment line\n"
                "vbatched d 512 256 2 16 64 1 0\n"
                "getrf d 256 256 1 32 64 0   # trailing comment\n"
                "getrf d 128 128 1 32 0 1\n"
                "getrf t 512 256 2 32 128 1\n"
                "getrf s 256 128 2 32 96 1\n")
        assert rs.set_tuning_table(text) == SUCCESS
        got = rs.tuning_table().splitlines()
        assert got == ["getrf d 128 128 1 32 0 1",
                       "getrf d 256 256 1 32 64 0",
                       "getrf s 256 128 2 32 96 1",
                       "getrf t 512 256 2 32 128 1",
                       "vbatched d 512 256 2 16 64 1 0"]
    finally:
        _restore(old)


def test_malformed_text_is_rejected_and_table_kept():
    old = rs.tuning_table()
    try:
        assert rs.set_tuning_table("getrf d 256 256 1 32 64 0\n") == SUCCESS
        for bad in ("getrf x 256 256 1 32 64 0", "getrf d 256 256 1 32 64",
                    "getrf d 256 256 1 32 64 0 9", "potrf d 64 1 2 3 4 5",
                    "getrf d 0 256 1 32 64 0", "getrf d 256 -1 1 32 64 0",
                    "vbatched d 512 256 2 16 64 1", "vbatched t 512 256 2 16 64 1 0"):
            assert rs.set_tuning_table(bad) == INVALID_VALUE, bad
            assert rs.tuning_table() == "getrf d 256 256 1 32 64 0\n"
        assert rs.lib().rocsolver_b200_tuning_set(None) == INVALID_POINTER
        assert rs.set_tuning_table("") == SUCCESS
        assert rs.tuning_table() == ""
    finally:
        _restore(old)


def test_load_from_file(tmp_path):
    old = rs.tuning_table()
    try:
        f = tmp_path / "t.txt"
        f.write_text("getrf s 512 256 2 16 128 0\n")
        assert rs.lib().rocsolver_b200_tuning_load(str(f).encode()) == SUCCESS
        assert rs.tuning_table() == "getrf s 512 256 2 16 128 0\n"
        assert rs.lib().rocsolver_b200_tuning_load(str(tmp_path / "missing").encode()) \
            == INVALID_VALUE
    finally:
        _restore(old)


def test_get_truncates_to_buffer():
    import ctypes
    old = rs.tuning_table()
    try:
        assert rs.set_tuning_table("getrf d 256 256 1 32 64 0\n") == SUCCESS
        buf = ctypes.create_string_buffer(8)
        full = rs.lib().rocsolver_b200_tuning_get(buf, 8)
        assert full == len("getrf d 256 256 1 32 64 0\n") + 1
        assert buf.value == b"getrf d"
    finally:
        _restore(old)


def test_tuner_keeps_the_built_in_choice_where_it_is_faster(tmp_path, monkeypatch):
    """A class whose best configuration is slower than the built-in choice gets a row of zeros
    (no configuration), also between classes that have one, and the library takes the file."""
    import sys

    import torch

    from rocsolver_b200 import tune
    times = {("d", 64): (1.6, 1.1), ("d", 128): (2.5, 3.0), ("s", 64): (1.0, 1.0),
             ("s", 128): (float("inf"), 2.0)}

    def fake_getrf(prec, n, bc, reps, quick, log):
        t, tb = times[prec, n]
        return (None if t == float("inf") else (256, 1, 32, 64, 1)), t, tb

    def fake_vbatched(prec, n, bc, reps, quick, log):
        return (256, 2, 32, 128, 0, 0), (5.0 if prec == "d" else 3.0), 4.0

    monkeypatch.setattr(tune, "tune_getrf", fake_getrf)
    monkeypatch.setattr(tune, "tune_vbatched", fake_vbatched)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "none")
    out = tmp_path / "table.txt"
    monkeypatch.setattr(sys, "argv", ["tune", "--out", str(out), "--classes", "64,128",
                                      "--vb-classes", "512", "--precisions", "d,s"])
    old = rs.tuning_table()
    tune.main()
    assert rs.tuning_table() == old
    try:
        assert rs.lib().rocsolver_b200_tuning_load(str(out).encode()) == SUCCESS
        assert rs.tuning_table().splitlines() == ["getrf d 64 0 0 0 0 0",
                                                  "getrf d 128 256 1 32 64 1",
                                                  "getrf s 64 0 0 0 0 0",
                                                  "getrf s 128 0 0 0 0 0",
                                                  "vbatched d 512 0 0 0 0 0 0",
                                                  "vbatched s 512 256 2 32 128 0 0"]
    finally:
        _restore(old)
