"""The build entry compiles the reference only where its sources are: an empty
directory in their place is as good as none."""
import __graft_entry__ as entry


def test_an_empty_tree_is_no_reference(tmp_path):
    assert not entry.reference_present(str(tmp_path))
    assert not entry.reference_present(str(tmp_path / "absent"))
    (tmp_path / "step_ch.c").write_text("")
    assert entry.reference_present(str(tmp_path))
