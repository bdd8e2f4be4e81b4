"""Where build() takes the reference's sources from: its tree where that holds
them, else the staged copy, else nowhere -- a directory without them (an empty
mount) is not the tree."""
import os


def make_tree(path):
    os.makedirs(path / "omp3")
    (path / "omp3" / "flow.c").write_text("/* a stand-in */\n")
    return str(path)


def test_empty_directory_is_no_reference(tmp_path):
    import __graft_entry__ as g
    empty = tmp_path / "empty"
    empty.mkdir()
    tree, staged = make_tree(tmp_path / "tree"), make_tree(tmp_path / "staged")
    assert g.reference_source(str(empty), str(empty)) is None
    assert g.reference_source(str(empty), staged) == staged
    assert g.reference_source(tree, staged) == tree
    assert g.reference_source(str(tmp_path / "missing"), str(tmp_path / "missing")) is None
