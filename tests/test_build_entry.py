"""build() where the reference checkout is missing or its folder is empty."""
import __graft_entry__ as entry


def test_an_empty_folder_is_no_reference_tree(tmp_path, monkeypatch):
    empty, tree = tmp_path / "empty", tmp_path / "tree"
    empty.mkdir()
    (tree / "tests" / "system_tests").mkdir(parents=True)
    monkeypatch.setenv("PHYSIS_REF", str(empty))
    assert entry.reference_tree() != str(empty)
    monkeypatch.setenv("PHYSIS_REF", str(tree))
    assert entry.reference_tree() == str(tree)
