"""Installing the reference's CPU route: a missing, an empty and a complete tree."""

import os

from baseline import install_reference


def test_install_needs_the_files(tmp_path, monkeypatch):
    monkeypatch.setattr(install_reference, "HERE", str(tmp_path / "base"))
    installed = tmp_path / "base" / "_ref" / "kernel"
    assert install_reference.install(str(tmp_path / "absent")) is False
    tree = tmp_path / "tree"
    tree.mkdir()
    assert install_reference.install(str(tree)) is False and not installed.exists()
    for f in install_reference.FILES:
        (tree / f).parent.mkdir(parents=True, exist_ok=True)
        (tree / f).write_text("x = 1\n")
    assert install_reference.install(str(tree)) is True
    assert all(os.path.exists(installed / f) for f in install_reference.FILES)
    assert install_reference.install(str(tmp_path / "absent")) is True       # in place from before
