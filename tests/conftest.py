"""Shared pytest set-up: the ``gpu`` marker and the import path of the repository root."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.dirname(os.path.abspath(__file__))):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def pytest_collection_modifyitems(config, items):
    import torch

    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(autouse=True)
def the_callers_choice_of_dependent_launches_ends_with_the_test():
    """A test may switch dependent launches on or off for the whole process (api.set_pdl); the next one runs as users do."""
    yield
    from dryft_challenge_htn_2026_b200.csrc import api

    api.set_pdl(None)
