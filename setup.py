"""The wheel carries compiled files (``physicsnemo_b200/lib``): it is for one platform and one Python."""
from setuptools import setup
from setuptools.dist import Distribution


class _Binary(Distribution):
    def has_ext_modules(self):
        return True


setup(distclass=_Binary)
