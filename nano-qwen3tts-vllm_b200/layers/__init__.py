"""Drop-in layer modules: the reference's class names, constructor
signatures, parameter names and forward signatures, with the arithmetic in libb200tts.so."""
